// frame.h -- framed sweep programs of the interpreting kernels.
//
// An interpreter that runs CNOT as an operation moves registers under
// run-time masks (some 100 instructions a thread, more than a rotation), and
// every case of its switch must leave the 16 amplitudes where the others do.
// A framed program has no such operations. The planner tracks, per register
// phase, an affine map over GF(2) from where an amplitude is (register index
// j, thread bits, CTA bits) to the register bits of its index,
//
//     index = M j + D(thread bits, CTA bits) + const,
//
// and a linear sign (-1)^S of the same bits. X, Y, Z, CNOT, the swaps inside
// Rx and Ry by more than half a turn and the sign inside H only change M, D,
// const and S, on the host. A rotation pairs register j with j ^ v (v = the
// column of M^-1 of its bit), its orientation the parity of j and of thread
// bits; the map itself is undone for nothing by the shared-memory addresses
// to which the phase writes its result, S by the last pass of the sweep.
// Phases on thread and CTA bits alone are one number per thread: they come
// first in a phase, in a loop that touches no amplitude.
//
// Bound: latency and instruction issue of the dispatch, with 16 warps an SM
// at 128 registers (issue 40 % of the cycles, FP64 pipe 19..28 %, DRAM idle);
// a register of one tile waits mostly for instruction fetches. Measured
// against the form with CNOT operations: a batch of 48 registers of 10..20
// qubits 5.30 -> 4.25 ms, the five sweeps of a 21-qubit Fourier transform
// 248 -> 190 us, one tile of a 10-qubit ansatz 33.9 -> 26.8 us. Phases on three
// qubits and more are chains of records (a list that held one ran on the
// general interpreter before): 12 rotation layers with four of them each, 14
// and 20 qubits, 215 -> 179 and 439 -> 408 us; 48 such registers of 10..18
// qubits in a batch 1335 -> 1147 us, one such among 48 944 -> 694 us.
#pragma once

#include <cstdint>
#include <vector>

#include "tile_program.h"

namespace dgq {

// Dispatch codes: kind << 4 | v, v = 1..15 the direction (pair ops) or the
// parity mask (FK_PH, FK_NEG); FK_PH2 and FK_NEG2 have v = 0.
enum FrameKind : uint8_t {
    FK_RY = 0,    // [[1, -t], [t, 1]]
    FK_RX = 1,    // [[1, -i t], [-i t, 1]]
    FK_RN = 2,    // [[1, p], [-conj(p), 1]]
    FK_PH = 3,    // (c + i s) where the parity of j & v and of the thread part is 1
    FK_NEG = 4,   // the same with -1
    FK_PH2 = 5,   // (c + i s) where two such parities are 1
    FK_NEG2 = 6,
    // before an FK_PH2 or FK_NEG2, for phases on three or four register bits
    // or under a thread or CTA condition:
    FK_AND = 7,   // and where two more such parities are 1
    FK_IF = 8,    // and where every bit of the condition lm, cm is 1
};

// 16 bytes, read uniformly.
struct FOp {
    uint8_t code;
    uint8_t rr;    // FK_*2, FK_AND: parity mask of j of the first (low 4 bits) and second functional
    uint16_t tab;  // pair ops: bit j = parity of j (and the constant); FK_*2, FK_AND: bits 0, 1 the constants
    uint16_t lm, lm2;  // thread bits (tile-local) and
    uint32_t cm, cm2;  // CTA bits: pair ops and FK_PH / FK_NEG: parity masks lm, cm, condition lm2, cm2
                       // (all ones); FK_*2, FK_AND: parity masks of the first and second functional;
                       // FK_IF and scalar ops: condition lm, cm
};
static_assert(sizeof(FOp) == 16, "FOp layout");

struct FPhase {
    uint8_t thrPos[8];      // tile-local bit of thread-index bit i
    uint16_t rdOff[kRegs];  // swizzled shared-memory offsets of register j: read,
    uint16_t wrOff[kRegs];  // and written (M applied)
    uint32_t dc[kRegBits];  // D: parity masks of CTA bits,
    uint16_t dl[kRegBits];  // of thread bits,
    uint16_t col[kRegBits]; // and the swizzled offset of the register bit
    uint16_t opBegin, scalarEnd, opEnd;
    uint8_t hasD, fold;     // fold: thread factors are gathered and applied after the ops
};

// The end of a sweep, in the order of the store (register j holds tile-local
// bits W-4.., thread t the others).
struct FrameTail {
    int32_t globalPhase;  // >= 0: that phase's factors start from the global factor
    uint32_t signCta;
    uint16_t signThr;     // sign: parity of the thread index, the CTA index
    uint16_t signTab;     // and bit j
    int32_t hasSign, hasGlobal;
    double globalRe, globalIm;
};

constexpr int kFrameMaxOps = 760;

// Kernel parameter of one sweep of a single register.
struct FrameProgram {
    int32_t numPhases, numBits, numReal, initKind, hasRestrict, renormIn, renormOut, pad;
    const double *normIn;
    double *normOut;
    uint64_t initIndex;
    double initAmp;
    uint64_t restrictMask, restrictValue;
    double restrictScale;
    uint32_t ctaOffset, pad1;
    uint8_t highPos[kMaxTileBits - kCoalescedBits];
    uint8_t ctaPos[kMaxStateBits];
    FrameTail tail;
    FPhase phases[kMaxPhases];
    FOp ops[kFrameMaxOps];
    double coef[2 * kFrameMaxOps];  // two per op
};
static_assert(sizeof(FrameProgram) <= 32764, "FrameProgram must fit the kernel parameter space");

struct FrameSweep {
    FrameTail tail;
    std::vector<FPhase> phases;
    std::vector<FOp> ops;
    std::vector<double> coef;  // two per op
};

// The framed form of a tile program of width W (unpaired, W <= 12); false
// when an op has none (dense ops, controlled rotations and general 2x2 ops,
// controlled Y, X with several controls, 2x2 matrices that are not unitary to
// rounding) or there are more than kFrameMaxOps.
bool frameProgram(const TileProgram &p, int W, FrameSweep &out);

// The sweep on the host, on 2^numBits amplitudes (re, im pairs).
void applyFramedHost(const TileProgram &p, const FrameSweep &f, int W, double *state);

}  // namespace dgq
