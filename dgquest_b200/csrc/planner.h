// planner.h -- cuts a recorded gate list into state sweeps ("fused blocks")
// and encodes each sweep as a TileProgram for the tile kernel.
//
// dgQuEST cuts its circuit twice with the same greedy DAG selection
// (src/cpp/QuEST_backend.cpp:118-141,152-182): into sections that fit a task
// and into 11-qubit fused gates seeded with the 5 coalesced low bits, then
// re-DAGs each fused gate with budget 1 to group gates by target
// (src/cpp/QuEST_gpu_kernel.cu:529-562). On one GPU with the state resident
// in HBM there are no sections: the planner takes blocks of W tile bits
// (seeded with the 5 low bits, padded from bit 5 upward like
// QuEST_gpu_kernel.cu:504-509), then phases of 4 register bits.
#pragma once

#include <functional>
#include <string>
#include <vector>

#include "ir.h"
#include "tile_program.h"

namespace dgq {

struct BlockPlan {
    u64 tileMask = 0;         // W address bits, bits 0..4 always included
    std::vector<Gate> gates;  // dependency order
    bool last = true;         // no gates are left after this block
};

struct PlanStats {
    int sweeps = 0;     // kernel launches (state read+write passes)
    int phases = 0;     // register layouts summed over sweeps
    int ops = 0;        // kernel ops summed over sweeps
    int gates = 0;      // gates after merging
    double flopsPerAmp = 0;  // algorithmic FP64 flops per amplitude, summed over ops
};

// Multi-qubit unitary matrices referenced by OP_MULTI_UNITARY gates.
struct MatrixPool {
    std::vector<std::vector<double>> mats;  // row-major 2^k x 2^k, (re, im) interleaved
};

// Values of `lookahead` below: -1 by register size, 0 greedy, 1 greedy with a
// step of lookahead, or a beam search of width 4 or 16.
constexpr int kSearchBeam4 = 2, kSearchBeam16 = 3;

// `complete` (if given) is set to false when gates are left that no tile
// can hold (a gate with more non-diagonal targets than the tile width).
// seedBits: the lowest address bits every tile holds (5: the coalesced bits
// of complex128 tiles; 6 for the complex64 paired form, whose tile-local
// bit 0 is the pair inside a slot and bits 1..5 the coalesced slot bits).
// lookahead: 1 scores each candidate addition of tile bits by the best
// follow-up addition as well (fewer sweeps on deep circuits, 3x the
// planning time), 0 does not, -1 uses it for registers of >= 24 address bits
// (DGQ_PLAN_LOOKAHEAD_BITS overrides the 24).
std::vector<BlockPlan> planBlocks(const std::vector<Gate> &gates, int numBits, int tileBits, bool *complete = nullptr,
                                  int seedBits = kCoalescedBits, int lookahead = -1);
// The same blocks, handed to `onBlock` one at a time as they are chosen
// (a caller can encode and launch a sweep while the next one is planned);
// stops early when onBlock returns false. Returns false when gates are left
// that no tile can hold.
bool planBlocksEach(const std::vector<Gate> &gates, int numBits, int tileBits, int seedBits,
                    const std::function<bool(BlockPlan &)> &onBlock, int lookahead = -1);
// Whether lookahead -1 means lookahead for a register of numBits bits.
bool lookaheadBySize(int numBits);

// Encodes one block. The gate list may not fit one TileProgram; then the
// block is emitted as several programs over the same tile (each one more
// sweep). Only the first program carries `first` (init / lazy collapse).
struct SweepHeader {
    int32_t initKind = INIT_NONE;
    uint64_t initIndex = 0;
    double initAmp = 0.0;
    bool hasRestrict = false;
    uint64_t restrictMask = 0, restrictValue = 0;
    double restrictScale = 1.0;
};

// The kernel a program is for, as far as the plan depends on it.
enum class Folding { None, Framed, Specialised };

// paired: encode for the complex64 paired form (TileProgram::paired); fails
// (with *err set) on a multi-qubit unitary that targets address bit 0.
// folds: the program is for a kernel that folds phase factors on thread bits
// into one factor per thread (a specialised one, or the framed interpreter);
// diagonal gates then move to the phases where they are such factors. carry (with folds): diagonal gates of
// the block before, run first here; the block's own that would be cheaper in
// the next block are left in it (none when the block is the last).
// single: a complex64 state. Its kernels apply a program's scalar (the product
// of the factors that rotations and Hadamards leave out) as one float, before,
// between or after the ops, so a program ends before it falls below
// 2^-kMaxScalarBitsF32: amplitudes then grow by at most 2^80 of the 2^127 a
// float holds, and what drops below its 2^-149 is under 2^-69 of the norm.
// (640 Hadamards in one sweep leave 2^-320: 0 as a float.) In complex128 the
// ops of one program cannot leave that range.
constexpr double kMaxScalarBitsF32 = 80.0;
bool encodeBlock(const BlockPlan &block, int numBits, int numReal, int tileBits, const MatrixPool &pool,
                 const SweepHeader &first, std::vector<TileProgram> &out, PlanStats *stats, std::string *err,
                 bool paired = false, Folding folds = Folding::None, std::vector<Gate> *carry = nullptr,
                 bool single = false);

// Whether the framed interpreter is likely to run every gate (frame.h) and
// placing diagonal gates for it pays (a general 2x2 without controls may still
// turn out to have no framed form, and then runs on the other interpreter,
// which runs any plan but the specialised kernels').
bool framedGates(const std::vector<Gate> &gates);

// A program that only applies the header (init and/or lazy collapse).
void encodeHeaderOnly(int numBits, int numReal, int tileBits, const SweepHeader &hdr, TileProgram &out,
                      bool paired = false);

// Algorithmic FP64 flops per amplitude of one kernel op (formulas of
// QuEST_gpu_kernel.cu:17-170 counted as multiplies + adds per amplitude,
// averaged over the amplitudes it touches when uncontrolled).
double opFlopsPerAmp(const KOp &op);

}  // namespace dgq
