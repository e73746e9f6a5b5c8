// kernels.cu -- the sm_100a kernels of the FP64 state-vector path.
//
//   frameKernel<W,V> one sweep of the state applying a fused block
//                    (dgQuEST statevec_fusedKernel, QuEST_gpu_kernel.cu:175-359)
//   tileKernel<W,V>  the same for programs without a framed form
//   probKernel       P(bit = 0) for every address bit in one read pass
//   probFinalize     (statevec_findProbabilityOfZeroKernel + reducePingpong,
//                    QuEST_gpu_kernel.cu:656-840)
//   swapBitsKernel   in-HBM exchange of address-bit pairs (the successor of
//                    reorder_data_kernel, QuEST_gpu_kernel.cu:589-654)
//   gatherKernel     logical-order copy-out of the state through the
//                    logical->virtual map
//
// The state is 2^numBits double2 (re, im) amplitudes in HBM, in place.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "frame.cuh"
#include "interp.cuh"
#include "kernels.h"
#include "tile_program.h"

namespace dgq {

__device__ __forceinline__ uint32_t swz(uint32_t x) { return x ^ (((x >> 3) ^ (x >> 6) ^ (x >> 9) ^ (x >> 12)) & 7u); }

// ------------------------------------------------------------ tile kernels
// Canonical order of a tile: element (tid, j) at base | lane bits | thread
// high bits | j bits. Prog: TileProgram or FrameProgram.
template <int W>
struct TileAddress {
    uint64_t tpart, jb[kRegBits];
    template <class Prog>
    __device__ __forceinline__ TileAddress(const Prog &prog, uint32_t tid, uint32_t cta) {
        tpart = tid & 31u;
        const int nCta = prog.numBits - W;
        for (int i = 0; i < nCta; i++) tpart |= (uint64_t) ((cta >> i) & 1u) << prog.ctaPos[i];
#pragma unroll
        for (int i = 0; i < W - 9; i++) tpart |= (uint64_t) ((tid >> (5 + i)) & 1u) << prog.highPos[i];
#pragma unroll
        for (int b = 0; b < kRegBits; b++) jb[b] = 1ULL << prog.highPos[W - 9 + b];
    }
    __device__ __forceinline__ uint64_t operator()(int j) const {
        return tpart | ((j & 1) ? jb[0] : 0ULL) | ((j & 2) ? jb[1] : 0ULL) | ((j & 4) ? jb[2] : 0ULL) | ((j & 8) ? jb[3] : 0ULL);
    }
};

template <int W, class V, class Prog>
__device__ __forceinline__ void loadTile(const V *st, const Prog &prog, const TileAddress<W> &gidx, V (&a)[kRegs]) {
    typedef typename Real<V>::T R;
    if (prog.initKind == INIT_NONE) {
#pragma unroll
        for (int j = 0; j < kRegs; j++) a[j] = st[gidx(j)];
    } else {
        const uint64_t ci = prog.initIndex;
        const double pa = prog.initAmp;
        const int kind = prog.initKind;
        const int nr = prog.numReal;
#pragma unroll
        for (int j = 0; j < kRegs; j++) {
            const uint64_t g = gidx(j);
            double re = 0.0;
            if (kind == INIT_CLASSICAL)
                re = (g == ci) ? 1.0 : 0.0;
            else if (kind == INIT_PLUS)
                re = ((g >> nr) == 0ULL) ? pa : 0.0;
            a[j] = mk<V>((R) re, (R) 0);
        }
    }
    if (prog.hasRestrict) {
        const uint64_t rm = prog.restrictMask, rv = prog.restrictValue;
        const R sc = (R) prog.restrictScale;
#pragma unroll
        for (int j = 0; j < kRegs; j++) {
            const bool keep = (gidx(j) & rm) == rv;
            a[j] = keep ? mk<V>(a[j].x * sc, a[j].y * sc) : mk<V>((R) 0, (R) 0);
        }
    }
}

// Adds the tile's sum of |a|^2 to *normOut.
template <int T, class V>
__device__ __forceinline__ void addNorm(const V (&a)[kRegs], uint32_t tid, double *normOut) {
    __shared__ double red[32];
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < kRegs; j++) acc += (double) a[j].x * (double) a[j].x + (double) a[j].y * (double) a[j].y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((tid & 31u) == 0) red[tid >> 5] = acc;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < T / 32; w++) t += red[w];
        atomicAdd(normOut, t);
    }
}

// 128 registers per thread: 16 warps per SM at every tile width. V is
// double2 (complex128) or float2 (complex64, with the per-sweep
// renormalisation of the complex64 form: scale by 1/sqrt(*normIn) with the
// global factor, add the output's sum of |a|^2 to *normOut).
// Programs with an op that no framed program holds (frame.h).
template <int W, class V>
__global__ void __launch_bounds__(1 << (W - kRegBits), 65536 / (128 << (W - kRegBits)))
    tileKernel(V *__restrict__ st, const __grid_constant__ TileProgram prog) {
    typedef typename Real<V>::T R;
    constexpr int T = 1 << (W - kRegBits);
    extern __shared__ __align__(16) unsigned char smRaw[];
    V *sm = reinterpret_cast<V *>(smRaw);
    const uint32_t tid = threadIdx.x;
    const uint32_t cta = blockIdx.x + prog.ctaOffset;
    const TileAddress<W> gidx(prog, tid, cta);
    V a[kRegs];
    loadTile<W>(st, prog, gidx, a);

    const int numPhases = prog.numPhases;
    if (numPhases > 0) {
#pragma unroll
        for (int j = 0; j < kRegs; j++) sm[swz(tid + (uint32_t) (T * j))] = a[j];
        __syncthreads();
        for (int p = 0; p < numPhases; p++) {
            const KPhase &ph = prog.phases[p];
            uint32_t loc = 0;
#pragma unroll
            for (int i = 0; i < W - kRegBits; i++) loc |= ((tid >> i) & 1u) << ph.thrPos[i];
            const uint32_t sb = swz(loc);
#pragma unroll
            for (int j = 0; j < kRegs; j++) a[j] = sm[sb ^ ph.regOff[j]];
            const int e = ph.opEnd;
            for (int o = ph.opBegin; o < e; o++) applyOp<V, true>(prog.ops[o], prog.coef, a, loc, cta);
#pragma unroll
            for (int j = 0; j < kRegs; j++) sm[sb ^ ph.regOff[j]] = a[j];
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < kRegs; j++) a[j] = sm[swz(tid + (uint32_t) (T * j))];
    }
    if (prog.hasGlobal || prog.renormIn) {
        double grd = prog.globalRe, gid = prog.globalIm;
        if (prog.renormIn) {
            const double sc = rsqrt(*prog.normIn);
            grd *= sc;
            gid *= sc;
        }
        const R gr = (R) grd, gi = (R) gid;
#pragma unroll
        for (int j = 0; j < kRegs; j++) a[j] = mk<V>(gr * a[j].x - gi * a[j].y, gr * a[j].y + gi * a[j].x);
    }
    if (prog.renormOut) addNorm<T>(a, tid, prog.normOut);
#pragma unroll
    for (int j = 0; j < kRegs; j++) st[gidx(j)] = a[j];
}

// The framed form (frame.h).
template <int W, class V>
__global__ void __launch_bounds__(1 << (W - kRegBits), 65536 / (128 << (W - kRegBits)))
    frameKernel(V *__restrict__ st, const __grid_constant__ FrameProgram prog) {
    constexpr int T = 1 << (W - kRegBits);
    extern __shared__ __align__(16) unsigned char smRaw[];
    V *sm = reinterpret_cast<V *>(smRaw);
    const uint32_t tid = threadIdx.x;
    const uint32_t cta = blockIdx.x + prog.ctaOffset;
    V a[kRegs];
    loadTile<W>(st, prog, TileAddress<W>(prog, tid, cta), a);
    if (prog.numPhases > 0) {
#pragma unroll
        for (int j = 0; j < kRegs; j++) sm[swz(tid + (uint32_t) (T * j))] = a[j];
        __syncthreads();
        framePhases<V, W>(
            prog.numPhases, prog.tail, sm, tid, cta, [&](int p) -> const FPhase & { return prog.phases[p]; },
            [&](int o) -> const FOp & { return prog.ops[o]; },
            [&](int o) { return make_double2(prog.coef[2 * o], prog.coef[2 * o + 1]); }, [] { __syncthreads(); });
#pragma unroll
        for (int j = 0; j < kRegs; j++) a[j] = sm[swz(tid + (uint32_t) (T * j))];
    }
    frameFinish(prog.tail, a, tid, cta, prog.renormIn != 0, prog.renormIn ? rsqrt(*prog.normIn) : 1.0);
    if (prog.renormOut) addNorm<T>(a, tid, prog.normOut);
    const TileAddress<W> gidx(prog, tid, cta);
#pragma unroll
    for (int j = 0; j < kRegs; j++) st[gidx(j)] = a[j];
}

template <int W, class V>
static cudaError_t launchTileW(V *st, const TileProgram &prog, cudaStream_t s) {
    const size_t smem = sizeof(V) << W;
    const unsigned grid = prog.ctaCount ? prog.ctaCount : 1u << (prog.numBits - W);
    FrameSweep f;
    if (!frameProgram(prog, W, f)) {
        static std::atomic<uint64_t> optIn{0};
        cudaError_t e = ensureSmemOptIn((const void *) tileKernel<W, V>, (int) smem, optIn);
        if (e != cudaSuccess) return e;
        tileKernel<W, V><<<grid, 1 << (W - kRegBits), smem, s>>>(st, prog);
        return cudaGetLastError();
    }
    static std::atomic<uint64_t> optIn{0};
    cudaError_t e = ensureSmemOptIn((const void *) frameKernel<W, V>, (int) smem, optIn);
    if (e != cudaSuccess) return e;
    FrameProgram fp;
    fp.numPhases = prog.numPhases;
    fp.numBits = prog.numBits;
    fp.numReal = prog.numReal;
    fp.initKind = prog.initKind;
    fp.hasRestrict = prog.hasRestrict;
    fp.renormIn = prog.renormIn;
    fp.renormOut = prog.renormOut;
    fp.normIn = prog.normIn;
    fp.normOut = prog.normOut;
    fp.initIndex = prog.initIndex;
    fp.initAmp = prog.initAmp;
    fp.restrictMask = prog.restrictMask;
    fp.restrictValue = prog.restrictValue;
    fp.restrictScale = prog.restrictScale;
    fp.ctaOffset = prog.ctaOffset;
    std::memcpy(fp.highPos, prog.highPos, sizeof(fp.highPos));
    std::memcpy(fp.ctaPos, prog.ctaPos, sizeof(fp.ctaPos));
    fp.tail = f.tail;
    std::copy(f.phases.begin(), f.phases.end(), fp.phases);
    std::copy(f.ops.begin(), f.ops.end(), fp.ops);
    std::copy(f.coef.begin(), f.coef.end(), fp.coef);
    frameKernel<W, V><<<grid, 1 << (W - kRegBits), smem, s>>>(st, fp);
    return cudaGetLastError();
}

template <class V>
static cudaError_t launchTileV(V *st, int tileBits, const TileProgram &prog, cudaStream_t s) {
    switch (tileBits) {
        case 9: return launchTileW<9>(st, prog, s);
        case 10: return launchTileW<10>(st, prog, s);
        case 11: return launchTileW<11>(st, prog, s);
        case 12: return launchTileW<12>(st, prog, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launchTile(void *st, bool single, int tileBits, const TileProgram &prog, cudaStream_t s) {
    if (prog.paired) return cudaErrorInvalidValue;  // the paired form is runtime-specialised only
    return single ? launchTileV((float2 *) st, tileBits, prog, s) : launchTileV((double2 *) st, tileBits, prog, s);
}

// ------------------------------------------------------- probabilities
// Sub-index s enumerates the amplitudes allowed by the lazy collapse
// (address bits outside `restrict` mask): address = rValue | deposit(s).
// With VB = 1 (complex64, address bit 0 free) s bit 0 is inside a 16-byte
// load. Above it 8 bits = thread, 4 = register j, kappa = unit within the
// CTA, the rest = blockIdx. Each CTA writes kProbSlots partial sums: the
// zero-sum of sub-index bit i at slot i (inside the CTA), its total last.
//
// Bound: HBM (one read of the state). Loads are 16 bytes a lane in either
// precision, 16 of them in flight; the 16 values are added as a tree whose
// nodes give the four j sums (26 adds for 16 values instead of 48), and
// lane-bit sums come out of the warp's butterfly (15 shuffles instead of
// 45). kappa keeps at least 2048 CTAs where the state has as many units: at
// 2^21 amplitudes 512 CTAs instead of the 32 that 16 units a CTA left.
// Measured (us, before -> now): complex128 2^17 61 -> 4.4, 2^21 73 -> 8.9,
// 2^25 141 -> 106, 2^30 2777 -> 2564 (6.7 TB/s); complex64 2^23 88 -> 15,
// 2^29 1204 -> 701 (6.1 TB/s).
template <class V, int VB>
__global__ void __launch_bounds__(256, 3) probKernel(const V *__restrict__ st, const __grid_constant__ ProbArgs args, double *partial) {
    const uint32_t tid = threadIdx.x;
    const uint32_t cta = blockIdx.x;
    const int nFree = args.nFree;
    const int kappa = args.kappa;
    auto bitOf = [&](int i) -> uint64_t { return i < nFree ? (1ULL << args.freePos[i]) : 0ULL; };
    uint64_t base = args.rValue;
#pragma unroll
    for (int i = 0; i < 8; i++)
        if ((tid >> i) & 1u) base |= bitOf(VB + i);
    for (int i = 0; VB + 12 + kappa + i < nFree; i++)
        if ((cta >> i) & 1u) base |= bitOf(VB + 12 + kappa + i);
    const uint64_t jb[4] = {bitOf(VB + 8), bitOf(VB + 9), bitOf(VB + 10), bitOf(VB + 11)};
    // registers narrower than one unit: only sub-indices below 2^nFree exist
    const bool full = nFree >= VB + 12;
    const uint32_t limit = full ? 0u : 1u << (nFree > VB ? nFree - VB : 0);

    double tot = 0.0, zb = 0.0;       // zb: sub-index bit 0 = 0 (VB = 1)
    double zj[4] = {0.0, 0.0, 0.0, 0.0};
    double zu[kProbMaxKappa] = {};
    const int units = 1 << kappa;
    for (int u = 0; u < units; u++) {
        uint64_t g0 = base;
        for (int b = 0; b < kappa; b++)
            if ((u >> b) & 1) g0 |= bitOf(VB + 12 + b);
        double p[16], lo = 0.0;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const uint64_t g = g0 | ((j & 1) ? jb[0] : 0ULL) | ((j & 2) ? jb[1] : 0ULL) | ((j & 4) ? jb[2] : 0ULL) |
                               ((j & 8) ? jb[3] : 0ULL);
            p[j] = 0.0;
            if (full || (tid | ((uint32_t) j << 8)) < limit) {
                if constexpr (VB == 1) {
                    const float4 v = *reinterpret_cast<const float4 *>(st + g);
                    const double ar = (double) v.x, ai = (double) v.y, br = (double) v.z, bi = (double) v.w;
                    const double l = ar * ar + ai * ai;
                    lo += l;
                    p[j] = l + (br * br + bi * bi);
                } else {
                    const V v = st[g];
                    const double re = (double) v.x, im = (double) v.y;
                    p[j] = re * re + im * im;
                }
            }
        }
        zb += lo;
        double a[8], c[4];
#pragma unroll
        for (int i = 0; i < 8; i++) a[i] = p[2 * i] + p[2 * i + 1];
#pragma unroll
        for (int i = 0; i < 4; i++) c[i] = a[2 * i] + a[2 * i + 1];
        zj[0] += ((p[0] + p[2]) + (p[4] + p[6])) + ((p[8] + p[10]) + (p[12] + p[14]));
        zj[1] += (a[0] + a[2]) + (a[4] + a[6]);
        zj[2] += c[0] + c[2];
        zj[3] += c[0] + c[1];
        const double ut = (c[0] + c[1]) + (c[2] + c[3]);
        tot += ut;
#pragma unroll
        for (int b = 0; b < kProbMaxKappa; b++)
            if (b < kappa && !((u >> b) & 1)) zu[b] += ut;
    }
    // per warp: [0..5) lane bits, 5 total, 6 bit 0 of a pair, [7..11) j, [11..) units
    __shared__ double red[8][11 + kProbMaxKappa];
    const int lane = tid & 31, warp = tid >> 5;
    double z[5], sum = tot;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const double other = __shfl_xor_sync(0xffffffffu, sum, 1 << k);
        z[k] = ((lane >> k) & 1) ? other : sum;
        sum += other;
#pragma unroll
        for (int i = 0; i < k; i++) z[i] += __shfl_xor_sync(0xffffffffu, z[i], 1 << k);
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 5; k++) red[warp][k] = z[k];
        red[warp][5] = sum;
    }
    auto reduce = [&](double x, int slot) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[warp][slot] = x;
    };
    if constexpr (VB == 1) reduce(zb, 6);
#pragma unroll
    for (int k = 0; k < 4; k++) reduce(zj[k], 7 + k);
#pragma unroll
    for (int b = 0; b < kProbMaxKappa; b++)
        if (b < kappa) reduce(zu[b], 11 + b);
    __syncthreads();
    const int inside = VB + 12 + kappa;
    if ((int) tid < inside || tid == kProbSlots - 1) {
        const int i = (int) tid - VB;  // sub-index bit above the load
        const bool warpBit = tid != kProbSlots - 1 && i >= 5 && i < 8;
        const int slot = tid == kProbSlots - 1 || warpBit ? 5 : i < 0 ? 6 : i < 5 ? i : i - 1;
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < 8; w++)
            if (!warpBit || !((w >> (i - 5)) & 1)) x += red[w][slot];
        partial[(size_t) cta * kProbSlots + tid] = x;
    }
}

// out[b] for sub-index bit b < nFree, out[nFree] = total.
__global__ void __launch_bounds__(256) probFinalize(const double *__restrict__ partial, int numCtas, int nFree,
                                                   int inside, double *out) {
    const int b = blockIdx.x;  // 0..nFree
    double x = 0.0;
    const int slot = b < nFree && b < inside ? b : kProbSlots - 1;
    const int skip = b < nFree && b >= inside ? 1 << (b - inside) : 0;
    for (int c = threadIdx.x; c < numCtas; c += blockDim.x)
        if (!(c & skip)) x += partial[(size_t) c * kProbSlots + slot];
    __shared__ double red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int) (blockDim.x >> 5); w++) t += red[w];
        out[b] = t;
    }
}

void probShape(ProbArgs &args, bool single) {
    args.pairs = single && args.nFree > 0 && args.freePos[0] == 0 ? 1 : 0;
    const int unitBits = std::max(0, args.nFree - 12 - args.pairs);
    args.kappa = std::min(kProbMaxKappa, std::max(0, unitBits - 11));
}

cudaError_t launchProb(const void *st, bool single, const ProbArgs &args, double *partial, double *out,
                       cudaStream_t s) {
    const int grid = probNumCtas(args);
    if (single && args.pairs)
        probKernel<float2, 1><<<grid, 256, 0, s>>>((const float2 *) st, args, partial);
    else if (single)
        probKernel<float2, 0><<<grid, 256, 0, s>>>((const float2 *) st, args, partial);
    else
        probKernel<double2, 0><<<grid, 256, 0, s>>>((const double2 *) st, args, partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    probFinalize<<<args.nFree + 1, 256, 0, s>>>(partial, grid, args.nFree, 12 + args.pairs + args.kappa, out);
    return cudaGetLastError();
}

int probNumCtas(const ProbArgs &args) {
    const int inside = 12 + args.pairs + args.kappa;
    return args.nFree > inside ? (1 << (args.nFree - inside)) : 1;
}

// Page-pair exchange of the host tier: pages a and b differ only in the
// page-index bit that is being exchanged with local bit `bit`; every
// amplitude of a whose local index has `bit` = 1 trades places with the
// amplitude of b at the same index with `bit` = 0 (the two halves that the
// exchange of the two address bits moves).
template <class V>
__global__ void pageSwapKernel(V *__restrict__ a, V *__restrict__ b, int pageBits, int bit) {
    const uint64_t half = 1ULL << (pageBits - 1);
    const uint64_t lo = (1ULL << bit) - 1;
    for (uint64_t k = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; k < half;
         k += (uint64_t) gridDim.x * blockDim.x) {
        const uint64_t i = ((k & ~lo) << 1) | (1ULL << bit) | (k & lo);
        const uint64_t j = i ^ (1ULL << bit);
        const V x = a[i];
        a[i] = b[j];
        b[j] = x;
    }
}

// --------------------------------------------------- bit-pair exchange
// The amplitude at each index moves to the index with the bits of every pair
// exchanged, in place. A tile spans the lowest address bits and their
// partners, so that runs of at least 128 bytes (64 in complex64 registers of
// up to 14 bits, whose tiles are of 2^6) are read and written whole whichever
// bits trade places; a CTA holds a tile and the one it trades with
// in shared memory and stores each in the other's place, permuted.
// Bound: HBM, every amplitude read and written once. (One thread per pair of
// amplitudes touched 16 bytes of a 64-byte DRAM access at one of the two ends
// and left the other half of the threads idle.) Bit reversal of 2^27
// complex128 amplitudes 3.81 -> 0.74 ms (5.8 TB/s), of 2^28 complex64 7.29 ->
// 1.26 ms, of 2^21 complex128, in L2, 28.0 -> 21.0 us.
constexpr int kSwapTileBits = 10;

template <class V>
__global__ void __launch_bounds__(256) swapBitsKernel(V *__restrict__ st, const __grid_constant__ SwapTileArgs args) {
    __shared__ V tile[2][1 << kSwapTileBits];
    constexpr int kPer = (1 << kSwapTileBits) / 256;
    // thread t's elements t + 256 k: address within the tile, and the element
    // that goes there
    auto address = [&](uint32_t t) {
        uint64_t g = 0;
        for (int i = 0; i < args.tileBits; i++) g |= (uint64_t) ((t >> i) & 1u) << args.tilePos[i];
        return g;
    };
    auto source = [&](uint32_t t) {
        for (int k = 0; k < args.tilePairs; k++) {
            const uint32_t d = ((t >> args.tileA[k]) ^ (t >> args.tileB[k])) & 1u;
            t ^= (d << args.tileA[k]) | (d << args.tileB[k]);
        }
        return t;
    };
    const uint32_t size = 1u << args.tileBits, tid = threadIdx.x;
    uint64_t g[kPer];
    uint32_t s[kPer];
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        g[k] = address(tid + 256u * (uint32_t) k);
        s[k] = swz(source(tid + 256u * (uint32_t) k));
    }
    for (uint64_t o = blockIdx.x; o < (1ULL << args.outBits); o += gridDim.x) {
        uint64_t base = 0;
        for (int i = 0; i < args.outBits; i++) base |= ((o >> i) & 1ULL) << args.outPos[i];
        uint64_t other = base;
        for (int k = 0; k < args.outPairs; k++) {
            const uint64_t d = ((base >> args.outA[k]) ^ (base >> args.outB[k])) & 1ULL;
            other ^= (d << args.outA[k]) | (d << args.outB[k]);
        }
        if (other < base) continue;  // that tile's CTA does both
        const bool two = other != base;
        V x[kPer], y[kPer];
#pragma unroll
        for (int k = 0; k < kPer; k++)
            if (tid + 256u * (uint32_t) k < size) {
                x[k] = st[base | g[k]];
                if (two) y[k] = st[other | g[k]];
            }
#pragma unroll
        for (int k = 0; k < kPer; k++)
            if (tid + 256u * (uint32_t) k < size) {
                tile[0][swz(tid + 256u * (uint32_t) k)] = x[k];
                if (two) tile[1][swz(tid + 256u * (uint32_t) k)] = y[k];
            }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; k++)
            if (tid + 256u * (uint32_t) k < size) {
                st[other | g[k]] = tile[0][s[k]];
                if (two) st[base | g[k]] = tile[1][s[k]];
            }
        __syncthreads();
    }
}

cudaError_t launchPageSwap(void *a, void *b, bool single, int pageBits, int bit, cudaStream_t s) {
    if (pageBits < 1 || bit < 0 || bit >= pageBits) return cudaErrorInvalidValue;
    const uint64_t half = 1ULL << (pageBits - 1);
    const unsigned grid = (unsigned) std::min<uint64_t>((half + 255) / 256, 148u * 16u);
    if (single)
        pageSwapKernel<float2><<<grid, 256, 0, s>>>((float2 *) a, (float2 *) b, pageBits, bit);
    else
        pageSwapKernel<double2><<<grid, 256, 0, s>>>((double2 *) a, (double2 *) b, pageBits, bit);
    return cudaGetLastError();
}

// Block exchange between two shards (sharded registers, several qubits at
// once): for every offset o whose bits at the m positions pos[] are 0,
// x[o | patX] trades places with y[o | patY] (patX, patY: patterns over those
// positions). k enumerates the offsets; inserting a 0 at each position in
// ascending order turns k into o, so consecutive threads touch consecutive
// amplitudes except across the inserted bits.
template <class V>
__global__ void blockSwapKernel(V *__restrict__ x, V *__restrict__ y, const __grid_constant__ BlockSwapArgs args) {
    const uint64_t count = 1ULL << (args.pageBits - args.m);
    for (uint64_t k = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; k < count;
         k += (uint64_t) gridDim.x * blockDim.x) {
        uint64_t o = k;
        for (int t = 0; t < args.m; t++) {
            const int b = args.pos[t];
            o = ((o >> b) << (b + 1)) | (o & ((1ULL << b) - 1));
        }
        const V v = x[o | args.patX];
        x[o | args.patX] = y[o | args.patY];
        y[o | args.patY] = v;
    }
}

cudaError_t launchBlockSwap(void *x, void *y, bool single, const BlockSwapArgs &args, cudaStream_t s) {
    // positions ascending, inside the shard, patterns on them only
    if (args.m < 1 || args.m > 4 || args.pageBits <= args.m || args.pageBits > 40) return cudaErrorInvalidValue;
    uint64_t mask = 0;
    for (int t = 0; t < args.m; t++) {
        if (args.pos[t] < 0 || args.pos[t] >= args.pageBits || (t > 0 && args.pos[t] <= args.pos[t - 1]))
            return cudaErrorInvalidValue;
        mask |= 1ULL << args.pos[t];
    }
    if ((args.patX & ~mask) || (args.patY & ~mask)) return cudaErrorInvalidValue;
    const uint64_t count = 1ULL << (args.pageBits - args.m);
    const unsigned grid = (unsigned) std::min<uint64_t>((count + 255) / 256, 148u * 16u);
    if (single)
        blockSwapKernel<float2><<<grid, 256, 0, s>>>((float2 *) x, (float2 *) y, args);
    else
        blockSwapKernel<double2><<<grid, 256, 0, s>>>((double2 *) x, (double2 *) y, args);
    return cudaGetLastError();
}

cudaError_t launchSwapBits(void *st, bool single, const SwapArgs &args, cudaStream_t s) {
    if (args.numPairs < 0 || args.numPairs > 32) return cudaErrorInvalidValue;
    int partner[kMaxStateBits];
    for (int b = 0; b < kMaxStateBits; b++) partner[b] = b;
    for (int k = 0; k < args.numPairs; k++) {
        const int a = args.a[k], b = args.b[k];
        if (a >= args.numBits || b >= args.numBits || a == b || partner[a] != a || partner[b] != b)
            return cudaErrorInvalidValue;
        partner[a] = b;
        partner[b] = a;
    }
    // the lowest bits with their partners; at least 2^8 tiles where that leaves
    // the 3 lowest bits, so that small states still fill the GPU
    const int tileBits = std::min(kSwapTileBits, std::max(6, args.numBits - 8));
    uint64_t mask = 0;
    int n = 0;
    auto take = [&](int b) {
        const uint64_t add = ((1ULL << b) | (1ULL << partner[b])) & ~mask;
        if (n + __builtin_popcountll(add) > tileBits) return;
        mask |= add;
        n += __builtin_popcountll(add);
    };
    for (int b = 0; b < args.numBits; b++) take(b);
    SwapTileArgs t;
    std::memset(&t, 0, sizeof(t));
    int local[kMaxStateBits];
    for (int b = 0; b < args.numBits; b++) {
        if ((mask >> b) & 1ULL) {
            local[b] = t.tileBits;
            t.tilePos[t.tileBits++] = (uint8_t) b;
        } else {
            t.outPos[t.outBits++] = (uint8_t) b;
        }
    }
    for (int k = 0; k < args.numPairs; k++) {
        if ((mask >> args.a[k]) & 1ULL) {
            t.tileA[t.tilePairs] = (uint8_t) local[args.a[k]];
            t.tileB[t.tilePairs++] = (uint8_t) local[args.b[k]];
        } else {
            t.outA[t.outPairs] = args.a[k];
            t.outB[t.outPairs++] = args.b[k];
        }
    }
    const unsigned blocks = (unsigned) std::min<uint64_t>(1ULL << t.outBits, 148ULL * 64);
    if (single)
        swapBitsKernel<float2><<<blocks, 256, 0, s>>>((float2 *) st, t);
    else
        swapBitsKernel<double2><<<blocks, 256, 0, s>>>((double2 *) st, t);
    return cudaGetLastError();
}

// ------------------------------------------------------------ gather
// out[l] = st[virt(l)] for logical indices l in [begin, begin + count),
// with virt() the logical->virtual bit map and the lazy collapse applied.
template <class V>
__global__ void gatherKernel(const V *__restrict__ st, const __grid_constant__ GatherArgs args, double2 *__restrict__ out) {
    for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < args.count;
         i += (uint64_t) gridDim.x * blockDim.x) {
        const uint64_t l = args.begin + i * (args.stride ? args.stride : 1ULL);
        uint64_t v = 0;
        for (int b = 0; b < args.numReal; b++) v |= ((l >> b) & 1ULL) << args.l2v[b];
        double2 x = make_double2((double) st[v].x, (double) st[v].y);
        if (args.hasRestrict) {
            if ((v & args.restrictMask) != args.restrictValue)
                x = make_double2(0.0, 0.0);
            else
                x = make_double2(x.x * args.restrictScale, x.y * args.restrictScale);
        }
        out[i] = x;
    }
}

cudaError_t launchGather(const void *st, bool single, const GatherArgs &args, double2 *out, cudaStream_t s) {
    uint64_t blocks = (args.count + 255) / 256;
    if (blocks > 148ULL * 32) blocks = 148ULL * 32;
    if (blocks == 0) blocks = 1;
    if (single)
        gatherKernel<float2><<<(unsigned) blocks, 256, 0, s>>>((const float2 *) st, args, out);
    else
        gatherKernel<double2><<<(unsigned) blocks, 256, 0, s>>>((const double2 *) st, args, out);
    return cudaGetLastError();
}

}  // namespace dgq

namespace dgq {

// ------------------------------------------------- amplitude upload
// out[i] = (re[i], im[i]) for i < count, zero for count <= i < total.
template <class V>
__global__ void interleaveKernel(const double *__restrict__ re, const double *__restrict__ im, uint64_t count,
                                 uint64_t total, V *__restrict__ out) {
    for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (uint64_t) gridDim.x * blockDim.x) {
        V v;
        v.x = i < count ? re[i] : 0.0;
        v.y = i < count ? im[i] : 0.0;
        out[i] = v;
    }
}

cudaError_t launchInterleave(const double *re, const double *im, uint64_t count, uint64_t total, void *out,
                             bool single, cudaStream_t s) {
    uint64_t blocks = (total + 255) / 256;
    if (blocks > 148ULL * 32) blocks = 148ULL * 32;
    if (single)
        interleaveKernel<float2><<<(unsigned) blocks, 256, 0, s>>>(re, im, count, total, (float2 *) out);
    else
        interleaveKernel<double2><<<(unsigned) blocks, 256, 0, s>>>(re, im, count, total, (double2 *) out);
    return cudaGetLastError();
}

}  // namespace dgq

namespace dgq {

// ------------------------------------------------ FP64 pipe microbenchmark
// Eight independent DFMA chains per thread; the result is written so the
// work cannot be removed. Used to state the FP64 roofline next to HBM.
__global__ void __launch_bounds__(256) fp64PeakKernel(double *out, int iters, double seed) {
    double x0 = seed + threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6,
           x7 = x0 + 7;
    const double m = 0.999999, c = 1e-7;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int u = 0; u < 16; u++) {
            x0 = fma(x0, m, c);
            x1 = fma(x1, m, c);
            x2 = fma(x2, m, c);
            x3 = fma(x3, m, c);
            x4 = fma(x4, m, c);
            x5 = fma(x5, m, c);
            x6 = fma(x6, m, c);
            x7 = fma(x7, m, c);
        }
    }
    out[blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}

cudaError_t launchFp64Peak(double *out, int blocks, int iters, cudaStream_t s) {
    fp64PeakKernel<<<blocks, 256, 0, s>>>(out, iters, 1.0);
    return cudaGetLastError();
}

}  // namespace dgq

namespace dgq {

// ------------------------------------------------------ inner product
// sum over logical indices of conj(bra) * ket, both registers read through
// their own logical->virtual maps and lazy collapses; FP64 accumulation,
// fixed reduction order (partials per CTA, then one finalise CTA).
template <class VB, class VK>
__global__ void __launch_bounds__(256) innerKernel(const VB *__restrict__ bra, const VK *__restrict__ ket,
                                                   const __grid_constant__ InnerArgs args, double2 *partial) {
    double re = 0.0, im = 0.0;
    const uint64_t n = 1ULL << args.numReal;
    for (uint64_t l = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; l < n; l += (uint64_t) gridDim.x * blockDim.x) {
        uint64_t vb = l, vk = l;
        if (!args.identity) {
            vb = 0;
            vk = 0;
            for (int b = 0; b < args.numReal; b++) {
                const uint64_t bit = (l >> b) & 1ULL;
                vb |= bit << args.l2vBra[b];
                vk |= bit << args.l2vKet[b];
            }
        }
        double br = (double) bra[vb].x, bi = (double) bra[vb].y;
        double kr = (double) ket[vk].x, ki = (double) ket[vk].y;
        if (args.braRestrict) {
            const bool keep = (vb & args.braMask) == args.braValue;
            br = keep ? br * args.braScale : 0.0;
            bi = keep ? bi * args.braScale : 0.0;
        }
        if (args.ketRestrict) {
            const bool keep = (vk & args.ketMask) == args.ketValue;
            kr = keep ? kr * args.ketScale : 0.0;
            ki = keep ? ki * args.ketScale : 0.0;
        }
        re += br * kr + bi * ki;
        im += br * ki - bi * kr;
    }
    __shared__ double sre[8], sim[8];
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sre[threadIdx.x >> 5] = re;
        sim[threadIdx.x >> 5] = im;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < 8; w++) {
            a += sre[w];
            b += sim[w];
        }
        partial[blockIdx.x] = make_double2(a, b);
    }
}

__global__ void innerFinalize(const double2 *__restrict__ partial, int n, double2 *out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double a = 0.0, b = 0.0;
    for (int i = 0; i < n; i++) {
        a += partial[i].x;
        b += partial[i].y;
    }
    *out = make_double2(a, b);
}

int innerNumCtas() { return 148 * 8; }

cudaError_t launchInner(const void *bra, bool braSingle, const void *ket, bool ketSingle, const InnerArgs &args,
                        double2 *partial, double2 *out, cudaStream_t s) {
    const int grid = innerNumCtas();
    if (braSingle && ketSingle)
        innerKernel<float2, float2><<<grid, 256, 0, s>>>((const float2 *) bra, (const float2 *) ket, args, partial);
    else if (braSingle)
        innerKernel<float2, double2><<<grid, 256, 0, s>>>((const float2 *) bra, (const double2 *) ket, args, partial);
    else if (ketSingle)
        innerKernel<double2, float2><<<grid, 256, 0, s>>>((const double2 *) bra, (const float2 *) ket, args, partial);
    else
        innerKernel<double2, double2><<<grid, 256, 0, s>>>((const double2 *) bra, (const double2 *) ket, args, partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    innerFinalize<<<1, 32, 0, s>>>(partial, grid, out);
    return cudaGetLastError();
}

}  // namespace dgq
