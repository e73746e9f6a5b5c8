// dense.cu -- one sweep applying a dense 2^K x 2^K unitary on K target bits
// (multiQubitUnitary with more targets than a register phase holds).
//
// A CTA owns a tile of 2^TB amplitudes (TB = min(12, numBits)) spanning the
// K target bits and the TB - K lowest other address bits ("columns"); the
// remaining bits come from blockIdx. The tile is loaded in address order
// (coalesced), laid out in shared memory as X[row][column] (row = matrix
// index over the targets, targs[0] its least significant bit), and Y = U X
// is computed on the FP64 matrix instruction (mma.sync m8n8k4; tcgen05 has
// no FP64 kind), in FP64 for both state precisions.
//
// Bound: FP64 arithmetic, 8 x 2^K flops per amplitude (K = 6: 15.0 ms per
// 2^30 amplitudes at 36.7 TFLOP/s, against 5.2 ms of complex128 HBM
// traffic). The matrix instruction reaches 36.4-37.1 TFLOP/s with 8 warps
// per SM where FMA chains reach 35.0, takes an eighth of the issue slots, and
// its fragments need 6 shared-memory loads for 8192 FMAs. Every warp keeps
// a 32 x 16 complex block of Y (64 accumulator registers); two CTAs per SM,
// so one loads or stores its tile while the other computes. U arrives in
// fragment order (packDenseMatrix) in 8 or 16 KiB chunks, copied from L2
// behind the arithmetic. Measured at 2^26 amplitudes: complex128 K = 5, 6, 7
// 0.81, 1.22, 2.19 ms (21, 28, 31 TFLOP/s), complex64 K = 7 2.06 ms; the
// kernel before it (4 x 4 blocks a thread on FMA instructions, bound by
// shared-memory bank conflicts) took 3.59 ms for complex128 K = 6.
#include <cuda_runtime.h>

#include <cstdint>

#include "interp.cuh"
#include "kernels.h"

namespace dgq {

namespace {

constexpr int kDenseTileBits = 12;
constexpr int kDenseThreads = 256;

// k-steps (4 matrix columns) of U per chunk: 8 KiB at K = 5, else 16 KiB
template <int K>
constexpr int kChunkSteps = K == 7 ? 2 : 4;

// c += a b on 8 x 8 x 4: lane l holds a[l / 4][l % 4], b[l % 4][l / 4] and
// c[l / 4][2 (l % 4) + {0, 1}]
__device__ __forceinline__ void mma8x8x4(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

__device__ __forceinline__ void copyAsync16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// Row pitch of X in elements: 32 bytes more than the columns, so the 4 rows
// x 2 (complex128) or 4 (complex64) columns of a fragment load's phase fall
// in distinct banks.
template <class V>
__host__ __device__ constexpr int densePitch(int G) {
    return G + 32 / (int) sizeof(V);
}

template <class V, int K>
__global__ void __launch_bounds__(kDenseThreads, 2) denseKernel(V *__restrict__ st, const __grid_constant__ DenseArgs a,
                                                               const double2 *__restrict__ U) {
    typedef typename Real<V>::T R;
    constexpr int D = 1 << K;
    constexpr int MB = D / 8;                    // 8-row blocks
    constexpr int CS = kChunkSteps<K>;
    constexpr int CHUNK = CS * MB * 32;          // double2 per chunk
    constexpr int CHUNKS = D / (4 * CS);
    const int TB = a.tileBits;
    const int G = 1 << (TB - K);       // columns in the tile
    const int pitch = densePitch<V>(G);
    extern __shared__ __align__(16) unsigned char smRaw[];
    double2 *Us = reinterpret_cast<double2 *>(smRaw);      // [2][CHUNK]
    V *Xs = reinterpret_cast<V *>(Us + 2 * CHUNK);         // [D][pitch]
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    const uint32_t cta = blockIdx.x;

    auto fetch = [&](int ch) {
        const double2 *src = U + (size_t) ch * CHUNK;
        double2 *dst = Us + (ch & 1) * CHUNK;
#pragma unroll
        for (int e = 0; e < CHUNK / kDenseThreads; e++)
            copyAsync16(dst + e * kDenseThreads + tid, src + e * kDenseThreads + tid);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);

    uint64_t base = 0;
    for (int i = 0; i < a.numBits - TB; i++) base |= (uint64_t) ((cta >> i) & 1u) << a.ctaPos[i];

    // address-ordered tile index i = tid + 256 j -> (address, row, column): the
    // bits of tid and of j are disjoint, so their parts OR together; the 16
    // j parts sit in a table
    __shared__ uint64_t jAddr[16];
    __shared__ uint32_t jAt[16];
    auto part = [&](uint32_t bits, int from, int to, uint64_t &addr, uint32_t &at) {
        uint32_t row = 0, col = 0;
        addr = 0;
        for (int b = from; b < to; b++) {
            if (!((bits >> (b - from)) & 1u)) continue;
            addr |= 1ULL << a.tilePos[b];
            const int r = a.rowBit[b];
            if (r >= 0)
                row |= 1u << r;
            else
                col |= 1u << a.colBit[b];
        }
        at = row * (uint32_t) pitch + col;
    };
    const int tidBits = TB < 8 ? TB : 8;
    const int nj = 1 << (TB - tidBits);
    const bool moves = tid < (1u << tidBits);
    if ((int) tid < nj) {
        uint64_t ad;
        uint32_t at;
        part(tid, tidBits, TB, ad, at);
        jAddr[tid] = ad;
        jAt[tid] = at;
    }
    uint64_t tAddr;
    uint32_t tAt;
    part(tid, 0, tidBits, tAddr, tAt);
    tAddr |= base;
    __syncthreads();

    if (moves) {
        double inScale = 1.0;
        if (a.normIn) inScale = rsqrt(*a.normIn);
        const bool scaled = a.normIn || a.hasRestrict;
        auto put = [&](int j, V v, uint64_t addr) {
            if (scaled) {
                double sc = inScale;
                if (a.hasRestrict) sc = (addr & a.restrictMask) != a.restrictValue ? 0.0 : sc * a.restrictScale;
                v = mk<V>((R) (v.x * (R) sc), (R) (v.y * (R) sc));
            }
            Xs[tAt + jAt[j]] = v;
        };
        if (nj == 16) {  // every load of a full tile in flight at once
            V v[16];
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = st[tAddr | jAddr[j]];
#pragma unroll
            for (int j = 0; j < 16; j++) put(j, v[j], tAddr | jAddr[j]);
        } else {
            for (int j = 0; j < nj; j++) put(j, st[tAddr | jAddr[j]], tAddr | jAddr[j]);
        }
    }

    // the warp's rows [wr, wr + 32) and columns [wc, wc + 16); a tile with
    // fewer columns repeats them and drops the repeats when Y is written
    const uint32_t wr = (warp % (D / 32)) * 32, wc = (warp / (D / 32)) * 16;
    const bool computes = (int) wc < G;
    double yr[4][2][2] = {}, yi[4][2][2] = {};
    for (int ch = 0; ch < CHUNKS; ch++) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // chunk ch (and X) visible; chunk ch - 1 no longer read
        if (ch + 1 < CHUNKS) fetch(ch + 1);
        if (!computes) continue;
        const double2 *u0 = Us + (ch & 1) * CHUNK + (wr / 8) * 32 + lane;
        const V *x0 = Xs + (ch * CS * 4 + (lane & 3u)) * pitch;
#pragma unroll
        for (int ks = 0; ks < CS; ks++) {
            double2 u[4];
            double xr[2], xi[2];
#pragma unroll
            for (int m = 0; m < 4; m++) u[m] = u0[(ks * MB + m) * 32];
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const V x = x0[ks * 4 * pitch + ((wc + n * 8 + (lane >> 2)) & (uint32_t) (G - 1))];
                xr[n] = (double) x.x;
                xi[n] = (double) x.y;
            }
#pragma unroll
            for (int m = 0; m < 4; m++)
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    mma8x8x4(yr[m][n], u[m].x, xr[n]);
                    mma8x8x4(yi[m][n], u[m].x, xi[n]);
                }
#pragma unroll
            for (int m = 0; m < 4; m++)
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    mma8x8x4(yr[m][n], -u[m].y, xi[n]);
                    mma8x8x4(yi[m][n], u[m].y, xr[n]);
                }
        }
    }
    __syncthreads();  // every read of X is done
    if (computes) {
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const uint32_t row = wr + m * 8 + (lane >> 2), col = wc + n * 8 + (lane & 3u) * 2 + e;
                    if ((int) col < G) Xs[row * pitch + col] = mk<V>((R) yr[m][n][e], (R) yi[m][n][e]);
                }
    }
    __syncthreads();
    double norm = 0.0;
    if (moves) {
#pragma unroll 4
        for (int j = 0; j < nj; j++) {
            const V y = Xs[tAt + jAt[j]];
            st[tAddr | jAddr[j]] = y;
            norm += (double) y.x * (double) y.x + (double) y.y * (double) y.y;
        }
    }
    if (a.normOut) {
        __shared__ double red[kDenseThreads / 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) norm += __shfl_xor_sync(0xffffffffu, norm, o);
        if (lane == 0) red[warp] = norm;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < kDenseThreads / 32; w++) t += red[w];
            atomicAdd(a.normOut, t);
        }
    }
}

template <class V, int K>
constexpr size_t denseSmem(int tileBits) {
    return sizeof(double2) * 2 * kChunkSteps<K> * (1u << K) * 4 +
           sizeof(V) * (size_t) (1 << K) * densePitch<V>(1 << (tileBits - K));
}

template <class V, int K>
cudaError_t launchDenseVK(V *st, const DenseArgs &a, const double *U, cudaStream_t s) {
    static std::atomic<uint64_t> optIn{0};
    cudaError_t e =
        ensureSmemOptIn((const void *) denseKernel<V, K>, (int) denseSmem<V, K>(kDenseTileBits), optIn);
    if (e != cudaSuccess) return e;
    const unsigned grid = 1u << (a.numBits - a.tileBits);
    denseKernel<V, K><<<grid, kDenseThreads, denseSmem<V, K>(a.tileBits), s>>>(st, a, (const double2 *) U);
    return cudaGetLastError();
}

template <class V>
cudaError_t launchDenseV(V *st, int K, const DenseArgs &a, const double *U, cudaStream_t s) {
    switch (K) {
        case 5: return launchDenseVK<V, 5>(st, a, U, s);
        case 6: return launchDenseVK<V, 6>(st, a, U, s);
        case 7: return launchDenseVK<V, 7>(st, a, U, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// Fragment order: k-step by k-step (4 columns), 8-row block by block, the 32
// lanes' values of one A fragment in a row.
void packDenseMatrix(int K, const double *U, double *out) {
    const int D = 1 << K;
    for (int ks = 0; ks < D / 4; ks++)
        for (int mb = 0; mb < D / 8; mb++)
            for (int l = 0; l < 32; l++) {
                const double *u = U + 2 * ((size_t) (mb * 8 + l / 4) * D + (size_t) (ks * 4 + l % 4));
                *out++ = u[0];
                *out++ = u[1];
            }
}

bool denseArgs(int numBits, int K, const uint8_t *targets, DenseArgs &a) {
    if (K < kMinDenseTargets || K > kMaxDenseTargets) return false;
    const int TB = numBits < kDenseTileBits ? numBits : kDenseTileBits;
    if (TB - K < 2) return false;
    a = DenseArgs();
    a.numBits = numBits;
    a.tileBits = TB;
    uint64_t tmask = 0;
    for (int i = 0; i < K; i++) tmask |= 1ULL << targets[i];
    // columns: the lowest non-target bits
    int cols = 0;
    uint64_t cmask = 0;
    for (int b = 0; b < numBits && cols < TB - K; b++)
        if (!((tmask >> b) & 1ULL)) {
            cmask |= 1ULL << b;
            cols++;
        }
    const uint64_t tile = tmask | cmask;
    int nt = 0, nc = 0, colRank = 0;
    for (int b = 0; b < numBits; b++) {
        if ((tile >> b) & 1ULL) {
            a.tilePos[nt] = (uint8_t) b;
            a.rowBit[nt] = -1;
            a.colBit[nt] = -1;
            if ((tmask >> b) & 1ULL) {
                for (int i = 0; i < K; i++)
                    if (targets[i] == b) a.rowBit[nt] = (int8_t) i;
            } else {
                a.colBit[nt] = (int8_t) colRank++;
            }
            nt++;
        } else {
            a.ctaPos[nc++] = (uint8_t) b;
        }
    }
    return nt == TB;
}

cudaError_t launchDense(void *st, bool single, int K, const DenseArgs &a, const double *U, cudaStream_t s) {
    return single ? launchDenseV((float2 *) st, K, a, U, s) : launchDenseV((double2 *) st, K, a, U, s);
}

}  // namespace dgq
