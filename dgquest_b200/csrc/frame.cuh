// frame.cuh -- the register phases of framed programs (frame.h) on the 16
// amplitudes a thread holds. Shared by the single-register tile kernel
// (kernels.cu) and the batched persistent kernel (batch.cu).
#pragma once

#include <cuda_runtime.h>

#include "frame.h"
#include "interp.cuh"

namespace dgq {

__device__ __forceinline__ double signFlip(double x, uint32_t bit31) {
    return __hiloint2double(__double2hiint(x) ^ (int) bit31, __double2loint(x));
}
__device__ __forceinline__ float signFlip(float x, uint32_t bit31) {
    return __uint_as_float(__float_as_uint(x) ^ bit31);
}

// The lower register of each pair (j, j ^ D), in order.
template <int D, class F>
__device__ __forceinline__ void forDirection(F f) {
#pragma unroll
    for (int j = 0; j < kRegs; j++)
        if ((j ^ D) > j) f(j, j ^ D);
}

template <int D, class V>
__device__ __forceinline__ void framePair(int kind, V (&a)[kRegs], typename Real<V>::T c0, typename Real<V>::T c1,
                                          uint32_t tab) {
    typedef typename Real<V>::T R;
    if (kind == FK_RY) {
        forDirection<D>([&](int j, int k) {
            const R t = signFlip(c0, (tab << (31 - j)) & 0x80000000u);
            const V x = a[j], y = a[k];
            a[j] = mk<V>(fma(-t, y.x, x.x), fma(-t, y.y, x.y));
            a[k] = mk<V>(fma(t, x.x, y.x), fma(t, x.y, y.y));
        });
    } else if (kind == FK_RX) {
        forDirection<D>([&](int j, int k) {
            const V x = a[j], y = a[k];
            a[j] = mk<V>(fma(c0, y.y, x.x), fma(-c0, y.x, x.y));
            a[k] = mk<V>(fma(c0, x.y, y.x), fma(-c0, x.x, y.y));
        });
    } else {
        forDirection<D>([&](int j, int k) {
            const R p = signFlip(c0, (tab << (31 - j)) & 0x80000000u);
            const V x = a[j], y = a[k];
            a[j] = mk<V>(fma(p, y.x, fma(-c1, y.y, x.x)), fma(p, y.y, fma(c1, y.x, x.y)));
            a[k] = mk<V>(fma(-p, x.x, fma(-c1, x.y, y.x)), fma(-p, x.y, fma(c1, x.x, y.y)));
        });
    }
}

template <int D, class V>
__device__ __forceinline__ void framePhase(V (&a)[kRegs], typename Real<V>::T c, typename Real<V>::T s) {
#pragma unroll
    for (int j = 0; j < kRegs; j++)
        if (__builtin_popcount(j & D) & 1) a[j] = mk<V>(c * a[j].x - s * a[j].y, c * a[j].y + s * a[j].x);
}

template <int D, class V>
__device__ __forceinline__ void frameNegate(V (&a)[kRegs]) {
#pragma unroll
    for (int j = 0; j < kRegs; j++)
        if (__builtin_popcount(j & D) & 1) a[j] = mk<V>(-a[j].x, -a[j].y);
}

// bit j: parity of j & r
__device__ __forceinline__ uint32_t parityTable(uint32_t r) {
    return ((r & 1u) ? 0xAAAAu : 0u) ^ ((r & 2u) ? 0xCCCCu : 0u) ^ ((r & 4u) ? 0xF0F0u : 0u) ^ ((r & 8u) ? 0xFF00u : 0u);
}

#define DGQ_FRAME_CASES(KIND, CALL)                                                                              \
    case KIND << 4 | 1: { constexpr int D = 1; CALL; } break;                                                    \
    case KIND << 4 | 2: { constexpr int D = 2; CALL; } break;                                                    \
    case KIND << 4 | 3: { constexpr int D = 3; CALL; } break;                                                    \
    case KIND << 4 | 4: { constexpr int D = 4; CALL; } break;                                                    \
    case KIND << 4 | 5: { constexpr int D = 5; CALL; } break;                                                    \
    case KIND << 4 | 6: { constexpr int D = 6; CALL; } break;                                                    \
    case KIND << 4 | 7: { constexpr int D = 7; CALL; } break;                                                    \
    case KIND << 4 | 8: { constexpr int D = 8; CALL; } break;                                                    \
    case KIND << 4 | 9: { constexpr int D = 9; CALL; } break;                                                    \
    case KIND << 4 | 10: { constexpr int D = 10; CALL; } break;                                                  \
    case KIND << 4 | 11: { constexpr int D = 11; CALL; } break;                                                  \
    case KIND << 4 | 12: { constexpr int D = 12; CALL; } break;                                                  \
    case KIND << 4 | 13: { constexpr int D = 13; CALL; } break;                                                  \
    case KIND << 4 | 14: { constexpr int D = 14; CALL; } break;                                                  \
    case KIND << 4 | 15: { constexpr int D = 15; CALL; } break;

// The phases of one sweep on the tile in sm (swizzled tile-local order, all
// stores before the call synchronised). fetchOp(o) / fetchCoef(o) read the
// program; cta holds the tile's index bits; sync() is a barrier of the
// tile's threads.
template <class V, int W, class FetchPhase, class FetchOp, class FetchCoef, class Sync>
__device__ __forceinline__ void framePhases(int numPhases, const FrameTail &tail, V *sm, uint32_t tid, uint32_t cta,
                                            FetchPhase phaseAt, FetchOp fetchOp, FetchCoef fetchCoef, Sync sync) {
    typedef typename Real<V>::T R;
    V a[kRegs];
    for (int p = 0; p < numPhases; p++) {
        const FPhase &ph = phaseAt(p);
        uint32_t loc = 0;
#pragma unroll
        for (int i = 0; i < W - kRegBits; i++) loc |= ((tid >> i) & 1u) << ph.thrPos[i];
        uint32_t sb = loc ^ (((loc >> 3) ^ (loc >> 6) ^ (loc >> 9) ^ (loc >> 12)) & 7u);  // tileSwizzle
#pragma unroll
        for (int j = 0; j < kRegs; j++) a[j] = sm[sb ^ ph.rdOff[j]];
        // one number for the thread's 16 amplitudes
        const bool start = p == tail.globalPhase;
        double ar = start ? tail.globalRe : 1.0, ai = start ? tail.globalIm : 0.0;
        const int se = ph.scalarEnd, e = ph.opEnd;
        uint32_t where = 0xFFFFu;  // registers left by FK_AND and FK_IF
        for (int o = ph.opBegin; o < se; o++) {
            const FOp op = fetchOp(o);
            const double2 c = fetchCoef(o);
            if ((loc & op.lm) == op.lm && (cta & op.cm) == op.cm) {
                const double r = c.x * ar - c.y * ai;
                ai = c.x * ai + c.y * ar;
                ar = r;
            }
        }
        for (int o = se; o < e; o++) {
            const FOp op = fetchOp(o);
            const double2 c = fetchCoef(o);
            uint32_t thr = (uint32_t) (__popc(loc & op.lm) + __popc(cta & op.cm)) << 31;
            if (op.code < FK_PH << 4) {
                R c0 = (R) c.x;
                const R c1 = (R) c.y;
                const uint32_t tab = op.tab;
                if (op.code < FK_RX << 4 || op.code >= FK_RN << 4) c0 = signFlip(c0, thr);
                switch (op.code) {
                    DGQ_FRAME_CASES(FK_RY, (framePair<D>(FK_RY, a, c0, c1, tab)))
                    DGQ_FRAME_CASES(FK_RX, (framePair<D>(FK_RX, a, c0, c1, tab)))
                    DGQ_FRAME_CASES(FK_RN, (framePair<D>(FK_RN, a, c0, c1, tab)))
                }
            } else if (op.code < FK_PH2 << 4) {
                if ((loc & op.lm2) != op.lm2 || (cta & op.cm2) != op.cm2) continue;
                double cs = c.x, sn = c.y;
                if (thr) {
                    // the other half of the registers: the phase on all of
                    // them, its inverse on these
                    const double r = cs * ar - sn * ai;
                    ai = cs * ai + sn * ar;
                    ar = r;
                    sn = -sn;
                }
                const R rc = (R) cs, rs = (R) sn;
                switch (op.code) {
                    DGQ_FRAME_CASES(FK_PH, (framePhase<D>(a, rc, rs)))
                    DGQ_FRAME_CASES(FK_NEG, (frameNegate<D>(a)))
                }
            } else {
                if (op.code == FK_IF << 4) {
                    if ((loc & op.lm) != op.lm || (cta & op.cm) != op.cm) where = 0u;
                    continue;
                }
                uint32_t m = where & (parityTable(op.rr & 15u) ^ ((op.tab & 1u) ? 0xFFFFu : 0u) ^ (thr ? 0xFFFFu : 0u));
                const uint32_t thr2 = (uint32_t) (__popc(loc & op.lm2) + __popc(cta & op.cm2)) & 1u;
                m &= parityTable(op.rr >> 4) ^ ((op.tab & 2u) ? 0xFFFFu : 0u) ^ (thr2 ? 0xFFFFu : 0u);
                where = op.code == FK_AND << 4 ? m : 0xFFFFu;
                if (op.code == FK_AND << 4) continue;
                if (op.code == FK_NEG2 << 4) {
#pragma unroll
                    for (int j = 0; j < kRegs; j++) {
                        const uint32_t s = (m << (31 - j)) & 0x80000000u;
                        a[j] = mk<V>(signFlip(a[j].x, s), signFlip(a[j].y, s));
                    }
                } else {
                    const R rc = (R) c.x, rs = (R) c.y;
#pragma unroll
                    for (int j = 0; j < kRegs; j++)
                        if ((m >> j) & 1u) a[j] = mk<V>(rc * a[j].x - rs * a[j].y, rc * a[j].y + rs * a[j].x);
                }
            }
        }
        if (ph.fold) {
            const R r = (R) ar, i = (R) ai;
#pragma unroll
            for (int j = 0; j < kRegs; j++) a[j] = mk<V>(r * a[j].x - i * a[j].y, r * a[j].y + i * a[j].x);
        }
        if (ph.hasD) {
#pragma unroll
            for (int b = 0; b < kRegBits; b++)
                if ((__popc(loc & ph.dl[b]) + __popc(cta & ph.dc[b])) & 1) sb ^= ph.col[b];
        }
        // M and D permute the thread's own 16 slots
#pragma unroll
        for (int j = 0; j < kRegs; j++) sm[sb ^ ph.wrOff[j]] = a[j];
        sync();
    }
}

// The global factor (times scale) and the sign on the amplitudes in store
// order; hasScale: scale != 1.
template <class V>
__device__ __forceinline__ void frameFinish(const FrameTail &tail, V (&a)[kRegs], uint32_t tid, uint32_t cta,
                                            bool hasScale, double scale) {
    typedef typename Real<V>::T R;
    if (hasScale || (tail.hasGlobal && tail.globalPhase < 0)) {
        const bool here = tail.globalPhase < 0;
        const R gr = (R) (here ? tail.globalRe * scale : scale), gi = (R) (here ? tail.globalIm * scale : 0.0);
#pragma unroll
        for (int j = 0; j < kRegs; j++) a[j] = mk<V>(gr * a[j].x - gi * a[j].y, gr * a[j].y + gi * a[j].x);
    }
    if (tail.hasSign) {
        uint32_t m = tail.signTab;
        if ((__popc(tid & tail.signThr) + __popc(cta & tail.signCta)) & 1) m = ~m;
#pragma unroll
        for (int j = 0; j < kRegs; j++) {
            const uint32_t s = (m << (31 - j)) & 0x80000000u;
            a[j] = mk<V>(signFlip(a[j].x, s), signFlip(a[j].y, s));
        }
    }
}

}  // namespace dgq
