// frame.cpp -- see frame.h.
#include "frame.h"

#include <cmath>
#include <cstring>

namespace dgq {

namespace {

int parity(uint32_t x) { return __builtin_parity(x); }

// bit j: parity of j & r
uint32_t parityTable(uint32_t r) {
    return ((r & 1u) ? 0xAAAAu : 0u) ^ ((r & 2u) ? 0xCCCCu : 0u) ^ ((r & 4u) ? 0xF0F0u : 0u) ^ ((r & 8u) ? 0xFF00u : 0u);
}

struct Framer {
    const TileProgram &p;
    FrameSweep &out;
    const KPhase *ph = nullptr;
    // register bits: value = row . j + dl . loc + dc . cta + cc
    uint8_t row[kRegBits], col[kRegBits];  // M and its inverse, whose column q is the direction of a pair on bit q
    uint16_t dl[kRegBits];
    uint32_t dc[kRegBits];
    uint8_t cc[kRegBits];
    // sign: zr . j + zl . loc + zc . cta (its constant is in the global factor)
    uint32_t zr = 0, zl = 0, zc = 0;
    long double gRe, gIm;  // one rounding per sweep: an error here is the same for every amplitude
    bool fold = false;
    std::vector<FOp> scalars, rest;
    std::vector<double> scalarCoef, restCoef;

    Framer(const TileProgram &prog, FrameSweep &o) : p(prog), out(o), gRe(prog.globalRe), gIm(prog.globalIm) {}

    void global(long double re, long double im) {
        const long double r = gRe * re - gIm * im, i = gRe * im + gIm * re;
        gRe = r;
        gIm = i;
    }
    void negateGlobal() {
        gRe = -gRe;
        gIm = -gIm;
    }
    void signBy(int q) {
        zr ^= row[q];
        zl ^= dl[q];
        zc ^= dc[q];
        if (cc[q]) negateGlobal();
    }
    void put(const FOp &op, double a, double b) {
        rest.push_back(op);
        restCoef.push_back(a);
        restCoef.push_back(b);
    }
    void scalar(uint32_t condLoc, uint32_t condCta, double c, double s) {
        if (!condLoc && !condCta) {
            global(c, s);
            return;
        }
        FOp op;
        std::memset(&op, 0, sizeof(op));
        op.lm = (uint16_t) condLoc;
        op.cm = condCta;
        scalars.push_back(op);
        scalarCoef.push_back(c);
        scalarCoef.push_back(s);
        fold = true;
    }
    // phase c + i s (neg: -1) where every register bit of regs and every
    // thread and CTA bit of the masks is 1
    bool diagonal(uint32_t regs, uint32_t condLoc, uint32_t condCta, double c, double s, bool neg) {
        const int n = __builtin_popcount(regs);
        if (neg && n + __builtin_popcount(condLoc) + __builtin_popcount(condCta) == 1) {
            // Z: part of the sign
            if (n)
                signBy(__builtin_ctz(regs));
            else
                zl ^= condLoc, zc ^= condCta;
            return true;
        }
        if (n == 0) {
            scalar(condLoc, condCta, c, s);
            return true;
        }
        FOp op;
        std::memset(&op, 0, sizeof(op));
        if (n == 1) {
            const int q = __builtin_ctz(regs);
            if (cc[q]) {
                // on the other half: the phase everywhere, its inverse on this half
                scalar(condLoc, condCta, c, s);
                s = -s;
            }
            op.code = (uint8_t) ((neg ? FK_NEG : FK_PH) << 4 | row[q]);
            op.lm = dl[q];
            op.cm = dc[q];
            op.lm2 = (uint16_t) condLoc;
            op.cm2 = condCta;
            fold = fold || op.lm || op.cm;
            put(op, c, s);
            return true;
        }
        if (condLoc || condCta) {
            op.code = (uint8_t) (FK_IF << 4);
            op.lm = (uint16_t) condLoc;
            op.cm = condCta;
            put(op, 0.0, 0.0);
        }
        // two register bits at a time, the last two with the phase
        uint32_t left = regs;
        while (left) {
            const int k = __builtin_popcount(left);
            const int a = __builtin_ctz(left), b = k == 3 ? -1 : __builtin_ctz(left & (left - 1));
            std::memset(&op, 0, sizeof(op));
            op.code = (uint8_t) ((k > 2 ? FK_AND : neg ? FK_NEG2 : FK_PH2) << 4);
            op.rr = row[a];
            op.tab = cc[a];
            op.lm = dl[a];
            op.cm = dc[a];
            if (b < 0) {
                op.tab |= 2;  // always 1
            } else {
                op.rr |= (uint8_t) (row[b] << 4);
                op.tab |= (uint16_t) (cc[b] << 1);
                op.lm2 = dl[b];
                op.cm2 = dc[b];
                left &= left - 1;
            }
            left &= left - 1;
            put(op, c, s);
        }
        return true;
    }
    // rotation on register bit q; (a, b) its coefficients
    void pair(int kind, int q, double a, double b) {
        const int v = col[q];
        FOp op;
        std::memset(&op, 0, sizeof(op));
        op.code = (uint8_t) (kind << 4 | v);
        if (kind != FK_RX) {
            // Rx is the same both ways round
            op.tab = (uint16_t) (parityTable(row[q]) ^ (cc[q] ? 0xFFFFu : 0u));
            op.lm = dl[q];
            op.cm = dc[q];
        }
        // partners of opposite sign see each other negated
        const bool flip = parity(zr & v);
        put(op, flip ? -a : a, flip ? -b : b);
    }

    // U = [[m0, m1], [m2, m3]] (complex) on register bit q, without controls:
    // with |m0| >= |m1| (else U X X), U = m0 diag(1, e) [[1, p], [-conj(p), 1]],
    // e = m3 / m0, p = m1 / m0; 96 FP64 instructions a thread instead of 128
    bool general(int q, const double *u) {
        double m[8];
        std::memcpy(m, u, sizeof(m));
        if (m[0] * m[0] + m[1] * m[1] < m[2] * m[2] + m[3] * m[3]) {
            for (int i = 0; i < 8; i++) m[i] = u[i ^ 2];
            cc[q] ^= 1;
        }
        const double d = m[0] * m[0] + m[1] * m[1];
        if (!(d > 0.0)) return false;
        auto over = [&](const double *x, double *y) {
            y[0] = (x[0] * m[0] + x[1] * m[1]) / d;
            y[1] = (x[1] * m[0] - x[0] * m[1]) / d;
        };
        double e[2], pp[2], l[2];
        over(m + 6, e);
        over(m + 2, pp);
        over(m + 4, l);
        // U must be unitary to rounding: |e| = 1 and m2 / m0 = -e conj(p), whose
        // residuals are dropped. Of 20000 random unitaries rounded to doubles
        // none has more than 1.9e-15 (2 % more than 9e-16), of products of two
        // one in 2000 more than 2e-15; matrices further off run as given.
        const double tol = 2e-15;
        if (std::fabs(e[0] * e[0] + e[1] * e[1] - 1.0) > tol || std::fabs(l[0] + e[0] * pp[0] + e[1] * pp[1]) > tol ||
            std::fabs(l[1] + e[1] * pp[0] - e[0] * pp[1]) > tol)
            return false;
        global(m[0], m[1]);
        pair(FK_RN, q, pp[0], pp[1]);
        return diagonal(1u << q, 0, 0, e[0], e[1], false);
    }

    bool op(const KOp &k) {
        const double *c = p.coef + k.coef;
        const int n = __builtin_popcount(k.ctrlReg) + __builtin_popcount(k.ctrlLoc) + __builtin_popcount(k.ctrlCta);
        switch (k.kind) {
            case KOP_X: {
                const int q = k.k;
                if (n > 1) return false;
                if (n == 0) {
                    cc[q] ^= 1;
                } else if (k.ctrlReg) {
                    const int s = __builtin_ctz(k.ctrlReg);
                    row[q] ^= row[s];
                    col[s] ^= col[q];
                    dl[q] ^= dl[s];
                    dc[q] ^= dc[s];
                    cc[q] ^= cc[s];
                } else {
                    dl[q] ^= k.ctrlLoc;
                    dc[q] ^= k.ctrlCta;
                }
                return true;
            }
            case KOP_Y:
            case KOP_YC:
                // +-i X Z
                if (n) return false;
                signBy(k.k);
                cc[k.k] ^= 1;
                global(0.0, k.kind == KOP_Y ? 1.0 : -1.0);
                return true;
            case KOP_NEG: return diagonal(k.ctrlReg, k.ctrlLoc, k.ctrlCta, -1.0, 0.0, true);
            case KOP_MULI: return diagonal(k.ctrlReg, k.ctrlLoc, k.ctrlCta, 0.0, 1.0, false);
            case KOP_MULNI: return diagonal(k.ctrlReg, k.ctrlLoc, k.ctrlCta, 0.0, -1.0, false);
            case KOP_PH: return diagonal(k.ctrlReg, k.ctrlLoc, k.ctrlCta, c[0], c[1], false);
            case KOP_PH1:
            case KOP_Z2: {
                const bool reg = k.kind == KOP_PH1 ? k.code != KC_PH1T : k.code < KC_Z2T;
                const uint32_t r = k.ctrlReg | (reg ? 1u << k.k : 0u), l = k.ctrlLoc | (reg ? 0u : k.selLoc),
                               t = k.ctrlCta | (!reg && k.selCta >= 0 ? 1u << k.selCta : 0u);
                if (k.kind == KOP_PH1) return diagonal(r, l, t, c[0], c[1], false);
                // diag(e^-ia, e^ia) = e^-ia diag(1, e^2ia)
                return diagonal(k.ctrlReg, k.ctrlLoc, k.ctrlCta, c[0], -c[1], false) &&
                       diagonal(r, l, t, (c[0] - c[1]) * (c[0] + c[1]), 2.0 * c[0] * c[1], false);
            }
            case KOP_RY1: pair(FK_RY, k.k, c[0], 0.0); return true;
            case KOP_RY2:
                // [[u, -1], [1, u]] = [[1, u], [-u, 1]] X Z
                signBy(k.k);
                cc[k.k] ^= 1;
                pair(FK_RY, k.k, -c[0], 0.0);
                return true;
            case KOP_H1:
                // [[1, 1], [1, -1]] = [[1, -1], [1, 1]] Z
                signBy(k.k);
                pair(FK_RY, k.k, 1.0, 0.0);
                return true;
            case KOP_RX1: pair(FK_RX, k.k, c[0], 0.0); return true;
            case KOP_RX2:
                // [[u, -i], [-i, u]] = -i [[1, i u], [i u, 1]] X
                cc[k.k] ^= 1;
                global(0.0, -1.0);
                pair(FK_RX, k.k, -c[0], 0.0);
                return true;
            case KOP_RN1: pair(FK_RN, k.k, c[0], c[1]); return true;
            case KOP_M2C: return !n && general(k.k, c);
            case KOP_M2R: {
                const double m[8] = {c[0], 0.0, c[1], 0.0, c[2], 0.0, c[3], 0.0};
                return !n && general(k.k, m);
            }
            case KOP_M2I: {
                const double m[8] = {c[0], 0.0, 0.0, c[1], 0.0, c[2], c[3], 0.0};
                return !n && general(k.k, m);
            }
            default: return false;
        }
    }

    bool phase(const KPhase &kp, int W, uint32_t &signLoc) {
        ph = &kp;
        uint32_t regMask = 0;
        zr = 0;
        for (int b = 0; b < kRegBits; b++) {
            row[b] = col[b] = (uint8_t) (1u << b);
            dl[b] = 0;
            dc[b] = 0;
            cc[b] = 0;
            regMask |= 1u << kp.regPos[b];
            if ((signLoc >> kp.regPos[b]) & 1u) zr |= 1u << b;
        }
        zl = signLoc & ~regMask;
        fold = false;
        scalars.clear();
        scalarCoef.clear();
        rest.clear();
        restCoef.clear();
        for (int o = kp.opBegin; o < kp.opEnd; o++)
            if (!op(p.ops[o])) return false;
        FPhase f;
        std::memset(&f, 0, sizeof(f));
        for (int i = 0; i < W - kRegBits; i++) f.thrPos[i] = kp.thrPos[i];
        uint32_t table[kRegBits];
        for (int b = 0; b < kRegBits; b++) table[b] = parityTable(row[b]) ^ (cc[b] ? 0xFFFFu : 0u);
        for (int j = 0; j < kRegs; j++) {
            f.rdOff[j] = kp.regOff[j];
            uint32_t loc = 0;
            for (int b = 0; b < kRegBits; b++) loc |= ((table[b] >> j) & 1u) << kp.regPos[b];
            f.wrOff[j] = (uint16_t) tileSwizzle(loc);
        }
        for (int b = 0; b < kRegBits; b++) {
            f.dl[b] = dl[b];
            f.dc[b] = dc[b];
            f.col[b] = (uint16_t) tileSwizzle(1u << kp.regPos[b]);
            if (dl[b] || dc[b]) f.hasD = 1;
        }
        f.fold = fold;
        f.opBegin = (uint16_t) out.ops.size();
        out.ops.insert(out.ops.end(), scalars.begin(), scalars.end());
        out.coef.insert(out.coef.end(), scalarCoef.begin(), scalarCoef.end());
        f.scalarEnd = (uint16_t) out.ops.size();
        out.ops.insert(out.ops.end(), rest.begin(), rest.end());
        out.coef.insert(out.coef.end(), restCoef.begin(), restCoef.end());
        f.opEnd = (uint16_t) out.ops.size();
        out.phases.push_back(f);
        // the sign in index bits: zr . j = m . (M j)
        uint32_t m = 0;
        for (int b = 0; b < kRegBits; b++) m |= (uint32_t) parity(zr & col[b]) << b;
        signLoc = zl;
        for (int b = 0; b < kRegBits; b++)
            if ((m >> b) & 1u) {
                signLoc ^= (1u << kp.regPos[b]) ^ dl[b];
                zc ^= dc[b];
                if (cc[b]) negateGlobal();
            }
        return true;
    }
};

}  // namespace

bool frameProgram(const TileProgram &p, int W, FrameSweep &out) {
    out.phases.clear();
    out.ops.clear();
    out.coef.clear();
    if (p.paired || p.denseK || W > kMaxTileBitsF64 || p.numBits - W > 32) return false;
    out.phases.reserve((size_t) p.numPhases);
    out.ops.reserve((size_t) p.numOps + 16);
    out.coef.reserve(2 * (size_t) p.numOps + 32);
    Framer f(p, out);
    uint32_t signLoc = 0;
    for (int i = 0; i < p.numPhases; i++)
        if (!f.phase(p.phases[i], W, signLoc)) return false;
    if (out.ops.size() > (size_t) kFrameMaxOps) return false;
    FrameTail &t = out.tail;
    std::memset(&t, 0, sizeof(t));
    t.globalRe = (double) f.gRe;
    t.globalIm = (double) f.gIm;
    t.hasGlobal = t.globalRe != 1.0 || t.globalIm != 0.0;
    t.globalPhase = -1;
    for (size_t i = 0; i < out.phases.size() && t.globalPhase < 0; i++)
        if (out.phases[i].fold) t.globalPhase = (int32_t) i;
    t.signCta = f.zc;
    t.signThr = (uint16_t) (signLoc & ((1u << (W - kRegBits)) - 1u));
    for (int j = 0; j < kRegs; j++) t.signTab |= (uint16_t) (parity((signLoc >> (W - kRegBits)) & j) << j);
    t.hasSign = t.signCta || t.signThr || t.signTab;
    return true;
}

// ------------------------------------------------------------ host emulation
void applyFramedHost(const TileProgram &p, const FrameSweep &f, int W, double *state) {
    const uint32_t T = 1u << (W - kRegBits), size = 1u << W;
    std::vector<double> sm(2 * (size_t) size);
    auto address = [&](uint32_t cta, uint32_t local) {
        uint64_t g = local & 31u;
        for (int i = 0; i < W - kCoalescedBits; i++) g |= (uint64_t) ((local >> (kCoalescedBits + i)) & 1u) << p.highPos[i];
        for (int i = 0; i < p.numBits - W; i++) g |= (uint64_t) ((cta >> i) & 1u) << p.ctaPos[i];
        return g;
    };
    auto mul = [](double *x, double c, double s) {
        const double r = c * x[0] - s * x[1], i = c * x[1] + s * x[0];
        x[0] = r;
        x[1] = i;
    };
    for (uint32_t cta = 0; cta < 1u << (p.numBits - W); cta++) {
        for (uint32_t l = 0; l < size; l++) {
            double *d = &sm[2 * tileSwizzle(l)];
            const uint64_t g = address(cta, l);
            d[0] = state[2 * g];
            d[1] = state[2 * g + 1];
            if (p.initKind != INIT_NONE) {
                d[0] = p.initKind == INIT_CLASSICAL ? (g == p.initIndex ? 1.0 : 0.0)
                       : p.initKind == INIT_PLUS    ? (!(g >> p.numReal) ? p.initAmp : 0.0)
                                                    : 0.0;
                d[1] = 0.0;
            }
            if (p.hasRestrict) mul(d, (g & p.restrictMask) == p.restrictValue ? p.restrictScale : 0.0, 0.0);
        }
        for (const FPhase &ph : f.phases) {
            std::vector<double> next(2 * (size_t) size);
            for (uint32_t tid = 0; tid < T; tid++) {
                uint32_t loc = 0;
                for (int i = 0; i < W - kRegBits; i++) loc |= ((tid >> i) & 1u) << ph.thrPos[i];
                const uint32_t sb = tileSwizzle(loc);
                double a[kRegs][2], acc[2] = {1.0, 0.0};
                uint32_t where = 0xFFFFu;  // registers left by FK_AND and FK_IF
                if (f.tail.globalPhase >= 0 && &ph == &f.phases[(size_t) f.tail.globalPhase]) {
                    acc[0] = f.tail.globalRe;
                    acc[1] = f.tail.globalIm;
                }
                for (int j = 0; j < kRegs; j++) std::memcpy(a[j], &sm[2 * (sb ^ ph.rdOff[j])], 16);
                for (int o = ph.opBegin; o < ph.opEnd; o++) {
                    const FOp &op = f.ops[(size_t) o];
                    const double c0 = f.coef[2 * (size_t) o], c1 = f.coef[2 * (size_t) o + 1];
                    if (o < ph.scalarEnd) {
                        if ((loc & op.lm) == op.lm && (cta & op.cm) == op.cm) mul(acc, c0, c1);
                        continue;
                    }
                    const int kind = op.code >> 4, v = op.code & 15;
                    const int thr = parity(loc & op.lm) ^ parity(cta & op.cm);
                    if (kind <= FK_RN) {
                        for (int j = 0; j < kRegs; j++) {
                            if ((j ^ v) < j) continue;
                            double *x = a[j], *y = a[j ^ v], nx[2], ny[2];
                            const double sg = (((op.tab >> j) & 1) ^ thr) ? -1.0 : 1.0;
                            const double pr = kind == FK_RY ? -sg * c0 : kind == FK_RX ? 0.0 : sg * c0;
                            const double pi = kind == FK_RY ? 0.0 : kind == FK_RX ? -c0 : c1;
                            nx[0] = x[0] + pr * y[0] - pi * y[1];
                            nx[1] = x[1] + pr * y[1] + pi * y[0];
                            ny[0] = y[0] - pr * x[0] - pi * x[1];
                            ny[1] = y[1] - pr * x[1] + pi * x[0];
                            std::memcpy(x, nx, 16);
                            std::memcpy(y, ny, 16);
                        }
                    } else if (kind <= FK_NEG) {
                        if ((loc & op.lm2) != op.lm2 || (cta & op.cm2) != op.cm2) continue;
                        for (int j = 0; j < kRegs; j++)
                            if (parity(j & v) ^ thr) mul(a[j], c0, c1);
                    } else if (kind == FK_IF) {
                        if ((loc & op.lm) != op.lm || (cta & op.cm) != op.cm) where = 0;
                    } else {
                        const int thr2 = parity(loc & op.lm2) ^ parity(cta & op.cm2);
                        for (int j = 0; j < kRegs; j++)
                            if (!((parity(j & (op.rr & 15)) ^ thr ^ (op.tab & 1)) &
                                  (parity(j & (op.rr >> 4)) ^ thr2 ^ ((op.tab >> 1) & 1))))
                                where &= ~(1u << j);
                        if (kind == FK_AND) continue;
                        for (int j = 0; j < kRegs; j++)
                            if ((where >> j) & 1u) mul(a[j], c0, c1);
                        where = 0xFFFFu;
                    }
                }
                uint32_t wb = sb;
                for (int b = 0; b < kRegBits; b++)
                    if (parity(loc & ph.dl[b]) ^ parity(cta & ph.dc[b])) wb ^= ph.col[b];
                for (int j = 0; j < kRegs; j++) {
                    if (ph.fold) mul(a[j], acc[0], acc[1]);
                    std::memcpy(&next[2 * (wb ^ ph.wrOff[j])], a[j], 16);
                }
            }
            sm.swap(next);
        }
        for (uint32_t tid = 0; tid < T; tid++)
            for (int j = 0; j < kRegs; j++) {
                const uint32_t l = tid + T * (uint32_t) j;
                double *d = &sm[2 * tileSwizzle(l)];
                if (f.tail.globalPhase < 0) mul(d, f.tail.globalRe, f.tail.globalIm);
                if (parity(tid & f.tail.signThr) ^ parity(cta & f.tail.signCta) ^ ((f.tail.signTab >> j) & 1))
                    mul(d, -1.0, 0.0);
                std::memcpy(&state[2 * address(cta, l)], d, 16);
            }
    }
}

}  // namespace dgq
