// planner.cpp -- see planner.h.
#include "planner.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "dag.h"

namespace dgq {

static const double kRsqrt2 = 0.7071067811865475244008443621;

// Block selection. dgQuEST's rule (DAG.cpp:219-259) walks the DAG depth
// first and admits gates while the target union fits; the tile bits then
// follow from the order of the walk. Here the tile's free bits are chosen
// first: starting from the 5 coalesced bits, add one at a time the bit that
// lets the most gates run (dependency-closed, non-diagonal targets inside
// the tile), considering only bits some runnable-next gate targets, then
// take every gate that fits. Phases inside a block use the same rule with
// the 4 register bits.
// Grows `mask` up to `budget` bits: each step adds the missing target bits
// of one runnable-next gate, choosing the addition that lets the most gates
// run (ties: fewer new bits; with preferHigh, bits above the 5 coalesced).
// Registers of at least this many address bits choose tile bits with a
// one-step lookahead unless told otherwise (measured on the 30-qubit random
// circuit of depth 20: 17 instead of 19 sweeps for 3x the planning time).
static int lookaheadMinBits() {
    static const int v = []() {
        const char *e = getenv("DGQ_PLAN_LOOKAHEAD_BITS");
        return e ? atoi(e) : 24;
    }();
    return v;
}

bool lookaheadBySize(int numBits) { return numBits >= lookaheadMinBits(); }

// lookahead: score each candidate addition by the best follow-up addition too
static void growMask(const GateDag &dag, u64 &mask, int budget, bool preferHigh, bool lookahead = false) {
    const u64 low = (1ULL << kCoalescedBits) - 1;
    std::vector<u64> sets;
    std::vector<size_t> counts, score;
    std::vector<std::pair<size_t, size_t>> uses;  // candidate, set
    while (popcount64(mask) < budget) {
        std::vector<u64> cands = dag.frontierSets(mask);
        cands.erase(std::remove_if(cands.begin(), cands.end(),
                                   [&](u64 add) { return popcount64(mask | add) > budget; }),
                    cands.end());
        // every candidate, and with lookahead every candidate with each
        // follow-up addition (most unions come up from both sides): counted
        // together
        sets.clear();
        uses.clear();
        auto use = [&](size_t cand, u64 set) {
            const size_t k = (size_t) (std::find(sets.begin(), sets.end(), set) - sets.begin());
            if (k == sets.size()) sets.push_back(set);
            uses.emplace_back(cand, k);
        };
        for (size_t i = 0; i < cands.size(); i++) {
            use(i, mask | cands[i]);
            if (lookahead && popcount64(mask | cands[i]) < budget)
                for (u64 add2 : dag.frontierSets(mask | cands[i]))
                    if (popcount64(mask | cands[i] | add2) <= budget) use(i, mask | cands[i] | add2);
        }
        counts.resize(sets.size());
        dag.countAllowed(sets.data(), sets.size(), counts.data());
        score.assign(cands.size(), 0);
        for (const auto &u : uses) score[u.first] = std::max(score[u.first], counts[u.second]);
        size_t best = 0;
        u64 bestAdd = 0;
        for (size_t i = 0; i < cands.size(); i++) {
            const u64 add = cands[i];
            const size_t c = score[i];
            bool better = c > best;
            if (!better && c == best && bestAdd) {
                const int pa = popcount64(add), pb = popcount64(bestAdd);
                if (pa < pb)
                    better = true;
                else if (pa == pb && preferHigh && (bestAdd & low) && !(add & low))
                    better = true;
            }
            if (better) {
                best = c;
                bestAdd = add;
            }
        }
        if (!bestAdd) break;
        mask |= bestAdd;
    }
}

// Grows `mask` keeping the `width` masks of each size that let the most gates
// run, and takes the best of all. Greedy growth commits to every bit, but no
// search is the best throughout, so the cost model plans with each. Sweeps of
// 12-bit tiles, greedy / with a step of lookahead / widths 4 / 16: 30 qubits at
// depth 20 19 / 18 / 19 / 17, a 26-qubit ansatz of depth 10 14 / 17 / 13 / 16,
// grids of depth 16, 4 x 7 14 / 14 / 13 / 13, 5 x 6 14 / 15 / 14 / 15.
static void beamMask(const GateDag &dag, u64 &mask, int budget, size_t width) {
    std::vector<u64> beam{mask}, sets, next;
    std::vector<size_t> counts, rank;
    size_t bestCount = 0;
    while (!beam.empty()) {
        sets.clear();
        for (u64 m : beam)
            for (u64 add : dag.frontierSets(m))
                if (popcount64(m | add) <= budget && std::find(sets.begin(), sets.end(), m | add) == sets.end())
                    sets.push_back(m | add);
        counts.resize(sets.size());
        rank.resize(sets.size());
        dag.countAllowed(sets.data(), sets.size(), counts.data());
        for (size_t i = 0; i < sets.size(); i++) {
            rank[i] = i;
            if (counts[i] > bestCount) {
                bestCount = counts[i];
                mask = sets[i];
            }
        }
        std::stable_sort(rank.begin(), rank.end(), [&](size_t a, size_t b) { return counts[a] > counts[b]; });
        next.clear();
        for (size_t i = 0; i < std::min(width, rank.size()); i++) next.push_back(sets[rank[i]]);
        beam.swap(next);
    }
}

bool planBlocksEach(const std::vector<Gate> &gates, int numBits, int tileBits, int seedBits,
                    const std::function<bool(BlockPlan &)> &onBlock, int lookahead) {
    GateDag dag(numBits, true);
    for (const Gate &g : gates) dag.add(g);
    const u64 seed = (1ULL << seedBits) - 1;
    const u64 all = numBits >= 64 ? ~0ULL : ((1ULL << numBits) - 1);
    const bool look = lookahead < 0 ? lookaheadBySize(numBits) : lookahead > 0;
    while (!dag.empty()) {
        BlockPlan b;
        u64 mask = seed & all;
        if (lookahead >= kSearchBeam4)
            beamMask(dag, mask, tileBits, lookahead == kSearchBeam4 ? 4 : 16);
        else
            growMask(dag, mask, tileBits, false, look);
        // pad to tileBits with the lowest unused bits above the seed
        for (int bit = seedBits; popcount64(mask) < tileBits && bit < numBits; bit++) mask |= 1ULL << bit;
        b.tileMask = mask & all;
        b.gates = dag.takeAllowed(b.tileMask);
        b.last = dag.empty();
        // only a gate wider than the tile is left: not plannable here
        if (b.gates.empty()) return false;
        if (!onBlock(b)) return true;
    }
    return true;
}

std::vector<BlockPlan> planBlocks(const std::vector<Gate> &gates, int numBits, int tileBits, bool *complete,
                                  int seedBits, int lookahead) {
    std::vector<BlockPlan> blocks;
    const bool ok = planBlocksEach(
        gates, numBits, tileBits, seedBits,
        [&](BlockPlan &b) {
            blocks.push_back(std::move(b));
            return true;
        },
        lookahead);
    if (complete) *complete = ok;
    return blocks;
}

namespace {

struct TileMap {
    int local[64];   // address bit -> tile-local bit, -1 if not in tile
    int ctaIdx[64];  // address bit -> blockIdx bit, -1 if in tile
    int tilePos[kMaxTileBits];
};

TileMap makeTileMap(u64 tileMask, int numBits) {
    TileMap m;
    int nl = 0, nc = 0;
    for (int b = 0; b < 64; b++) {
        m.local[b] = -1;
        m.ctaIdx[b] = -1;
    }
    for (int b = 0; b < numBits; b++) {
        if ((tileMask >> b) & 1ULL) {
            m.tilePos[nl] = b;
            m.local[b] = nl++;
        } else {
            m.ctaIdx[b] = nc++;
        }
    }
    return m;
}

struct Split {
    uint32_t tileLocal = 0;  // tile-local mask
    uint32_t cta = 0;        // blockIdx-space mask
};

Split splitMask(u64 m, const TileMap &tm) {
    Split s;
    for (; m; m &= m - 1) {
        const int b = __builtin_ctzll(m);
        if (tm.local[b] >= 0)
            s.tileLocal |= 1u << tm.local[b];
        else
            s.cta |= 1u << tm.ctaIdx[b];
    }
    return s;
}

struct PhaseLayout {
    int regPos[kRegBits];
    int thrPos[kMaxThreadBits];
    uint32_t regLocalMask = 0;
    bool direct = false;
};

// Register bits: `front` first (dense-gate target order), then the other
// targets, then padding from the top tile bit down. Thread bits: three bits
// of distinct (position mod 3) first, so that each quarter-warp touches 8
// distinct swizzled bank groups, then the rest in increasing order.
PhaseLayout makeLayout(const std::vector<int> &front, uint32_t targetsLocal, int tileBits, bool paired = false) {
    PhaseLayout L;
    int nr = 0;
    // paired form: tile-local bit 0 is the pair inside a slot, never a
    // register or thread bit
    uint32_t used = paired ? 1u : 0u;
    if (paired) targetsLocal &= ~1u;
    for (int p : front) {
        L.regPos[nr++] = p;
        used |= 1u << p;
    }
    for (int p = 0; p < tileBits && nr < kRegBits; p++) {
        if (((targetsLocal >> p) & 1u) && !((used >> p) & 1u)) {
            L.regPos[nr++] = p;
            used |= 1u << p;
        }
    }
    for (int p = tileBits - 1; p >= 0 && nr < kRegBits; p--) {
        if (!((used >> p) & 1u)) {
            L.regPos[nr++] = p;
            used |= 1u << p;
        }
    }
    if (paired) used &= ~1u;
    L.regLocalMask = used;
    std::vector<int> thr;
    for (int p = paired ? 1 : 0; p < tileBits; p++)
        if (!((used >> p) & 1u)) thr.push_back(p);
    // slots (16 B) are indexed by tile-local bits 1.. in the paired form
    const int sh = paired ? 1 : 0;
    L.direct = ((used >> sh) & ((1u << kCoalescedBits) - 1)) == 0;
    if (L.direct) {
        // lanes on tile bits 0..4 (address bits 0..4): the phase can read and
        // write HBM directly in 512-byte runs; bits 0..2 have distinct
        // classes mod 3, so its shared-memory accesses stay conflict-free
        int i = 0;
        for (int p : thr) L.thrPos[i++] = p;
        return L;
    }
    std::vector<int> lanes, rest;
    int classes = 0;
    for (int p : thr) {
        const int q = p - sh;
        if ((int) lanes.size() < 3 && !((classes >> (q % 3)) & 1)) {
            lanes.push_back(p);
            classes |= 1 << (q % 3);
        } else {
            rest.push_back(p);
        }
    }
    int i = 0;
    for (int p : lanes) L.thrPos[i++] = p;
    for (int p : rest) L.thrPos[i++] = p;
    return L;
}

uint8_t regSpace(uint32_t tileLocal, const PhaseLayout &L) {
    uint8_t r = 0;
    for (int b = 0; b < kRegBits; b++)
        if ((tileLocal >> L.regPos[b]) & 1u) r |= (uint8_t) (1u << b);
    return r;
}

bool isZero(double x) { return x == 0.0; }

// A register phase of a block: gates in order, dense-gate target order.
struct Phase {
    std::vector<Gate> gates;
    std::vector<int> front;
    uint32_t targetsLocal = 0;
};

// FP64 (complex64: packed FP32) instructions a thread spends on diagonal
// gate g in a phase of layout L. A phase factor on thread and CTA bits only
// is one number for the thread's 16 amplitudes: a few scalar instructions
// where the phase folds such factors (one closing multiply of all 16,
// kFoldCost), 64 by itself. With qubits among the register bits (or, paired,
// inside the slot) it multiplies the amplitudes they select.
constexpr int kFoldCost = 64;

struct DiagCost {
    int folded;   // in a phase that folds thread factors
    int alone;    // in one that does not
};

// c, t: g's controls and targets in the tile.
DiagCost diagCost(const Gate &g, const Split &c, const Split &t, const PhaseLayout &L, bool paired) {
    const uint32_t inThread = L.regLocalMask | (paired ? 1u : 0u);
    const uint32_t qubits = c.tileLocal | t.tileLocal;
    const bool signOnly = g.type < 8 && !(g.type & 1);  // +-1, +-i
    if (!(qubits & inThread)) return signOnly ? DiagCost{2, 16} : DiagCost{6, 64};
    // amplitudes touched, out of 16; the bit inside a slot halves nothing
    // (both halves go through a packed instruction)
    int amps = 16 >> popcount64(c.tileLocal & L.regLocalMask);
    if (g.type == OP_ROTATE_Z && g.controlMask == 0 && (t.tileLocal & L.regLocalMask)) amps = 8;
    const int cost = signOnly ? amps : 4 * amps;
    return {cost, cost};
}

// Moves every diagonal gate of a block to the phase where it costs least.
// Diagonal gates commute with all but the non-diagonal gates on their
// qubits, so a gate may run in any phase between the last such gate before
// it and the next one after it (at the end of an earlier phase, at the start
// of a later one). The phases that fold thread factors are chosen greedily
// (each pays for its closing multiply; the sweep's global factor pays for
// the first). Rz on a register bit costs 32 instructions a thread and on a
// thread bit 6, and one closing multiply serves the sweep instead of one per
// phase: 10 % of the arithmetic of the 30-qubit random circuit of depth 20
// (20890 -> 18764 instructions a thread over its 18 sweeps, 151.0 -> 145.7
// ms), 45 % of a 27-qubit Fourier transform's.
// carry (set unless the block is the last): receives the gates that stay on
// register bits and that no later gate of the block needs; the next block
// runs them, where their qubits may be thread bits.
void placeDiagonals(std::vector<Phase> &phases, const TileMap &tm, int tileBits, bool paired,
                    std::vector<Gate> *carry) {
    const int np = (int) phases.size();
    std::vector<PhaseLayout> layouts;
    for (const Phase &p : phases) layouts.push_back(makeLayout(p.front, p.targetsLocal, tileBits, paired));
    struct Item {
        int phase, index;  // where the gate is
        int lo, hi;        // phases it may run in
        bool open;         // no gate of the block must follow it
        int at;            // where it goes
        int best;          // its least cost so far
        size_t costs;      // its costs in phases lo..hi, in `costs`
    };
    std::vector<Item> items;
    std::vector<DiagCost> costs;
    // windows: from the last non-diagonal gate on its qubits (a pass forward,
    // with that gate's phase per qubit) to the next one (a pass backward)
    int lastOn[64], nextOn[64];
    std::fill(lastOn, lastOn + 64, 0);
    std::fill(nextOn, nextOn + 64, np);
    for (int p = 0; p < np; p++)
        for (int i = 0; i < (int) phases[p].gates.size(); i++) {
            const Gate &g = phases[p].gates[i];
            if (!isDiagonalType(g.type)) {
                for (u64 m = g.targetMask; m; m &= m - 1) lastOn[__builtin_ctzll(m)] = p;
                continue;
            }
            if (g.type == OP_ONE) continue;
            int lo = 0;
            for (u64 m = g.targetMask | g.controlMask; m; m &= m - 1) lo = std::max(lo, lastOn[__builtin_ctzll(m)]);
            items.push_back({p, i, lo, np - 1, true, p, 0, 0});
        }
    size_t back = items.size();
    for (int p = np - 1; p >= 0; p--)
        for (int i = (int) phases[p].gates.size() - 1; i >= 0; i--) {
            const Gate &g = phases[p].gates[i];
            if (!isDiagonalType(g.type)) {
                for (u64 m = g.targetMask; m; m &= m - 1) nextOn[__builtin_ctzll(m)] = p;
                continue;
            }
            if (g.type == OP_ONE) continue;
            Item &it = items[--back];
            for (u64 m = g.targetMask | g.controlMask; m; m &= m - 1) it.hi = std::min(it.hi, nextOn[__builtin_ctzll(m)]);
            for (u64 m = g.targetMask | g.controlMask; m; m &= m - 1) it.open = it.open && nextOn[__builtin_ctzll(m)] == np;
        }
    for (Item &it : items) {
        const Gate &g = phases[it.phase].gates[it.index];
        const Split c = splitMask(g.controlMask, tm), t = splitMask(g.targetMask, tm);
        it.costs = costs.size();
        for (int q = it.lo; q <= it.hi; q++) costs.push_back(diagCost(g, c, t, layouts[q], paired));
        const DiagCost *cost = &costs[it.costs];
        it.best = cost[it.phase - it.lo].alone;
        for (int q = it.lo; q <= it.hi; q++)
            if (cost[q - it.lo].alone < it.best) {
                it.best = cost[q - it.lo].alone;
                it.at = q;
            }
    }
    // uncontrolled rotations and Hadamards leave a global factor
    bool global = false;
    for (const Phase &p : phases)
        for (const Gate &g : p.gates)
            global = global || (!g.controlMask && (g.type == OP_ROTATE_Z || g.type == OP_ROTATE_X ||
                                                   g.type == OP_ROTATE_Y || g.type == OP_HADAMARD));
    std::vector<char> folds((size_t) np, 0);
    for (bool first = global;; first = false) {
        int bestPhase = -1, bestGain = 0;
        std::vector<int> gain((size_t) np, first ? 0 : -kFoldCost);
        for (const Item &it : items)
            for (int q = it.lo; q <= it.hi; q++)
                gain[q] += std::max(0, it.best - costs[it.costs + (size_t) (q - it.lo)].folded);
        for (int q = 0; q < np; q++)
            if (!folds[q] && gain[q] > bestGain) {
                bestGain = gain[q];
                bestPhase = q;
            }
        if (bestPhase < 0) break;
        folds[bestPhase] = 1;
        for (Item &it : items)
            if (bestPhase >= it.lo && bestPhase <= it.hi &&
                costs[it.costs + (size_t) (bestPhase - it.lo)].folded < it.best) {
                it.best = costs[it.costs + (size_t) (bestPhase - it.lo)].folded;
                it.at = bestPhase;
            }
    }
    std::vector<std::vector<Gate>> head((size_t) np), tail((size_t) np);
    std::vector<std::vector<char>> moved((size_t) np);
    for (int p = 0; p < np; p++) moved[p].assign(phases[p].gates.size(), 0);
    for (const Item &it : items) {
        const Gate &g = phases[it.phase].gates[it.index];
        const int scalar = g.type < 8 && !(g.type & 1) ? 2 : 6;
        if (carry && it.open && it.best > scalar)
            carry->push_back(g);
        else if (it.at != it.phase)
            (it.at > it.phase ? head : tail)[it.at].push_back(g);
        else
            continue;
        moved[it.phase][it.index] = 1;
    }
    for (int p = 0; p < np; p++) {
        std::vector<Gate> gates = std::move(head[p]);
        for (size_t i = 0; i < phases[p].gates.size(); i++)
            if (!moved[p][i]) gates.push_back(phases[p].gates[i]);
        gates.insert(gates.end(), tail[p].begin(), tail[p].end());
        phases[p].gates = std::move(gates);
    }
    phases.erase(std::remove_if(phases.begin(), phases.end(), [](const Phase &p) { return p.gates.empty(); }),
                 phases.end());
}

// Bits (-log2) by which a gate may shrink the scalar that its sweep leaves to
// one multiply: the factors of uncontrolled rotations, Hadamards and XY-plane
// unitaries, and the first entry of a general 2x2 in a framed program.
double scalarBits(const Gate &g) {
    if (g.controlMask || isDiagonalType(g.type) || g.type == OP_MULTI_UNITARY) return 0.0;
    switch (g.type) {
        case OP_PAULI_X:
        case OP_PAULI_Y:
        case OP_PAULI_Y_CONJ: return 0.0;
        case OP_HADAMARD: return 0.5;
        case OP_ROTATE_X:
        case OP_ROTATE_Y: return -std::log2(std::max(std::fabs(std::cos(g.op[0])), std::fabs(std::sin(g.op[0]))));
        default: {
            double m[8];
            gateMatrix(g, m);
            const double d = std::max(std::hypot(m[0], m[1]), std::hypot(m[4], m[5]));
            return d > 0.0 && d < 1.0 ? -std::log2(d) : 0.0;
        }
    }
}

// Cuts phases whose ops, coefficients or scalar could exceed a program's
// capacity (gates gathered in one phase); the parts keep the phase's layout.
void splitLongPhases(std::vector<Phase> &phases, bool scalarLimited) {
    auto coefs = [](const Gate &g) {
        return g.type == OP_MULTI_UNITARY ? 2 << (2 * g.numMultiTargets) : isDiagonalType(g.type) ? 2 : 8;
    };
    std::vector<Phase> out;
    for (Phase &p : phases) {
        int n = 0, c = 0;
        double b = 0.0;
        for (const Gate &g : p.gates) {
            n++;
            c += coefs(g);
            if (scalarLimited) b += scalarBits(g);
        }
        if (n <= kMaxOps && c <= kMaxCoef && b <= kMaxScalarBitsF32) {
            out.push_back(std::move(p));
            continue;
        }
        Phase part{{}, p.front, p.targetsLocal};
        n = c = 0;
        b = 0.0;
        for (const Gate &g : p.gates) {
            const double bits = scalarLimited ? scalarBits(g) : 0.0;
            if (n + 1 > kMaxOps || c + coefs(g) > kMaxCoef || b + bits > kMaxScalarBitsF32) {
                out.push_back(part);
                part.gates.clear();
                n = c = 0;
                b = 0.0;
            }
            part.gates.push_back(g);
            n++;
            c += coefs(g);
            b += bits;
        }
        out.push_back(std::move(part));
    }
    phases.swap(out);
}

}  // namespace

double opFlopsPerAmp(const KOp &op) {
    double f = 0.0;
    switch (op.kind) {
        case KOP_M2R:
        case KOP_M2I:
        case KOP_PH:
        case KOP_Z2: f = 6.0; break;
        case KOP_M2C: f = 14.0; break;
        case KOP_DENSE: f = 8.0 * (double) (1 << op.k) - 2.0; break;
        case KOP_RY1:
        case KOP_RY2:
        case KOP_RX1:
        case KOP_RX2: f = 4.0; break;   // one FMA per output component
        case KOP_H1: f = 2.0; break;    // one add per output component
        case KOP_PH1: f = 3.0; break;   // a complex multiply on half of the amplitudes
        case KOP_RN1: f = 8.0; break;   // x + p y: two complex FMAs per amplitude
        default: f = 0.0; break;
    }
    const int c = __builtin_popcount(op.ctrlReg) + __builtin_popcount(op.ctrlLoc) + __builtin_popcount(op.ctrlCta);
    return f / (double) (1u << c);
}

void encodeHeaderOnly(int numBits, int numReal, int tileBits, const SweepHeader &hdr, TileProgram &out,
                      bool paired) {
    std::memset(&out, 0, sizeof(out));
    out.paired = paired ? 1 : 0;
    out.globalRe = 1.0;
    out.numBits = numBits;
    out.numReal = numReal;
    out.initKind = hdr.initKind;
    out.initIndex = hdr.initIndex;
    out.initAmp = hdr.initAmp;
    out.hasRestrict = hdr.hasRestrict ? 1 : 0;
    out.restrictMask = hdr.restrictMask;
    out.restrictValue = hdr.restrictValue;
    out.restrictScale = hdr.restrictScale;
    // tile = the lowest tileBits bits
    for (int i = 0; i < tileBits - kCoalescedBits; i++) out.highPos[i] = (uint8_t) (kCoalescedBits + i);
    for (int i = 0; i < numBits - tileBits; i++) out.ctaPos[i] = (uint8_t) (tileBits + i);
}

// (Phases on three qubits and more have a framed form too, but placing the
// diagonal gates of such lists costs more on the host, 50 us of 770 at 14
// qubits, than it saves on the GPU, 5 us of 179.)
bool framedGates(const std::vector<Gate> &gates) {
    for (const Gate &g : gates) {
        const int controls = popcount64(g.controlMask);
        if (isDiagonalType(g.type) ? controls + popcount64(g.targetMask) > 2
                                   : g.type == OP_MULTI_UNITARY || controls > (g.type == OP_PAULI_X ? 1 : 0))
            return false;
    }
    return true;
}

bool encodeBlock(const BlockPlan &block, int numBits, int numReal, int tileBits, const MatrixPool &pool,
                 const SweepHeader &first, std::vector<TileProgram> &out, PlanStats *stats, std::string *err,
                 bool paired, Folding folds, std::vector<Gate> *carry, bool single) {
    // (at most half a bit a gate: few blocks can reach the limit)
    int pairGates = 0;
    if (single || paired)
        for (const Gate &g : block.gates) pairGates += !isDiagonalType(g.type) && !g.controlMask;
    const bool scalarLimited = 0.5 * pairGates > kMaxScalarBitsF32;
    const TileMap tm = makeTileMap(block.tileMask, numBits);
    std::vector<Gate> carried;
    if (carry) carried.swap(*carry);

    // ---- phases: greedy DAG selection with the register budget
    std::vector<Phase> phases;
    {
        GateDag dag(numBits, false);
        for (const Gate &g : carried) dag.add(g);
        for (const Gate &g : block.gates) dag.add(g);
        while (!dag.empty()) {
            // paired form: address bit 0 is always inside the thread
            u64 mask = paired ? 1ULL : 0ULL;
            growMask(dag, mask, kRegBits + (paired ? 1 : 0), true, true);
            std::vector<Gate> gs = dag.takeAllowed(mask);
            if (gs.empty()) {
                // a multi-target gate wider than the register bits
                u64 m2 = 0;
                gs = dag.takeBlock(kRegBits, m2, 1u << 20);
            }
            if (gs.empty()) {
                if (err) *err = "a gate has more non-diagonal targets than the register tile holds";
                return false;
            }
            // the interpreting kernels' (and the paired form's) dense op acts on
            // register bits 0..k-1, so the gate fixes the register order and has
            // a phase of its own; a specialised kernel takes any register bits
            // (12-qubit density matrix, two layers with a channel per qubit: some
            // 45 phases become 21, 2.19 -> 1.50 ms)
            Phase cur;
            auto flush = [&]() {
                if (!cur.gates.empty()) phases.push_back(cur);
                cur = Phase();
            };
            for (const Gate &g : gs) {
                if (g.type == OP_MULTI_UNITARY) {
                    if (paired && (g.targetMask & 1ULL)) {
                        if (err) *err = "paired form: a multi-qubit unitary targets address bit 0";
                        return false;
                    }
                    if (folds == Folding::Specialised && !paired) {
                        cur.gates.push_back(g);
                        cur.targetsLocal |= splitMask(g.targetMask, tm).tileLocal;
                        continue;
                    }
                    flush();
                    Phase d;
                    d.gates.push_back(g);
                    for (int i = 0; i < g.numMultiTargets; i++) d.front.push_back(tm.local[g.multiTargets[i]]);
                    d.targetsLocal = splitMask(g.targetMask, tm).tileLocal;
                    phases.push_back(d);
                    continue;
                }
                cur.gates.push_back(g);
                if (!isDiagonalType(g.type)) cur.targetsLocal |= splitMask(g.targetMask, tm).tileLocal;
            }
            flush();
        }
    }

    if (folds != Folding::None) placeDiagonals(phases, tm, tileBits, paired, block.last ? nullptr : carry);
    splitLongPhases(phases, scalarLimited);

    // ---- programs
    auto newProgram = [&](bool isFirst) {
        out.emplace_back();
        TileProgram &p = out.back();
        std::memset(&p, 0, sizeof(p));
        p.numBits = numBits;
        p.numReal = numReal;
        p.globalRe = 1.0;
        p.globalIm = 0.0;
        p.hasGlobal = 0;
        p.paired = paired ? 1 : 0;
        if (isFirst) {
            p.initKind = first.initKind;
            p.initIndex = first.initIndex;
            p.initAmp = first.initAmp;
            p.hasRestrict = first.hasRestrict ? 1 : 0;
            p.restrictMask = first.restrictMask;
            p.restrictValue = first.restrictValue;
            p.restrictScale = first.restrictScale;
        } else {
            p.initKind = INIT_NONE;
        }
        for (int i = 0; i < tileBits - kCoalescedBits; i++) p.highPos[i] = (uint8_t) tm.tilePos[kCoalescedBits + i];
        for (int b = 0; b < numBits; b++)
            if (tm.ctaIdx[b] >= 0) p.ctaPos[tm.ctaIdx[b]] = (uint8_t) b;
        if (stats) stats->sweeps++;
        return &out.back();
    };
    TileProgram *prog = newProgram(true);
    int numCoef = 0;
    double scalar = 0.0;  // the program's scalar may have shrunk by so many bits

    for (const Phase &ph : phases) {
        const PhaseLayout L = makeLayout(ph.front, ph.targetsLocal, tileBits, paired);
        // encode the phase's ops into a scratch list first; uncontrolled
        // rotations leave their scalar factor in (phRe, phIm)
        std::vector<KOp> ops;
        std::vector<double> coef;
        double phRe = 1.0, phIm = 0.0, phBits = 0.0;
        auto scaleBy = [&](double fr, double fi) {
            const double r = phRe * fr - phIm * fi, i = phRe * fi + phIm * fr;
            phRe = r;
            phIm = i;
        };
        for (const Gate &g : ph.gates) {
            if (scalarLimited) phBits += scalarBits(g);
            KOp op;
            std::memset(&op, 0, sizeof(op));
            op.selCta = -1;
            const Split c = splitMask(g.controlMask, tm);
            op.ctrlReg = regSpace(c.tileLocal, L);
            op.ctrlLoc = (uint16_t) (c.tileLocal & ~L.regLocalMask);
            op.ctrlCta = c.cta;
            op.coef = (uint16_t) coef.size();  // phase-relative, rebased when copied
            auto targetReg = [&](u64 tmask) -> int {
                const Split t = splitMask(tmask, tm);
                if (paired && t.tileLocal == 1u) return 4;  // the pair inside a slot
                for (int b = 0; b < kRegBits; b++)
                    if (t.tileLocal == (1u << L.regPos[b])) return b;
                return -1;
            };
            bool emit = true;
            bool selIsReg = false;
            const int t = (int) g.type;
            if (t < 8) {
                switch (t) {
                    case OP_ONE: emit = false; break;
                    case OP_S_GATE: op.kind = KOP_MULI; break;
                    case OP_PAULI_Z: op.kind = KOP_NEG; break;
                    case OP_S_GATE_CONJ: op.kind = KOP_MULNI; break;
                    default: {
                        // odd powers: e^{i pi t / 4} with (+-1 +- i)/sqrt(2)
                        op.kind = KOP_PH;
                        const double c0 = (t == 1 || t == 7) ? kRsqrt2 : -kRsqrt2;
                        const double s0 = (t == 1 || t == 3) ? kRsqrt2 : -kRsqrt2;
                        coef.push_back(c0);
                        coef.push_back(s0);
                        break;
                    }
                }
            } else if (g.type == OP_PHASE_SHIFT) {
                op.kind = KOP_PH;
                coef.push_back(std::cos(g.op[0]));
                coef.push_back(std::sin(g.op[0]));
            } else if (g.type == OP_ROTATE_Z && g.controlMask == 0) {
                // diag(e^{-ia}, e^{ia}) = e^{-ia} diag(1, e^{2ia})
                op.kind = KOP_PH1;
                coef.push_back(std::cos(2.0 * g.op[0]));
                coef.push_back(std::sin(2.0 * g.op[0]));
                scaleBy(std::cos(g.op[0]), -std::sin(g.op[0]));
                const Split s = splitMask(g.targetMask, tm);
                if (s.tileLocal) {
                    const uint8_t r = regSpace(s.tileLocal, L);
                    if (r) {
                        op.k = (uint8_t) __builtin_ctz(r);
                        selIsReg = true;
                    } else {
                        op.selLoc = (uint16_t) s.tileLocal;
                    }
                } else {
                    op.selCta = (int8_t) __builtin_ctz(s.cta);
                }
            } else if (g.type == OP_ROTATE_Z) {
                op.kind = KOP_Z2;
                coef.push_back(std::cos(g.op[0]));
                coef.push_back(std::sin(g.op[0]));
                const Split s = splitMask(g.targetMask, tm);
                if (s.tileLocal) {
                    const uint8_t r = regSpace(s.tileLocal, L);
                    if (r) {
                        op.k = (uint8_t) __builtin_ctz(r);
                        selIsReg = true;
                    } else {
                        op.selLoc = (uint16_t) s.tileLocal;
                    }
                } else {
                    op.selCta = (int8_t) __builtin_ctz(s.cta);
                }
            } else if (g.type == OP_MULTI_UNITARY) {
                op.kind = KOP_DENSE;
                op.k = (uint8_t) g.numMultiTargets;
                const auto &m = pool.mats[(size_t) g.multiIndex];
                coef.insert(coef.end(), m.begin(), m.end());
                if (folds == Folding::Specialised && !paired) {
                    op.selLoc = (uint16_t) (kDenseAnyBits | g.multiShape << 8);
                    for (int i = 0; i < g.numMultiTargets; i++)
                        for (int b = 0; b < kRegBits; b++)
                            if (L.regPos[b] == tm.local[g.multiTargets[i]]) op.selLoc |= (uint16_t) (b << (2 * i));
                }
            } else {
                const int k = targetReg(g.targetMask);
                if (k < 0) {
                    if (err) *err = "internal: pair-gate target is not a register bit";
                    return false;
                }
                op.k = (uint8_t) k;
                const bool free = g.controlMask == 0;
                switch (g.type) {
                    case OP_HADAMARD:
                        if (!free) {
                            op.kind = KOP_M2R;
                            coef.insert(coef.end(), {kRsqrt2, kRsqrt2, kRsqrt2, -kRsqrt2});
                        } else {
                            op.kind = KOP_H1;
                            scaleBy(kRsqrt2, 0.0);
                        }
                        break;
                    case OP_ROTATE_Y:
                    case OP_ROTATE_X: {
                        const double cs = std::cos(g.op[0]), sn = std::sin(g.op[0]);
                        const bool isY = g.type == OP_ROTATE_Y;
                        if (!free) {
                            op.kind = isY ? KOP_M2R : KOP_M2I;
                            if (isY)
                                coef.insert(coef.end(), {cs, -sn, sn, cs});
                            else
                                coef.insert(coef.end(), {cs, -sn, -sn, cs});
                        } else if (std::fabs(cs) >= std::fabs(sn)) {
                            op.kind = isY ? KOP_RY1 : KOP_RX1;
                            coef.push_back(sn / cs);
                            scaleBy(cs, 0.0);
                        } else {
                            op.kind = isY ? KOP_RY2 : KOP_RX2;
                            coef.push_back(cs / sn);
                            scaleBy(sn, 0.0);
                        }
                        break;
                    }
                    case OP_PAULI_X: op.kind = KOP_X; break;
                    case OP_PAULI_Y: op.kind = KOP_Y; break;
                    case OP_PAULI_Y_CONJ: op.kind = KOP_YC; break;
                    default: {
                        double m[8];
                        gateMatrix(g, m);
                        // uncontrolled rotation about an axis in the XY plane:
                        // U = d [[1, p], [-conj(p), 1]] with d = U00 = U11,
                        // |p| <= 1; d goes to the sweep's global factor
                        const double d2 = m[0] * m[0] + m[1] * m[1];
                        const double o2 = m[2] * m[2] + m[3] * m[3];
                        const double tol = 1e-15 * std::sqrt(d2 + o2);
                        if (free && d2 > 0.0 && o2 <= d2 * (1.0 + 1e-12) && std::fabs(m[6] - m[0]) <= tol &&
                            std::fabs(m[7] - m[1]) <= tol) {
                            // p = U01 / U00, q = U10 / U00 must equal -conj(p)
                            const double pr = (m[2] * m[0] + m[3] * m[1]) / d2, pi = (m[3] * m[0] - m[2] * m[1]) / d2;
                            const double qr = (m[4] * m[0] + m[5] * m[1]) / d2, qi = (m[5] * m[0] - m[4] * m[1]) / d2;
                            if (std::fabs(qr + pr) <= 1e-14 && std::fabs(qi - pi) <= 1e-14) {
                                scaleBy(m[0], m[1]);
                                if (std::fabs(pi) <= 1e-16) {
                                    op.kind = KOP_RY1;  // p = -t
                                    coef.push_back(-pr);
                                } else if (std::fabs(pr) <= 1e-16) {
                                    op.kind = KOP_RX1;  // p = -i t
                                    coef.push_back(-pi);
                                } else {
                                    op.kind = KOP_RN1;
                                    coef.push_back(pr);
                                    coef.push_back(pi);
                                }
                                break;
                            }
                        }
                        if (isZero(m[1]) && isZero(m[3]) && isZero(m[5]) && isZero(m[7])) {
                            op.kind = KOP_M2R;
                            coef.insert(coef.end(), {m[0], m[2], m[4], m[6]});
                        } else if (isZero(m[1]) && isZero(m[2]) && isZero(m[4]) && isZero(m[7])) {
                            op.kind = KOP_M2I;
                            coef.insert(coef.end(), {m[0], m[3], m[5], m[6]});
                        } else {
                            op.kind = KOP_M2C;
                            coef.insert(coef.end(), m, m + 8);
                        }
                        break;
                    }
                }
            }
            if (emit) {
                const int rc = op.ctrlReg ? 1 : 0;
                const uint8_t kSaved = op.k;
                if (op.k == 4 && op.kind != KOP_DENSE) op.k = 0;  // codes index k < 4; paired ops keep k = 4
                op.thrCtl = (op.ctrlLoc || op.ctrlCta) ? 1 : 0;
                switch (op.kind) {
                    case KOP_M2R: op.code = (uint8_t) (KC_M2R + op.k + 4 * rc); break;
                    case KOP_M2I: op.code = (uint8_t) (KC_M2I + op.k + 4 * rc); break;
                    case KOP_M2C: op.code = (uint8_t) (KC_M2C + op.k + 4 * rc); break;
                    case KOP_X: op.code = (uint8_t) (KC_X + op.k + 4 * rc); break;
                    case KOP_Y: op.code = (uint8_t) (KC_Y + op.k + 4 * rc); break;
                    case KOP_YC: op.code = (uint8_t) (KC_YC + op.k + 4 * rc); break;
                    case KOP_Z2: op.code = (uint8_t) (selIsReg ? KC_Z2R + op.k + 4 * rc : KC_Z2T + rc); break;
                    case KOP_PH: op.code = (uint8_t) (KC_PH + rc); break;
                    case KOP_NEG: op.code = (uint8_t) (KC_NEG + rc); break;
                    case KOP_MULI: op.code = (uint8_t) (KC_MULI + rc); break;
                    case KOP_MULNI: op.code = (uint8_t) (KC_MULNI + rc); break;
                    case KOP_DENSE: op.code = (uint8_t) (KC_DENSE + op.k - 1); break;
                    case KOP_RY1: op.code = (uint8_t) (KC_RY1 + op.k); break;
                    case KOP_RY2: op.code = (uint8_t) (KC_RY2 + op.k); break;
                    case KOP_RX1: op.code = (uint8_t) (KC_RX1 + op.k); break;
                    case KOP_RX2: op.code = (uint8_t) (KC_RX2 + op.k); break;
                    case KOP_H1: op.code = (uint8_t) (KC_H1 + op.k); break;
                    case KOP_PH1: op.code = (uint8_t) (selIsReg ? KC_PH1R + op.k : KC_PH1T); break;
                    case KOP_RN1: op.code = (uint8_t) (KC_RN1 + op.k); break;
                    default: break;
                }
                op.k = kSaved;
                ops.push_back(op);
            }
        }
        if (ops.size() > (size_t) kMaxOps || coef.size() > (size_t) kMaxCoef) {
            if (err) *err = "a single register phase exceeds the tile program capacity";
            return false;
        }
        // start a new program (one more sweep over the same tile) when full
        if (prog->numPhases + 1 > kMaxPhases || prog->numOps + (int) ops.size() > kMaxOps ||
            numCoef + (int) coef.size() > kMaxCoef || scalar + phBits > kMaxScalarBitsF32) {
            prog = newProgram(false);
            numCoef = 0;
            scalar = 0.0;
        }
        scalar += phBits;
        if (phRe != 1.0 || phIm != 0.0) {
            const double gr = prog->globalRe, gi = prog->globalIm;
            prog->globalRe = gr * phRe - gi * phIm;
            prog->globalIm = gr * phIm + gi * phRe;
            prog->hasGlobal = 1;
        }
        KPhase &kp = prog->phases[prog->numPhases++];
        std::memset(&kp, 0, sizeof(kp));
        for (int i = 0; i < tileBits - kRegBits - (paired ? 1 : 0); i++) kp.thrPos[i] = (uint8_t) L.thrPos[i];
        for (int b = 0; b < kRegBits; b++) kp.regPos[b] = (uint8_t) L.regPos[b];
        kp.direct = L.direct ? 1 : 0;
        kp.opBegin = (uint16_t) prog->numOps;
        for (KOp o : ops) {
            o.coef = (uint16_t) (o.coef + numCoef);
            prog->ops[prog->numOps++] = o;
            if (stats) {
                stats->ops++;
                stats->flopsPerAmp += opFlopsPerAmp(o);
            }
        }
        kp.opEnd = (uint16_t) prog->numOps;
        for (int j = 0; j < kRegs; j++) {
            uint32_t loc = 0;
            for (int b = 0; b < kRegBits; b++)
                if ((j >> b) & 1) loc |= 1u << L.regPos[b];
            kp.regOff[j] = (uint16_t) tileSwizzle(paired ? loc >> 1 : loc);
        }
        for (double c : coef) prog->coef[numCoef++] = c;
        prog->numCoef = (uint16_t) numCoef;
        if (stats) stats->phases++;
    }
    if (stats) stats->gates += (int) block.gates.size();
    return true;
}

}  // namespace dgq
