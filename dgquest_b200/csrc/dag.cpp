// dag.cpp -- see dag.h for the behaviour and its dgQuEST citations.
#include "dag.h"

#include <algorithm>
#include <cmath>

namespace dgq {

static const double kPiOn4 = 0.78539816339744830961566084581987572;
static const double kRsqrt2 = 0.7071067811865475244008443621;

void matMul2(const double a[8], const double b[8], double c[8]) {
    // element (r, k) lives at [4r + 2k] (re) and [4r + 2k + 1] (im)
    for (int r = 0; r < 2; r++) {
        for (int k = 0; k < 2; k++) {
            double re = 0.0, im = 0.0;
            for (int m = 0; m < 2; m++) {
                const double xr = a[4 * r + 2 * m], xi = a[4 * r + 2 * m + 1];
                const double yr = b[4 * m + 2 * k], yi = b[4 * m + 2 * k + 1];
                re += xr * yr - xi * yi;
                im += xr * yi + xi * yr;
            }
            c[4 * r + 2 * k] = re;
            c[4 * r + 2 * k + 1] = im;
        }
    }
}

void gateMatrix(const Gate &g, double m[8]) {
    for (int i = 0; i < 8; i++) m[i] = 0.0;
    const double a = g.op[0];
    switch (g.type) {
        case OP_ROTATE_Z:
            m[0] = std::cos(a); m[1] = -std::sin(a);
            m[6] = std::cos(a); m[7] = std::sin(a);
            break;
        case OP_PAULI_X: m[2] = 1.0; m[4] = 1.0; break;
        case OP_PAULI_Y: m[3] = -1.0; m[5] = 1.0; break;
        case OP_PAULI_Y_CONJ: m[3] = 1.0; m[5] = -1.0; break;
        case OP_HADAMARD: m[0] = kRsqrt2; m[2] = kRsqrt2; m[4] = kRsqrt2; m[6] = -kRsqrt2; break;
        case OP_ROTATE_X:
            m[0] = std::cos(a); m[3] = -std::sin(a);
            m[5] = -std::sin(a); m[6] = std::cos(a);
            break;
        case OP_ROTATE_Y:
            m[0] = std::cos(a); m[2] = -std::sin(a);
            m[4] = std::sin(a); m[6] = std::cos(a);
            break;
        case OP_COMPACT_UNITARY:  // [[alpha, -conj(beta)], [beta, conj(alpha)]]
            m[0] = g.op[0]; m[1] = g.op[1];
            m[2] = -g.op[2]; m[3] = g.op[3];
            m[4] = g.op[2]; m[5] = g.op[3];
            m[6] = g.op[0]; m[7] = -g.op[1];
            break;
        case OP_UNITARY:
            for (int i = 0; i < 8; i++) m[i] = g.op[i];
            break;
        default:
            break;
    }
}

GateDag::GateDag(int numQubits, bool mergeGates)
    : numQubits_(numQubits), merge_(mergeGates), qubitStack_((size_t) numQubits) {}

// Merge the new gate g into node `top` (identical masks, no successors).
// Returns true when g was absorbed (top updated or deleted).
bool GateDag::tryMerge(int top, const Gate &g) {
    Node &t = nodes_[(size_t) top];
    if (t.g.targetMask != g.targetMask || t.g.controlMask != g.controlMask) return false;
    // lower type first; on equal types the later gate (g) plays "first"
    const bool newIsHigher = g.type > t.g.type;
    const Gate &lo = newIsHigher ? t.g : g;
    const Gate &hi = newIsHigher ? g : t.g;
    auto removeTop = [&]() {
        unlinkDeleted(top);
        return true;
    };
    if ((int) hi.type < 8) {
        const int sum = ((int) lo.type + (int) hi.type) % 8;
        if (sum == 0) return removeTop();
        t.g.type = (GateType) sum;
        return true;
    }
    if (hi.type == OP_PHASE_SHIFT) {
        Gate merged = hi;
        merged.op[0] = hi.op[0] + (lo.type == OP_PHASE_SHIFT ? lo.op[0] : kPiOn4 * (int) lo.type);
        t.g = merged;
        return true;
    }
    if (hi.type == OP_UNITARY) {
        // time order: t (earlier) then g (later): result = later * earlier
        double mLater[8], mEarlier[8], prod[8];
        if (g.type == OP_UNITARY) {
            for (int i = 0; i < 8; i++) mLater[i] = g.op[i];
        } else {
            gateMatrix(g, mLater);
        }
        if (t.g.type == OP_UNITARY) {
            for (int i = 0; i < 8; i++) mEarlier[i] = t.g.op[i];
        } else {
            gateMatrix(t.g, mEarlier);
        }
        matMul2(mLater, mEarlier, prod);
        if (t.g.type != OP_UNITARY) remerge_ = true;
        Gate merged = hi;
        merged.type = OP_UNITARY;
        for (int i = 0; i < 8; i++) merged.op[i] = prod[i];
        t.g = merged;
        return true;
    }
    if (lo.type == hi.type) {
        if (lo.type >= OP_PAULI_X && lo.type <= OP_HADAMARD) return removeTop();
        if (lo.type == OP_ROTATE_X || lo.type == OP_ROTATE_Y || lo.type == OP_ROTATE_Z) {
            if (lo.op[0] == -hi.op[0]) return removeTop();
            t.g.op[0] = lo.op[0] + hi.op[0];
            return true;
        }
    }
    return false;
}

void GateDag::unlinkDeleted(int idx) {
    flatValid_ = false;
    Node &d = nodes_[(size_t) idx];
    // the top of its own qubits' stacks, and of no other's
    for (u64 m = d.g.targetMask | d.g.controlMask; m; m &= m - 1) {
        auto &st = qubitStack_[(size_t) __builtin_ctzll(m)];
        if (!st.empty() && st.back() == idx) st.pop_back();
    }
    for (int i = 0; i < d.prevCount; i++) nodes_[(size_t) prevPool_[(size_t) (d.prevBegin + i)]].next--;
    d.alive = false;
    d.prevCount = 0;
    alive_--;
}

void GateDag::add(const Gate &g) {
    if (stale_) rebuild();
    flatValid_ = false;
    const int idx = (int) nodes_.size();
    if (!merge_) {
        // nothing asks for its neighbours
        Node &node = nodes_.emplace_back();
        node.g = g;
        alive_++;
        return;
    }
    const u64 barrier = g.targetMask | g.controlMask;
    const int prevBegin = (int) prevPool_.size();
    bool linked = false;
    for (u64 m = barrier; m; m &= m - 1) {
        const int q = __builtin_ctzll(m);
        auto &st = qubitStack_[(size_t) q];
        if (!st.empty()) {
            const int top = st.back();
            if (!linked && nodes_[(size_t) top].next == 0 && tryMerge(top, g)) {
                // absorbed; the stacks pushed so far for this gate must be undone
                for (u64 u = barrier & ((1ULL << q) - 1); u; u &= u - 1) {
                    auto &s2 = qubitStack_[(size_t) __builtin_ctzll(u)];
                    if (!s2.empty() && s2.back() == idx) s2.pop_back();
                }
                prevPool_.resize((size_t) prevBegin);
                return;
            }
            if (std::find(prevPool_.begin() + prevBegin, prevPool_.end(), top) == prevPool_.end()) {
                prevPool_.push_back(top);
                nodes_[(size_t) top].next++;
            }
            linked = true;
        }
        st.push_back(idx);
    }
    Node &node = nodes_.emplace_back();
    node.g = g;
    node.prevBegin = prevBegin;
    node.prevCount = (int) prevPool_.size() - prevBegin;
    alive_++;
}

// The alive gates added again, as to a fresh DAG (with merging).
void GateDag::rebuild() {
    std::vector<Gate> rest = gatesInOrder();
    nodes_.clear();
    prevPool_.clear();
    flatValid_ = false;
    remerge_ = stale_ = false;
    alive_ = 0;
    for (auto &st : qubitStack_) st.clear();
    for (const Gate &g : rest) add(g);
}

std::vector<Gate> GateDag::takeBlock(int budget, u64 &mask, size_t maxGates) {
    const size_t N = nodes_.size();
    // successors in insertion order, and the gates without predecessors
    std::vector<std::vector<int>> next(N);
    std::vector<size_t> remain(N, 0);
    std::vector<int> fronts, last((size_t) numQubits_, -1);
    std::vector<u64> cost(N, 0);
    std::vector<char> visited(N, 0), selected(N, 0);
    for (size_t i = 0; i < N; i++) {
        if (!nodes_[i].alive) continue;
        const Gate &g = nodes_[i].g;
        cost[i] = isDiagonalType(g.type) ? 0 : g.targetMask;
        for (u64 m = g.targetMask | g.controlMask; m; m &= m - 1) {
            const size_t q = (size_t) __builtin_ctzll(m);
            if (last[q] >= 0) {
                auto &nx = next[(size_t) last[q]];
                if (nx.empty() || nx.back() != (int) i) {
                    nx.push_back((int) i);
                    remain[i]++;
                }
            }
            last[q] = (int) i;
        }
        if (!remain[i]) fronts.push_back((int) i);
    }
    // iterative depth-first walk: (node, next child position)
    std::vector<std::pair<int, size_t>> stack;
    auto enter = [&](int v) {
        visited[(size_t) v] = 1;
        if (popcount64(mask | cost[(size_t) v]) <= budget) {
            selected[(size_t) v] = 1;
            mask |= cost[(size_t) v];
            stack.emplace_back(v, 0);
        }
    };
    for (int f : fronts) {
        if (visited[(size_t) f]) continue;
        enter(f);
        while (!stack.empty()) {
            auto &top = stack.back();
            const auto &nx = next[(size_t) top.first];
            if (top.second >= nx.size()) {
                stack.pop_back();
                continue;
            }
            const int c = nx[top.second++];
            if (!visited[(size_t) c] && --remain[(size_t) c] == 0) enter(c);
        }
    }
    std::vector<Gate> taken;
    for (size_t i = 0; i < N; i++) {
        if (!nodes_[i].alive || !selected[i] || taken.size() >= maxGates) continue;
        taken.push_back(nodes_[i].g);
        nodes_[i].alive = false;
    }
    rebuild();
    return taken;
}

void GateDag::refreshFlat() const {
    if (flatValid_) return;
    flatTouch_.clear();
    flatCost_.clear();
    flatNode_.clear();
    for (size_t i = 0; i < nodes_.size(); i++) {
        const Node &nd = nodes_[i];
        if (!nd.alive) continue;
        const u64 touch = nd.g.targetMask | nd.g.controlMask;
        flatTouch_.push_back(touch);
        flatCost_.push_back(touchCost_ ? touch : isDiagonalType(nd.g.type) ? 0 : nd.g.targetMask);
        flatNode_.push_back((int) i);
    }
    flatValid_ = true;
}

// Insertion order is a topological order, so one forward pass decides
// which gates are reachable inside `allowed`: a gate held back holds back
// every later gate on its qubits. One scan for 8 candidate sets, without
// branches: with 256- or 512-bit vectors a gate costs the eight sets little
// more than one (the scans were 55 % of a plan's time, most of it in
// mispredicted branches).
typedef u64 Sets8 __attribute__((vector_size(64)));

#if defined(__x86_64__)
__attribute__((target_clones("arch=x86-64-v4", "avx2", "default")))
#endif
static void countAllowed8(const u64 *touch, const u64 *cost, size_t n, u64 all, const u64 *allowed, size_t *counts) {
    Sets8 outside, blocked = {}, free = {};
    for (int k = 0; k < 8; k++) outside[k] = ~allowed[k];
    for (size_t i = 0; i < n;) {
        const size_t e = std::min(n, i + 16);
        for (; i < e; i++) {
            const Sets8 hit = (touch[i] & blocked) | (cost[i] & outside);
            const Sets8 runs = (Sets8) (hit == 0);  // ~0 where it does
            blocked |= touch[i] & ~runs;
            free -= runs;
        }
        // every later gate is held back in all sets
        u64 open = 0;
        for (int k = 0; k < 8; k++) open |= ~blocked[k];
        if (!(open & all)) break;
    }
    for (int k = 0; k < 8; k++) counts[k] = free[k];
}

void GateDag::countAllowed(const u64 *allowed, size_t total, size_t *counts) const {
    refreshFlat();
    const u64 all = numQubits_ >= 64 ? ~0ULL : ((1ULL << numQubits_) - 1);
    for (size_t c = 0; c < total; c += 8) {
        u64 set[8];
        size_t count[8];
        const size_t m = std::min<size_t>(8, total - c);
        for (size_t k = 0; k < 8; k++) set[k] = allowed[c + std::min(k, m - 1)];
        countAllowed8(flatTouch_.data(), flatCost_.data(), flatTouch_.size(), all, set, count);
        std::copy(count, count + m, counts + c);
    }
}

std::vector<u64> GateDag::frontierSets(u64 allowed) const {
    refreshFlat();
    const size_t n = flatTouch_.size();
    const u64 *touch = flatTouch_.data(), *cost = flatCost_.data();
    const u64 all = numQubits_ >= 64 ? ~0ULL : ((1ULL << numQubits_) - 1);
    std::vector<u64> sets;
    u64 blocked = 0;
    for (size_t i = 0; i < n && blocked != all; i++) {
        if (touch[i] & blocked) {
            blocked |= touch[i];
            continue;
        }
        const u64 missing = cost[i] & ~allowed;
        if (missing) {
            if (std::find(sets.begin(), sets.end(), missing) == sets.end()) sets.push_back(missing);
            blocked |= touch[i];
        }
    }
    return sets;
}

std::vector<Gate> GateDag::takeAllowed(u64 allowed) {
    refreshFlat();
    std::vector<Gate> taken;
    const size_t n = flatTouch_.size();
    u64 blocked = 0;
    size_t kept = 0;
    for (size_t i = 0; i < n; i++) {
        if ((flatTouch_[i] & blocked) || (flatCost_[i] & ~allowed)) {
            blocked |= flatTouch_[i];
            flatTouch_[kept] = flatTouch_[i];
            flatCost_[kept] = flatCost_[i];
            flatNode_[kept++] = flatNode_[i];
        } else {
            Node &nd = nodes_[(size_t) flatNode_[i]];
            taken.push_back(nd.g);
            nd.alive = false;
            alive_--;
        }
    }
    flatTouch_.resize(kept);
    flatCost_.resize(kept);
    flatNode_.resize(kept);
    // the neighbour links are of use to add only, which renews them
    stale_ = merge_;
    if (remerge_) rebuild();
    return taken;
}

std::vector<Gate> GateDag::gatesInOrder() const {
    std::vector<Gate> out;
    for (const auto &n : nodes_)
        if (n.alive) out.push_back(n.g);
    return out;
}

}  // namespace dgq
