// Host planner: fusion of a circuit's ops into blocks (compiler.fuse_symbolic, fuse_frontier).
//
// No counterpart in the reference, which applies gate by gate (core/base_sim.py:30-53).
// Native because a new circuit pays for it before its first launch: with the planner in Python a
// compilation took 14 ms for 28 qubits at depth 20, 23 ms for a noisy 13-site circuit and 327 ms for 5000 random
// pairs, more than the passes that the frontier blocks save in one run; now 2.6, 2.6 and 32 ms.
#include <algorithm>
#include <cstdint>
#include <exception>
#include <vector>

#include "qgb_common.cuh"

namespace {

constexpr int kMaxBits = 2 * QGB_MAX_QUBITS;

struct BitSet {
    uint64_t w[2] = {0, 0};
    void add(int b) { w[b >> 6] |= uint64_t(1) << (b & 63); }
    bool has(int b) const { return (w[b >> 6] >> (b & 63)) & 1; }
    BitSet with(const BitSet& o) const { return BitSet{{w[0] | o.w[0], w[1] | o.w[1]}}; }
    bool meets(const BitSet& o) const { return (w[0] & o.w[0]) || (w[1] & o.w[1]); }
    bool within(const BitSet& o) const { return !(w[0] & ~o.w[0]) && !(w[1] & ~o.w[1]); }
    int size() const { return __builtin_popcountll(w[0]) + __builtin_popcountll(w[1]); }
};
static_assert(kMaxBits <= 128, "bit set");

struct Ops {  // op i: bits[begin[i] .. begin[i + 1])
    int count;
    const int32_t *begin, *bits;
    int size(int i) const { return begin[i + 1] - begin[i]; }
    int bit(int i, int j) const { return bits[begin[i] + j]; }
};

struct Block {
    BitSet set;
    std::vector<int> ops;
};

// Blocks in the ops' order: an op joins the latest block it depends on while the union stays within
// the width, and takes earlier blocks that the union covers and nothing in between touches.
std::vector<Block> in_order(const Ops& ops, int width) {
    std::vector<Block> blocks;
    std::vector<char> alive;
    int last[kMaxBits];
    std::fill(last, last + kMaxBits, -1);
    for (int i = 0; i < ops.count; ++i) {
        BitSet set;
        int deps[QGB_MAX_K * 4], nd = 0, cand = -1;
        for (int j = 0; j < ops.size(i); ++j) {
            const int b = ops.bit(i, j);
            set.add(b);
            if (last[b] >= 0) {
                cand = std::max(cand, last[b]);
                if (nd < int(sizeof(deps) / sizeof(int))) deps[nd++] = last[b];
            }
        }
        if (cand >= 0 && alive[size_t(cand)] && blocks[size_t(cand)].set.with(set).size() <= width) {
            Block& blk = blocks[size_t(cand)];
            blk.set = blk.set.with(set);
            blk.ops.push_back(i);
            for (int j = 0; j < ops.size(i); ++j) last[ops.bit(i, j)] = cand;
            std::sort(deps, deps + nd, [](int x, int y) { return x > y; });
            for (int d = 0; d < nd; ++d) {
                const int e = deps[d];
                if (e == cand || (d > 0 && deps[d - 1] == e)) continue;
                Block& from = blocks[size_t(e)];
                if (!alive[size_t(e)] || !from.set.within(blk.set)) continue;
                bool touched = false;
                for (int x = e + 1; x < cand && !touched; ++x) touched = alive[size_t(x)] && blocks[size_t(x)].set.meets(from.set);
                if (touched) continue;
                blk.ops.insert(blk.ops.begin(), from.ops.begin(), from.ops.end());
                alive[size_t(e)] = 0;
                for (int b = 0; b < kMaxBits; ++b)
                    if (from.set.has(b) && last[b] == e) last[b] = cand;
            }
            continue;
        }
        blocks.push_back(Block{set, {i}});
        alive.push_back(1);
        for (int j = 0; j < ops.size(i); ++j) last[ops.bit(i, j)] = int(blocks.size()) - 1;
    }
    std::vector<Block> out;
    for (size_t b = 0; b < blocks.size(); ++b)
        if (alive[b]) out.push_back(std::move(blocks[b]));
    return out;
}

// A set of bits and how far each has advanced through its ops.
struct Front {
    int bits[kMaxBits], size = 0;  // in the order they joined
    int pos[kMaxBits];             // next op of a member bit; -1: not a member
    Front() { std::fill(pos, pos + kMaxBits, -1); }
    void join(int b, int at) {
        bits[size++] = b;
        pos[b] = at;
    }
};

struct Grown {
    double total = 0;
    Front front;
    std::vector<int> ops;  // taken, in order
    BitSet seen;           // bits looked at
    bool valid = false;
};

struct Frontier {
    const Ops& ops;
    int width;
    std::vector<int> queue[kMaxBits];  // bit -> its ops in order, then -1
    std::vector<int> used;             // bits in order of first appearance
    int head[kMaxBits] = {};

    Frontier(const Ops& o, int w) : ops(o), width(w) {
        for (int i = 0; i < ops.count; ++i)
            for (int j = 0; j < ops.size(i); ++j) {
                const int b = ops.bit(i, j);
                if (queue[b].empty()) used.push_back(b);
                queue[b].push_back(i);
            }
        for (int b : used) queue[b].push_back(-1);
    }

    // In-order application on the front's bits from where they stand; the weight of the ops taken
    // (ops on several bits count, single-bit ops break ties).
    double take(Front& f, std::vector<int>& got) const {
        double total = 0;
        int work[kMaxBits], n = f.size;
        BitSet waiting;
        for (int j = 0; j < n; ++j) waiting.add(work[j] = f.bits[j]);
        while (n > 0) {
            const int b = work[--n];
            waiting.w[b >> 6] &= ~(uint64_t(1) << (b & 63));
            while (true) {
                const int i = queue[b][size_t(f.pos[b])];
                if (i < 0) break;
                bool ok = true;
                for (int j = 0; j < ops.size(i) && ok; ++j) {
                    const int y = ops.bit(i, j);
                    ok = f.pos[y] >= 0 && queue[y][size_t(f.pos[y])] == i;
                }
                if (!ok) break;
                got.push_back(i);
                total += ops.size(i) > 1 ? 1.0 : 1e-3;
                for (int j = 0; j < ops.size(i); ++j) {
                    const int y = ops.bit(i, j);
                    ++f.pos[y];
                    if (y != b && !waiting.has(y)) {
                        work[n++] = y;
                        waiting.add(y);
                    }
                }
            }
        }
        return total;
    }

    Grown grow(int start) const {
        Grown g;
        g.valid = true;
        for (int j = 0; j < ops.size(start); ++j) {
            const int b = ops.bit(start, j);
            g.front.join(b, head[b]);
            g.seen.add(b);
        }
        g.total = take(g.front, g.ops);
        Front f, best_front;
        std::vector<int> got, best_ops;
        while (g.front.size < width) {
            bool any = false;
            double best = 0;
            std::vector<BitSet> tried;
            int order[kMaxBits];
            std::copy(g.front.bits, g.front.bits + g.front.size, order);
            std::sort(order, order + g.front.size);
            for (int o = 0; o < g.front.size; ++o) {
                const int i = queue[order[o]][size_t(g.front.pos[order[o]])];
                if (i < 0) continue;
                BitSet set;
                int ext[kMaxBits], ne = 0;
                for (int j = 0; j < ops.size(i); ++j)
                    if (g.front.pos[ops.bit(i, j)] < 0) set.add(ext[ne++] = ops.bit(i, j));
                if (ne == 0 || g.front.size + ne > width) continue;
                if (std::any_of(tried.begin(), tried.end(), [&](const BitSet& t) { return t.within(set) && set.within(t); }))
                    continue;
                tried.push_back(set);
                std::sort(ext, ext + ne);
                f = g.front;
                for (int j = 0; j < ne; ++j) {
                    g.seen.add(ext[j]);
                    f.join(ext[j], head[ext[j]]);
                }
                got.clear();
                const double gain = take(f, got) / double(ne);
                if (!any || gain > best) {
                    any = true;
                    best = gain;
                    best_front = f;
                    best_ops.swap(got);
                }
            }
            if (!any) break;
            // (rounded before it is added, on every host: no fused multiply-add)
            const volatile double more = best * double(best_front.size - g.front.size);
            g.total += more;
            g.front = best_front;
            g.ops.insert(g.ops.end(), best_ops.begin(), best_ops.end());
        }
        return g;
    }

    // While ops are left: every op whose predecessors are done grows a set of bits, each time by the
    // bits of a next op that let the set take the most further ops per added bit; the best set
    // becomes a block. A set is kept while none of the bits it looked at has moved.
    std::vector<Block> run() {
        std::vector<Block> out;
        std::vector<Grown> cache = std::vector<Grown>(kMaxBits);  // by the start op's first bit
        int done = 0;
        while (done < ops.count) {
            Grown* best = nullptr;
            for (int b : used) {
                const int i = queue[b][size_t(head[b])];
                if (i < 0 || ops.bit(i, 0) != b) continue;
                bool ready = true;
                for (int j = 0; j < ops.size(i) && ready; ++j) ready = queue[ops.bit(i, j)][size_t(head[ops.bit(i, j)])] == i;
                if (!ready) continue;
                if (!cache[size_t(b)].valid) cache[size_t(b)] = grow(i);
                if (!best || cache[size_t(b)].total > best->total) best = &cache[size_t(b)];
            }
            out.emplace_back();
            out.back().ops = best->ops;
            done += int(best->ops.size());
            for (int j = 0; j < best->front.size; ++j) {
                const int b = best->front.bits[j];
                out.back().set.add(b);
                head[b] = best->front.pos[b];
            }
            for (int b : used)
                if (cache[size_t(b)].valid && cache[size_t(b)].seen.meets(out.back().set)) cache[size_t(b)].valid = false;
        }
        return out;
    }
};

std::vector<Block> frontier(const Ops& ops, int width) { return Frontier(ops, width).run(); }

// The same from the circuit's end.
std::vector<Block> frontier_back(const Ops& ops, int width) {
    std::vector<int32_t> begin(size_t(ops.count) + 1, 0), bits;
    for (int i = 0; i < ops.count; ++i) {
        const int o = ops.count - 1 - i;
        bits.insert(bits.end(), ops.bits + ops.begin[o], ops.bits + ops.begin[o + 1]);
        begin[size_t(i) + 1] = int32_t(bits.size());
    }
    std::vector<Block> out = frontier(Ops{ops.count, begin.data(), bits.data()}, width);
    std::reverse(out.begin(), out.end());
    for (Block& b : out) {
        std::reverse(b.ops.begin(), b.ops.end());
        for (int& i : b.ops) i = ops.count - 1 - i;
    }
    return out;
}

}  // namespace

extern "C" int qgb_plan_blocks(int method, const int32_t* begin, const int32_t* bits, int nops, int width,
                               int32_t* out_ops, int32_t* out_begin, int32_t* out_bits, int32_t* out_nbits) {
    using qgb_host::set_error;
    if (method < 0 || method > 2) return set_error(QGB_EINVAL, "planner method %d unknown", method);
    if (nops < 0 || width < 1 || (nops > 0 && (!begin || !bits || !out_ops || !out_begin || !out_bits || !out_nbits)))
        return set_error(QGB_EINVAL, "null or empty planner tables");
    for (int i = 0; i < nops; ++i) {
        const int k = begin[i + 1] - begin[i];
        if (begin[i] < 0 || k < 1 || k > width || k > 4 * QGB_MAX_K)
            return set_error(QGB_EINVAL, "op %d on %d bits, width %d", i, k, width);
        BitSet seen;
        for (int j = 0; j < k; ++j) {
            const int b = bits[begin[i] + j];
            if (b < 0 || b >= kMaxBits) return set_error(QGB_EINVAL, "op %d: bit %d out of range", i, b);
            if (seen.has(b)) return set_error(QGB_EINVAL, "op %d: repeated bit %d", i, b);
            seen.add(b);
        }
    }
    try {
        const Ops ops{nops, begin, bits};
        std::vector<Block> best = method == 1 ? frontier(ops, width) : in_order(ops, width);
        if (method == 2)  // the fewest, the first on ties
            for (auto* plan : {frontier, frontier_back}) {
                std::vector<Block> other = plan(ops, width);
                if (other.size() < best.size()) best.swap(other);
            }
        int at = 0;
        for (size_t b = 0; b < best.size(); ++b) {
            out_begin[b] = at;
            for (int i : best[b].ops) out_ops[at++] = i;
            int n = 0;
            for (int x = kMaxBits - 1; x >= 0; --x)
                if (best[b].set.has(x)) out_bits[b * size_t(width) + size_t(n++)] = x;
            out_nbits[b] = n;
        }
        if (!best.empty()) out_begin[best.size()] = at;
        return int(best.size());
    } catch (const std::exception&) {
        return set_error(QGB_EINVAL, "no memory for the planner");
    }
}
