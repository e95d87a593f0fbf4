// Upstream's array heaps (extension/inc/heapq.cuh:13-87) driven by one warp: the
// routines shared by the refinement kernel and the traversal for small batches.
#pragma once

#include "pa_common.cuh"

namespace pa {

constexpr unsigned kAll = 0xffffffffu;

// ---- upstream's heaps, 1-based {key, id} pairs, one warp ------------------------
struct __align__(8) HeapEntry {
    float k;
    int32_t v;
};

// h[1 .. n] is the heap (upstream index c lives at c + 1); h[n + 1] exists and is
// never meaningful: the pair load of the last parent may touch it.  Both children
// of node c sit in one aligned 16-byte pair at h + 2c.
//
// Upstream's routines walk from the root to a leaf, one dependent comparison per
// level.  Here the 32 lanes of the heap warp look at the five levels below the
// current node at once: lane l owns the l-th node of that sub-tree (heap order),
// compares its two children, a ballot collects the 31 decisions, every lane then
// tests with one mask compare whether its own node lies on the path those
// decisions describe, and a second ballot yields the path -- its highest set bit
// is the node five levels down.  Two such steps cover a heap of 1024 entries.  The
// keys along the path are then loaded one per lane and a ballot tells how far the
// moving key travels; the shift of the path is one store per lane.  The heap is
// not touched between the decisions and the stores, so the result is upstream's
// array, entry for entry (checked on the host against the oracle's routines over
// 2 M random operations at sizes 1 .. 4096, odd sizes included).

struct WalkLane {    // what a lane needs to know about its place in a 5-level sub-tree
    int depth, off;  // node = (root << depth) + off
    unsigned care, want;  // on the path iff (decisions & care) == want
};

__device__ __forceinline__ WalkLane walk_lane(int lane) {
    WalkLane L;
    const int r = lane + 1;
    L.depth = 31 - __clz(r);
    L.off = r - (1 << L.depth);
    L.care = L.want = 0;
#pragma unroll
    for (int t = 1; t <= 4; ++t) {
        if (t <= L.depth) {
            const int q = r >> t;  // ancestor; it has to point at (r >> (t - 1))
            L.care |= 1u << (q - 1);
            L.want |= static_cast<unsigned>((r >> (t - 1)) & 1) << (q - 1);
        }
    }
    return L;
}

// Leaf reached from the root by taking the larger (kLarger) or the smaller child
// at every node; the right child wins only if it exists and is strictly larger /
// smaller (heapq.cuh:17-21, 53-57).
template <bool kLarger>
__device__ __forceinline__ int warp_walk(const HeapEntry *h, int n, int lane, const WalkLane &L) {
    int a = 1;
    while (2 * a <= n) {
        const int node = (a << L.depth) + L.off;
        const bool valid = lane < 31 && node <= n;
        const bool has_child = valid && 2 * node <= n;
        bool right = false;
        if (has_child) {
            const int4 p = *reinterpret_cast<const int4 *>(h + 2 * node);
            const float lk = __int_as_float(p.x), rk = __int_as_float(p.z);
            right = (2 * node + 1 <= n) && (kLarger ? rk > lk : rk < lk);
        }
        const unsigned B = __ballot_sync(kAll, right);
        const unsigned HC = __ballot_sync(kAll, has_child);
        const unsigned P = __ballot_sync(kAll, valid && (B & L.care) == L.want);
        const int rs = 32 - __clz(P);  // deepest node of the path inside the sub-tree (P has bit 0)
        const int ds = 31 - __clz(rs);
        const int ns = (a << ds) + (rs - (1 << ds));
        a = ((HC >> (rs - 1)) & 1u) ? 2 * ns + static_cast<int>((B >> (rs - 1)) & 1u) : ns;
    }
    return a;
}

// heapq.cuh:13-29: the root sinks while a child is strictly smaller.  `me` takes
// the root's place first (callers have read the root if they need it).
__device__ __forceinline__ void warp_sink(HeapEntry *h, int n, HeapEntry me, int lane,
                                          const WalkLane &L) {
    const int leaf = warp_walk<false>(h, n, lane, L);
    const int D = 31 - __clz(leaf);       // path nodes below the root
    const bool on = lane < D;
    const int node = on ? leaf >> (D - 1 - lane) : 1;   // lane l: the path node at depth l + 1
    const HeapEntry e = h[node];
    const unsigned m = __ballot_sync(kAll, on && e.k < me.k);
    const int cnt = __ffs(~m) - 1;        // children that move up one level
    if (lane < cnt) h[node >> 1] = e;
    if (lane == 0) h[cnt == 0 ? 1 : leaf >> (D - cnt)] = me;
    __syncwarp();
}

// heapq.cuh:38-45
__device__ __forceinline__ HeapEntry warp_pop(HeapEntry *h, int n, int lane, const WalkLane &L) {
    const HeapEntry out = h[1];
    __syncwarp();
    warp_sink(h, n, HeapEntry{CUDART_INF_F, -1}, lane, L);
    return out;
}

// heapq.cuh:79-87
__device__ __forceinline__ void warp_pushpop(HeapEntry *h, int n, float k, int32_t v, int lane,
                                             const WalkLane &L) {
    if (k <= h[1].k) return;
    __syncwarp();
    warp_sink(h, n, HeapEntry{k, v}, lane, L);
}

// heapq.cuh:47-77: the leaf at the end of the larger-child walk is replaced if the
// new key is smaller, then sifted up while the parent is strictly larger.
__device__ __forceinline__ void warp_replace(HeapEntry *h, int n, float k, int32_t v, int lane,
                                             const WalkLane &L) {
    const int leaf = warp_walk<true>(h, n, lane, L);
    if (k >= h[leaf].k) return;
    const int D = 31 - __clz(leaf);
    const bool on = lane < D;
    const HeapEntry e = h[on ? leaf >> (lane + 1) : 1];  // lane l: the ancestor l + 1 levels up
    const unsigned m = __ballot_sync(kAll, on && e.k > k);
    const int cnt = __ffs(~m) - 1;        // ancestors that move down one level
    if (lane < cnt) h[leaf >> lane] = e;
    if (lane == 0) h[leaf >> cnt] = HeapEntry{k, v};
    __syncwarp();
}

// The same operations with the outcome of every comparison kept: bit n of a set of
// words (uniform over the warp, in registers) says whether the right child of node n
// is strictly larger (open heap) or smaller (result heap).  The walk is then a few
// integer instructions instead of two rounds of loads and ballots; lane t looks at the
// path node at depth t + 1, its parent and its sibling, and says whether the bit of
// the parent (depth t) turns.  Heaps of up to 64 W nodes.
template <int W> struct PathBits {
    static constexpr int kUniform = W > 4 ? 2 : W;  // words every lane holds
    uint32_t w[kUniform];
    uint32_t deep;  // W = 8: lane i holds word i (six registers less, two shuffles more)

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < kUniform; ++i) w[i] = 0;
        deep = 0;
    }
    template <bool kLarger>
    __device__ __forceinline__ void build(const HeapEntry *h, int n, int lane) {
        deep = 0;
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const int node = 32 * i + lane;
            bool right = false;
            if (node >= 1 && 2 * node + 1 <= n) {
                const int4 p = *reinterpret_cast<const int4 *>(h + 2 * node);
                const float lk = __int_as_float(p.x), rk = __int_as_float(p.z);
                right = kLarger ? rk > lk : rk < lk;
            }
            const uint32_t word = __ballot_sync(kAll, right);
            if (i < kUniform) w[i < kUniform ? i : 0] = word;
            else if (lane == i) deep = word;
        }
    }
    __device__ __forceinline__ void build_larger(const HeapEntry *h, int n, int lane) {
        build<true>(h, n, lane);
    }
    __device__ __forceinline__ void build_smaller(const HeapEntry *h, int n, int lane) {
        build<false>(h, n, lane);
    }
    // The leaf at the end of the path in a heap of n nodes.  All nodes of the first kSure
    // levels below the root exist for every n that comes with this many words.
    __device__ __forceinline__ int leaf(int n) const {
        constexpr int kDepth = W == 1 ? 6 : W == 2 ? 7 : W == 4 ? 8 : 9;
        constexpr int kSure = W == 1 ? 3 : W == 2 ? 4 : W == 4 ? 6 : 7;
        unsigned a = 1;
#pragma unroll
        for (int l = 0; l < kDepth; ++l) {
            uint32_t word = 0;
            if (l < 5) word = w[0];
            if (l == 5 && W >= 2) word = w[W >= 2 ? 1 : 0];
            if (l == 6 && W == 4) word = (a & 32u) ? w[W == 4 ? 3 : 0] : w[W == 4 ? 2 : 0];
            if ((l == 6 || l == 7) && W == 8) word = __shfl_sync(kAll, deep, a >> 5);
            const unsigned c = (a << 1) | (__funnelshift_r(word, 0u, a) & 1u);
            a = l < kSure || 2 * a <= static_cast<unsigned>(n) ? c : a;
        }
        return static_cast<int>(a);
    }
    // Turns the bits of the path's nodes for which the lane of their depth says so.
    __device__ __forceinline__ void turn(bool flip, int leaf, int depth, int lane) {
        const unsigned F = __ballot_sync(kAll, flip);
        w[0] ^= __reduce_or_sync(kAll, flip && lane < 5 ? 1u << ((leaf >> (depth - lane)) & 31) : 0u);
        auto node = [&](int t) { return leaf >> ((depth - t) & 31); };  // of the path, at depth t
        auto bit = [&](int t) { return ((F >> t) & 1u) << (node(t) & 31); };
        if constexpr (W >= 2) w[1] ^= bit(5);
        if constexpr (W == 4) {
            w[2] ^= (node(6) & 32) ? 0u : bit(6);
            w[3] ^= (node(6) & 32) ? bit(6) : 0u;
        }
        if constexpr (W == 8) {
            deep ^= lane == node(6) >> 5 ? bit(6) : 0u;
            deep ^= lane == node(7) >> 5 ? bit(7) : 0u;
        }
    }
};

// What lane t sees of a path: the node at depth t + 1 and its sibling's key.
struct PathLane {
    int depth, node;
    bool on, sib;  // the path reaches this lane; the node has a sibling
    float sk;
};
__device__ __forceinline__ PathLane path_lane(const HeapEntry *h, int n, int leaf, int lane) {
    PathLane p;
    p.depth = 31 - __clz(leaf);
    p.on = lane < p.depth;
    p.node = p.on ? leaf >> (p.depth - 1 - lane) : 2;
    p.sib = p.on && (p.node | 1) <= n;
    p.sk = h[p.sib ? p.node ^ 1 : p.node].k;
    return p;
}

// warp_sink over the bits of the smaller children (result heap).
template <int W>
__device__ __forceinline__ void bit_sink(HeapEntry *h, int n, HeapEntry me, PathBits<W> &smaller,
                                         int lane) {
    const int leaf = smaller.leaf(n);
    const PathLane p = path_lane(h, n, leaf, lane);
    const HeapEntry e = h[p.node];
    const unsigned m = __ballot_sync(kAll, p.on && e.k < me.k);
    const int cnt = __ffs(~m) - 1;
    const float below = __shfl_down_sync(kAll, e.k, 1);
    const float nk = lane + 1 == cnt ? me.k : below;  // the node's new key (lane < cnt)
    __syncwarp();
    if (lane < cnt) h[p.node >> 1] = e;
    if (lane == 0) h[cnt == 0 ? 1 : leaf >> (p.depth - cnt)] = me;
    // the path went to the node: right if strictly smaller than its sibling
    const bool stays = (p.node & 1) ? nk < p.sk : !(p.sk < nk);
    smaller.turn(lane < cnt && p.sib && !stays, leaf, p.depth, lane);
    __syncwarp();
}

// warp_pop of a heap with the bits of its larger children (open heap).
template <int W>
__device__ __forceinline__ HeapEntry bit_pop(HeapEntry *h, int n, PathBits<W> &larger, int lane,
                                             const WalkLane &L) {
    const HeapEntry out = h[1];
    const int leaf = warp_walk<false>(h, n, lane, L);
    const PathLane p = path_lane(h, n, leaf, lane);
    const HeapEntry e = h[p.node];
    const unsigned m = __ballot_sync(kAll, p.on && e.k < CUDART_INF_F);
    const int cnt = __ffs(~m) - 1;
    const float below = __shfl_down_sync(kAll, e.k, 1);
    const float nk = lane + 1 == cnt ? CUDART_INF_F : below;
    __syncwarp();
    if (lane < cnt) h[p.node >> 1] = e;
    if (lane == 0) h[cnt == 0 ? 1 : leaf >> (p.depth - cnt)] = HeapEntry{CUDART_INF_F, -1};
    const bool was = (p.node & 1) ? e.k > p.sk : p.sk > e.k;
    const bool is = (p.node & 1) ? nk > p.sk : p.sk > nk;
    larger.turn(lane < cnt && p.sib && was != is, leaf, p.depth, lane);
    __syncwarp();
    return out;
}

// warp_replace over the bits of the larger children (open heap): what lies along the
// path first -- it depends on the heap only -- then the second half for an entry that is
// below the key of the leaf.
struct ReplaceLane {
    PathLane p;
    HeapEntry e;  // the parent of the path node
    float limit;  // key of the leaf
};
__device__ __forceinline__ ReplaceLane bit_replace_load(const HeapEntry *h, int n, int leaf, int lane) {
    ReplaceLane r;
    r.p = path_lane(h, n, leaf, lane);
    r.e = h[r.p.node >> 1];
    r.limit = h[leaf].k;
    return r;
}
template <int W>
__device__ __forceinline__ void bit_replace_apply(HeapEntry *h, int leaf, const ReplaceLane &r,
                                                  float k, int32_t v, PathBits<W> &larger, int lane) {
    const PathLane &p = r.p;
    const unsigned m = __ballot_sync(kAll, p.on && r.e.k > k);
    const int s = m != 0 ? __ffs(m) - 1 : p.depth;  // depth at which the new entry lands
    const bool moves = p.on && lane >= s;
    __syncwarp();
    if (moves) h[p.node] = r.e;
    if (lane == 0) h[leaf >> (p.depth - s)] = HeapEntry{k, v};
    const float nk = moves ? r.e.k : k;  // the node's new key (lane >= s - 1)
    const bool stays = (p.node & 1) ? nk > p.sk : !(p.sk > nk);
    larger.turn(p.sib && lane + 1 >= s && !stays, leaf, p.depth, lane);
    __syncwarp();
}
template <int W>
__device__ __forceinline__ void bit_replace(HeapEntry *h, int n, float k, int32_t v,
                                            PathBits<W> &larger, int lane) {
    const int leaf = larger.leaf(n);
    const ReplaceLane r = bit_replace_load(h, n, leaf, lane);
    if (k >= r.limit) return;
    bit_replace_apply(h, leaf, r, k, v, larger, lane);
}

// 32 E entries, ascending by key, entry lane * E + e in element e of the lane (a bitonic
// network in registers; equal keys in no particular order).
template <int E>
__device__ __forceinline__ void warp_sort(float (&k)[E], int32_t (&v)[E], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * E; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= E) {
                const int across = stride / E;
                const bool lower = (lane & across) == 0;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const float ok = __shfl_xor_sync(kAll, k[e], across);
                    const int32_t ov = __shfl_xor_sync(kAll, v[e], across);
                    const bool up = ((lane * E + e) & size) == 0;
                    const bool take = lower == up ? ok < k[e] : ok > k[e];
                    k[e] = take ? ok : k[e];
                    v[e] = take ? ov : v[e];
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int f = e ^ stride;
                    if ((e & stride) != 0) continue;
                    const bool up = ((lane * E + e) & size) == 0;
                    const bool swap = up ? k[e] > k[f] : k[e] < k[f];
                    const float tk = k[e];
                    const int32_t tv = v[e];
                    k[e] = swap ? k[f] : tk;
                    v[e] = swap ? v[f] : tv;
                    k[f] = swap ? tk : k[f];
                    v[f] = swap ? tv : v[f];
                }
            }
        }
    }
}

// Whether a heap of 32 E nodes shows entries equal to their parents (empty ones, -inf, aside), in
// two lanes at least: a single pair is chance, and where equal keys are common many stand
// so, since a sinking key stops above its equal.
template <int E, class Key>
__device__ __forceinline__ bool heap_shows_twins(int lane, Key key_of) {
    bool twins = false;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int node = 32 * e + lane + 1;
        const float k = key_of(node);
        twins = twins || (node > 1 && k == key_of(max(node >> 1, 1)) && k > -CUDART_INF_F);
    }
    return __popc(__ballot_sync(kAll, twins)) >= 2;
}

// Whether two neighbours of the sorted entries from position `from` on (or the first of
// them and the one in front of it) have equal keys; empty entries (id -1) are alike.
template <int E>
__device__ __forceinline__ bool warp_has_twins(const float (&k)[E], const int32_t (&v)[E], int from,
                                               int lane) {
    const float first_k = __shfl_down_sync(kAll, k[0], 1);
    const int32_t first_v = __shfl_down_sync(kAll, v[0], 1);
    bool twins = false;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = lane * E + e;
        const float nk = e + 1 < E ? k[e + 1 < E ? e + 1 : 0] : first_k;
        const int32_t nv = e + 1 < E ? v[e + 1 < E ? e + 1 : 0] : first_v;
        twins = twins || (i + 1 >= from && i + 1 < 32 * E && k[e] == nk && (v[e] >= 0 || nv >= 0));
    }
    return __any_sync(kAll, twins);
}

}  // namespace pa
