// Refinement of the candidate handoff on the GPU: the two stages upstream runs on
// the CPU in `traverse_refine` (extension/traverse_cpu.cpp:261-369), each of them
// one call of `traverse_cpu_kernel` (:12-163):
//
//   stage 2  the [batch, 4 * ef] candidates of the reduced-space traversal get
//            their distances completed over dims d_principle .. d_model (:41-62),
//            seed a best-first search on the SUB-graph that is cut off after
//            REFINE_STEP = 2 expansions (:64-136), and the best H of candidates
//            and newly found nodes are written back, ascending, behind (-1, -inf)
//            pads (:138-162);
//   stage 3  the same search, seeded with the stage-2 result, on the FULL graph
//            with full-dimension distances, up to 2 * ef expansions, top-k out.
//
// The candidates are consumed where the traversal left them, in HBM; nothing of
// the handoff crosses PCIe.  One CTA of five warps (three for rows of at most 512
// bytes; sixteen or eight while the SMs have few queries) per query, persistent:
// CTA i owns slot i of the visited-set pool (visited.cu), starts on query i and
// claims further queries from a counter.
// Warp 0 is the heap warp, the other warps gather: adjacency row, visited marks,
// vector rows, distances.  Four serial pieces of upstream's routine -- the result
// heap, pushing the seeds into the open heap of the two-expansion stage, seeding the
// full-graph stage, merging seeds and result -- are computed from their outcome when
// the keys involved are pairwise different (TopList, brief_search, the seeding in
// heap_loop, select_sort_output and merge_sorted_output) and run as upstream wrote
// them otherwise.  In the full-graph stage the two sides overlap: the node the next
// pop will return is known as soon as the distances of the current expansion are
// (it is the better of the open heap's root and the best new neighbour -- a new
// key below the root always sifts up to the root, equal keys never pass it), so
// the gather warps start on that node while the heap warp still inserts the
// current expansion's neighbours and pops.  The pop then either confirms the
// node or ends the search (when the best new neighbour is not admitted to the
// heaps the next pop fails the stop test), in which case the speculative marks
// are never looked at again.  The sub-graph stage does not speculate: its marks
// are inherited by the full-graph stage.  Semantics are upstream's, operation
// for operation:
//   * the open heap (2H entries) is upstream's array heap with upstream's routines
//     (extension/inc/heapq.cuh:13-87) -- heap_replace evicts the leaf reached by
//     walking larger children, not the maximum, so the layout is part of the
//     result; it lives in shared memory, stored 1-based as {key, id} pairs so that
//     both children of a node come in one 16-byte load, and is driven by the 32
//     lanes of the heap warp together (see the routines below).  So does the result
//     heap (H entries) where H > 256, and for queries with several equal distances or a
//     NaN (finish_query); the others' results are a sorted list in registers (TopList);
//   * H follows upstream's CPU dispatch (traverse_cpu.cpp:228-254);
//   * exact visited marks (extension/inc/bitmask.hpp:12-45) shared by the two
//     stages of a query, as upstream shares one marker between them;
//   * neighbours are taken in row order, a row ends at its first negative id.
// Distances: one warp per vector row, lane t owns floats [128m + 4t, +4),
// acc += fma(dx,dx,dy*dy); acc += fma(dz,dz,dw*dw) in ascending m, butterfly
// 16..1.  Upstream's AVX2 order (eight running sums, built with -ffast-math)
// differs from this in the last bits, so results agree with upstream's within a
// relative 1e-5 and with the CPU oracle, which restates this order, bit for bit.
#include "pa_common.cuh"
#include "warp_heap.cuh"

namespace pa {

// Warp 0 runs the heaps, the other warps gather.  Where the SMs are full the kernel has
// up to five warps (wider CTAs: refine_launch_for); vector rows of at most 512 bytes are served by two gather warps
// (96 threads), which lets twelve instead of seven queries share an SM -- at those
// sizes the heap warp, not the gather, sets the pace of a query -- or by three when
// the batch leaves room for them (nine queries per SM).
#ifndef PA_REFINE_WIDE_THREADS
#define PA_REFINE_WIDE_THREADS 160
#endif
#ifndef PA_REFINE_NARROW_THREADS
#define PA_REFINE_NARROW_THREADS 96
#endif
#ifndef PA_REFINE_NARROW_DIM
#define PA_REFINE_NARROW_DIM 128
#endif
constexpr int kRefThreads = 160;  // what that kernel is compiled for
constexpr int kRefThreadsWide = PA_REFINE_WIDE_THREADS;
constexpr int kRefThreadsNarrow = PA_REFINE_NARROW_THREADS;
constexpr int kNarrowMaxDim = PA_REFINE_NARROW_DIM;
static_assert(kRefThreadsWide <= kRefThreads && kRefThreadsNarrow <= kRefThreads &&
                  kRefThreadsNarrow >= 64 && kRefThreadsWide % 32 == 0 && kRefThreadsNarrow % 32 == 0,
              "a heap warp plus one to four gather warps");
__host__ __device__ inline int ref_threads_for(int d) {
    return d <= kNarrowMaxDim ? kRefThreadsNarrow : kRefThreadsWide;
}
#ifndef PA_REFINE_MIN_CTAS
#define PA_REFINE_MIN_CTAS 7
#endif
// PA_REFINE_PROFILE (experiments only): 1 = thread 0 (heap warp) accumulates clock
// deltas per phase into stats[b * 24 + 4 ..] and thread 32 (first gather warp) into
// stats[b * 24 + 12 ..]; 2 = thread 32 only.  The stats rows are then 24 ints wide.
// A clock read may still move across a barrier, so a wait can land in the
// neighbouring phase's count; and the heap warp's own clocks slow its heap routines
// several times over while the gather warps run beside it -- read the heap warp's
// cost from mode 2 (how long the gather warps wait for it).
#ifndef PA_REFINE_PROFILE
#define PA_REFINE_PROFILE 0
#endif
#if PA_REFINE_PROFILE
__device__ __forceinline__ long long pinned_clock() {
    long long t;
    asm volatile("mov.u64 %0, %%clock64;" : "=l"(t)::"memory");
    return t;
}
#define PA_TICK(slot) do { if (PA_REFINE_PROFILE == 1 && threadIdx.x == 0) { const long long now__ = pinned_clock(); prof[slot] += static_cast<int>(now__ - prof_t); prof_t = now__; } } while (0)
#define PA_GTICK(slot) do { if (threadIdx.x == 32) { const long long now__ = pinned_clock(); prof[slot] += static_cast<int>(now__ - prof_t); prof_t = now__; } } while (0)
#else
#define PA_TICK(slot) do { } while (0)
#define PA_GTICK(slot) do { } while (0)
#endif
constexpr int kMaxDegree = 64;

struct RefGraph {
    const int32_t *nbr;     // neighbour ids
    const int32_t *row_of;  // node -> row, or nullptr when the row is the node id
    int64_t row_stride;     // ints between rows
    int elem_stride;        // ints between the ids of a row
    int degree;             // slots per row
};

struct RefineArgs {
    const int64_t *cand_I;  // [batch, n_cand]
    const float *cand_D;
    const float *query;     // [batch, ldq] full rotated queries
    int64_t ldq;
    const float *storage;   // [n_nodes, d] full vectors
    int64_t n_nodes;
    int d, d_p;
    RefGraph sub, full;
    int n_cand, ef, H, k, stages, batch;
    int64_t *out_I;         // stages 2: [batch, n_cand]; stages 3: [batch, k]
    float *out_D;
    uint8_t *marks;         // visited pool: slot s at marks + s * slot_stride
    int32_t *epoch;         // [slots] last marker used by the slot
    unsigned *claim;        // queries handed out beyond each CTA's first, this launch
    int64_t slot_stride;
    int slot_begin;
    int32_t *stats;         // nullptr or [batch, 4]
};

// ---- the H best results, in the registers of the heap warp -----------------------
// Upstream keeps them in an array heap (heap_pushpop, heapq.cuh:79-87).  With pairwise
// different distances its layout is never seen: a push drops the worst entry, the root
// is the largest distance, and the pops of the end come out sorted.  So up to 256 of
// them are held sorted, ascending, in registers (position i of the list in slot
// i + 32 R - H, slot s in register s / 32 of lane s mod 32; the slots before hold -inf
// and never move): an insertion is one rotation by a lane per register, about 70 cycles
// where heap_pushpop took 600 to 900.  Where distances are equal the layout decides
// which of two entries is dropped or comes first; the admitted entries are logged in
// shared memory, and a merge that meets equal distances among the entries that matter
// replays the log through heap_pushpop (search_stage).
//
// What it gave, with the open heap's comparison bits (PathBits) and the merge of two
// sorted lists: the launch in ms, heaps as arrays -> now: 1024 queries of 768 dimensions
// at ef 128 2.29 -> 2.11, 8192 of them 16.1 -> 15.4; 96 dimensions at ef 256: 1024 2.81 ->
// 1.99, 16384 13.5 -> 12.3; 200 dimensions at ef 192, k 100: 1024 2.29 -> 1.97; seven
// queries of 96 dimensions at ef 96 0.40 -> 0.31.
template <int R> struct TopList {
    float k[R];
    int32_t v[R];

    __device__ __forceinline__ void clear(int H, int lane) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            k[r] = 32 * r + lane < 32 * R - H ? -CUDART_INF_F : CUDART_INF_F;
            v[r] = -1;
        }
    }
    __device__ __forceinline__ float worst() const { return __shfl_sync(kAll, k[R - 1], 31); }
    // The last entry leaves; true if the one before it is its equal.
    __device__ __forceinline__ bool worst_twice(float worst_k) const {
        return __shfl_sync(kAll, k[R - 1], 30) == worst_k;
    }
    __device__ __forceinline__ void insert(float nk, int32_t nv, int lane) {
        // downwards, so that few rotated copies are alive at a time
        const int from = (lane + 31) & 31;
        float pk = __shfl_sync(kAll, k[R - 1], from);
        int32_t pv = __shfl_sync(kAll, v[R - 1], from);
#pragma unroll
        for (int r = R - 1; r >= 0; --r) {
            const float below_k = r > 0 ? __shfl_sync(kAll, k[r > 0 ? r - 1 : 0], from) : -CUDART_INF_F;
            const int32_t below_v = r > 0 ? __shfl_sync(kAll, v[r > 0 ? r - 1 : 0], from) : -1;
            // the entry one position before this one
            const float qk = lane != 0 ? pk : below_k;
            const int32_t qv = lane != 0 ? pv : below_v;
            if (k[r] > nk) {
                v[r] = qk > nk ? qv : nv;
                k[r] = qk > nk ? qk : nk;
            }
            pk = below_k;
            pv = below_v;
        }
    }
};

// Words of comparison bits of a result heap where the open heap, twice as large, has R.
__host__ __device__ constexpr int result_words(int R) { return R >= 4 ? R / 2 : 1; }

// Registers per lane of the list for a capacity of H; 0: the array heap is used.
__host__ __device__ constexpr int list_regs_for(int H) {
    return H <= 64 ? 2 : H <= 128 ? 4 : H <= 256 ? 8 : 0;
}

// ---- distances: one warp per row, two rows in flight ----------------------------
__device__ __forceinline__ float ref_stripe(float acc, float4 c, float4 p) {
    const float dx = __fsub_rn(c.x, p.x), dy = __fsub_rn(c.y, p.y);
    const float dz = __fsub_rn(c.z, p.z), dw = __fsub_rn(c.w, p.w);
    acc = __fadd_rn(acc, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
    return __fadd_rn(acc, __fmaf_rn(dz, dz, __fmul_rn(dw, dw)));
}

__device__ __forceinline__ float butterfly(float acc) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(kAll, acc, off));
    return acc;
}

// Squared distances of the query to rows r0 and r1 over dims [from, d); every lane
// returns both sums.  Three stripes of each row are loaded before any arithmetic.
__device__ __forceinline__ void two_rows(const float *__restrict__ r0, const float *__restrict__ r1,
                                         const float *q_s, int d, int from, int lane, float &o0,
                                         float &o1) {
    float a0 = 0.0f, a1 = 0.0f;
    for (int o = from + 4 * lane; o < d; o += 384) {
        float4 x0[3], x1[3];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const bool in = o + 128 * m < d;
            x0[m] = in ? __ldg(reinterpret_cast<const float4 *>(r0 + o + 128 * m))
                       : make_float4(0, 0, 0, 0);
            x1[m] = in ? __ldg(reinterpret_cast<const float4 *>(r1 + o + 128 * m))
                       : make_float4(0, 0, 0, 0);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            if (o + 128 * m < d) {
                const float4 qa = *reinterpret_cast<const float4 *>(q_s + o + 128 * m);
                a0 = ref_stripe(a0, qa, x0[m]);
                a1 = ref_stripe(a1, qa, x1[m]);
            }
        }
    }
    o0 = butterfly(a0);
    o1 = butterfly(a1);
}

// One row over dims [from, d) with six stripes (768 floats) loaded before any
// arithmetic: a row of up to 3 KB makes a single round trip.  Same order of
// additions as two_rows.
__device__ __forceinline__ float one_row(const float *__restrict__ r0, const float *q_s, int d,
                                         int from, int lane) {
    float a0 = 0.0f;
    for (int o = from + 4 * lane; o < d; o += 768) {
        float4 x0[6];
#pragma unroll
        for (int m = 0; m < 6; ++m)
            x0[m] = o + 128 * m < d ? __ldg(reinterpret_cast<const float4 *>(r0 + o + 128 * m))
                                    : make_float4(0, 0, 0, 0);
#pragma unroll
        for (int m = 0; m < 6; ++m)
            if (o + 128 * m < d)
                a0 = ref_stripe(a0, *reinterpret_cast<const float4 *>(q_s + o + 128 * m), x0[m]);
    }
    return butterfly(a0);
}

// A third row rides along without registers: cp.async copies it into the warp's
// own staging buffer while the two register rows make their round trips; every
// lane later reads back exactly the 16-byte pieces it copied itself.
__device__ __forceinline__ void row_to_stage(float *stage, const float *__restrict__ row, int d,
                                             int from, int lane) {
    for (int o = from + 4 * lane; o < d; o += 128) {
        const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(stage + o));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(row + o) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ float staged_row(const float *stage, const float *q_s, int d, int from,
                                            int lane) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float a = 0.0f;
    for (int o = from + 4 * lane; o < d; o += 128)
        a = ref_stripe(a, *reinterpret_cast<const float4 *>(q_s + o),
                       *reinterpret_cast<const float4 *>(stage + o));
    return butterfly(a);
}

// Seeds completed over a few trailing dimensions, at most 4 G of them: G lanes have a
// row in one load, so a warp takes 32 / G rows at a time and has four such sets in flight.
// The lanes that the order of additions above would leave idle only ever add zero, so the
// butterfly over G lanes gives the same bits.  32 of 96 dimensions, a warp per row / four
// rows per warp, ms: 16384 queries at ef 256 12.2 / 11.1, 2000 at ef 128 1.63 / 1.49, 1024 at
// ef 256 1.97 / 1.93, seven at ef 96 0.276 / 0.259.
template <int G>
__device__ __forceinline__ void short_residuals(const float *__restrict__ storage, const float *q,
                                                const int32_t *c_id, float *c_d, int n_seed, int d,
                                                int from, int w, int n_w, int lane) {
    const int t = lane & (G - 1);
    const bool in = from + 4 * t < d;
    const float4 qa = in ? *reinterpret_cast<const float4 *>(q + from + 4 * t) : make_float4(0, 0, 0, 0);
    const int step = n_w * (32 / G);  // seeds of one set over all warps
    for (int base = w * (32 / G); base < n_seed; base += 4 * step) {
        float4 x[4];
        int id[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int i = base + m * step + lane / G;
            id[m] = i < n_seed ? c_id[i] : -1;
            x[m] = in && id[m] >= 0
                ? __ldg(reinterpret_cast<const float4 *>(storage + static_cast<int64_t>(id[m]) * d + from + 4 * t))
                : make_float4(0, 0, 0, 0);
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            float acc = in ? ref_stripe(0.0f, qa, x[m]) : 0.0f;
#pragma unroll
            for (int off = G / 2; off > 0; off >>= 1)
                acc = __fadd_rn(acc, __shfl_xor_sync(kAll, acc, off));
            const int i = base + m * step + lane / G;
            if (t == 0 && id[m] >= 0) c_d[i] = __fadd_rn(c_d[i], acc);
        }
    }
}

struct RefShared {
    float *q;          // [d]
    HeapEntry *open;   // [2H + 2]
    HeapEntry *buf;    // [H + 2] result heap; with the result list in registers: the first
                       //         H entries of the log, the list once the stage is over
    int32_t *c_id;     // [n_cand] seeds of the running stage, then its output
    float *c_d;
    int32_t *nb_id;    // [2][kMaxDegree] unvisited neighbours of an expanded node
    float *nb_d;       //                 (two expansions are in flight)
    float *stage;      // [warps][d] one staged vector row per warp
};

// What the heap warp publishes after a pop, and the gather side's guess.
struct RefCtl {
    unsigned long long m1, m2;  // brief_search: the two smallest seeds, key bits << 32 | index
    int c1, c2;                 //               other seeds with the same distances
    int pop_u[2];       // node popped for expansion i (slot i & 1), -1: the search ends
    float root_k[2];    // open heap's root right after that pop
    int root_v[2];
    int guess[2];       // node the gather warps prepared expansion i for
    int n_new[2];       // unvisited neighbours found for expansion i
    int tie;            // the merge gave up: run upstream's sequence
    unsigned next;      // the query claimed for the CTA's next round
    int sorted;         // the stage's output: kAscending | kHeadStrict
    int n_taken, n_equal;
    int marker;
    float amb;          // TopList: smallest distance of which one of several was dropped
    int n_log;          //          entries admitted
    int st[4];          // expansions and evaluations of the two stages
    int rerun;          //          the query has to be run on the array heaps
    int half;           // the first stage stands, the second shall be run on the array heaps
    int tied;           // equal neighbours in the first stage's output, where its merge gave up
#if PA_REFINE_PROFILE
    int heap_prof[12];      // thread 0's phases on their way in and out of heap_side
    long long heap_clock;
    int phases[2][12];      // of threads 0 and 32 on their way to finish_query
    long long clock[2];
#endif
};
constexpr int kAscending = 1;   // the real entries ascend
constexpr int kHeadStrict = 2;  // the first kSeedHead of them strictly
constexpr int kManyTied = 2;    // RefCtl::tied from which on more are expected
constexpr int kSeedHead = 26;   // entries the seeding of the open heap may look at

// Every thread of the CTA, whichever side of the warp specialisation it is on.
__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 0;" ::: "memory"); }

__device__ __forceinline__ void gather_sync() {  // the gather warps only
    asm volatile("bar.sync 1, %0;" ::"r"(static_cast<int>(blockDim.x) - 32) : "memory");
}

// The gather half of one expansion (traverse_cpu.cpp:105-135 without the heap
// updates): the row of u in order up to its first negative id, unvisited ids
// marked and compacted in row order into buffer p, their full-dimension distances.
// Called by all gather warps.
__device__ __forceinline__ void gather_node(const RefineArgs &A, const RefShared &S,
                                            const RefGraph &G, uint8_t *vis, uint8_t marker,
                                            RefCtl *ctl, int u, int p, int gw, int lane, int *prof,
                                            long long &prof_t) {
    (void)prof; (void)prof_t;
    PA_GTICK(0);  // since the last tick: prediction, barriers, waiting for the heap warp
    int32_t *nb_id = S.nb_id + p * kMaxDegree;
    float *nb_d = S.nb_d + p * kMaxDegree;
    const int d = A.d;
    if (gw == 0) {
        const int64_t row = G.row_of != nullptr ? __ldg(G.row_of + u) : u;
        int count = 0;
        bool ended = row < 0;
        for (int c = 0; c < G.degree; c += 32) {
            const int slot = c + lane;
            int v = -1;
            if (!ended && slot < G.degree)
                v = __ldg(G.nbr + row * G.row_stride + static_cast<int64_t>(slot) * G.elem_stride);
            const unsigned end_mask = __ballot_sync(kAll, v < 0 && v != kDupTag);
            PA_GTICK(1);  // adjacency row
            const int first_end = end_mask ? __ffs(end_mask) - 1 : 32;
            const bool live = lane < first_end && v >= 0;
            bool fresh = false;
            if (live) {
                fresh = vis[v] != marker;
                if (fresh) vis[v] = marker;
            }
            const unsigned m = __ballot_sync(kAll, fresh);
            if (fresh) nb_id[count + __popc(m & ((1u << lane) - 1u))] = v;
            count += __popc(m);
            ended = ended || end_mask != 0;
        }
        if (lane == 0) ctl->n_new[p] = count;
    }
    PA_GTICK(5);  // visited bytes
    gather_sync();
    PA_GTICK(2);
    const int n_new = ctl->n_new[p];
    float *stage = S.stage + (gw + 1) * d;
    const int n_gw = static_cast<int>(blockDim.x >> 5) - 1;  // gather warps
    if (d > 384) {
        // two rows per warp and trip, each in one round trip: one through registers,
        // one staged by cp.async
        for (int j = gw; j < n_new; j += 2 * n_gw) {
            const int j1 = j + n_gw;
            if (j1 < n_new) row_to_stage(stage, A.storage + static_cast<int64_t>(nb_id[j1]) * d, d, 0, lane);
            const float r0 = one_row(A.storage + static_cast<int64_t>(nb_id[j]) * d, S.q, d, 0, lane);
            float r1 = 0.0f;
            if (j1 < n_new) r1 = staged_row(stage, S.q, d, 0, lane);
            if (lane == 0) {
                nb_d[j] = r0;
                if (j1 < n_new) nb_d[j1] = r1;
            }
        }
        PA_GTICK(3);  // vector rows
        return;
    }
    // short rows, three per warp and trip: two through registers, one staged
    for (int j = gw; j < n_new; j += 3 * n_gw) {
        const int j1 = j + n_gw, j2 = j + 2 * n_gw;
        const int v0 = nb_id[j], v1 = j1 < n_new ? nb_id[j1] : v0;
        if (j2 < n_new) row_to_stage(stage, A.storage + static_cast<int64_t>(nb_id[j2]) * d, d, 0, lane);
        float r0, r1;
        two_rows(A.storage + static_cast<int64_t>(v0) * d, A.storage + static_cast<int64_t>(v1) * d,
                 S.q, d, 0, lane, r0, r1);
        float r2 = 0.0f;
        if (j2 < n_new) r2 = staged_row(stage, S.q, d, 0, lane);
        if (lane == 0) {
            nb_d[j] = r0;
            if (j1 < n_new) nb_d[j1] = r1;
            if (j2 < n_new) nb_d[j2] = r2;
        }
    }
}

// The end of traverse_cpu_kernel (traverse_cpu.cpp:139-162) without heap operations.
// Upstream pushes every seed into the result heap (heap_pushpop keeps the H
// smallest distances; one equal to the current worst stays out), pops the H - k_out
// worst entries and stores the others worst first, i.e. ascending.  When the
// distances that matter are pairwise different, that is the n_real smallest of
// (results + seeds) in ascending order, whatever the heaps looked like on the
// way.  So: (1) a radix select over the float bit patterns (non-negative floats
// order like their bits; eight 4-bit passes with 16 shared counters) finds the H-th
// smallest distance T, (2) the entries below T and as many of those equal to T as
// still fit are gathered into the open heap's memory (dead by now), (3) a bitonic
// network sorts them, (4) the first n_real are stored.
// Which equal distances matter: those among the first n_check entries and the one
// behind them (pads, (-1, +inf), excepted: they are interchangeable).  The sub-graph
// stage of a search that goes on hands n_check = max(k, kSeedHead): entries further
// back are too far for the seeding of the full-graph stage, and the final k are no
// larger than the k smallest here -- exchanging two ids of equal distance behind
// them exchanges these ids in every later heap and nothing else.  Equal distances
// that matter, or a distance that is negative or NaN, make the outcome depend on
// upstream's exact sequence: nothing is written then and the caller runs that
// sequence.  Returns true (CTA-uniform) if the output is written.
template <bool kList>
__device__ __forceinline__ bool select_sort_output(const RefShared &S, int H, int seed_lo,
                                                   int n_seed, int n_real, int k_out, int n_check,
                                                   RefCtl *ctl) {
    const int tid = threadIdx.x, n_thr = blockDim.x;
    const int32_t *c_id = S.c_id + seed_lo;
    const float *c_d = S.c_d + seed_lo;
    // the array heap holds negated distances, the dumped list distances
    auto result_at = [&](int x) {
        HeapEntry e = S.buf[1 + x];
        if (!kList) e.k = -e.k;
        return e;
    };
    const int N = H + n_seed - seed_lo;
    int *bins = reinterpret_cast<int *>(S.open);  // 16 counters, then the gathered entries
    HeapEntry *a = S.open;
    if (tid == 0) {
        ctl->tie = 0;
        ctl->n_taken = 0;
        ctl->n_equal = 0;
    }
    // (1) the H-th smallest key
    unsigned prefix = 0, mask = 0;
    int want = H, at_T = 0;
    bool bad = false;
    for (int shift = 28; shift >= 0; shift -= 4) {
        __syncthreads();
        if (tid < 16) bins[tid] = 0;
        __syncthreads();
        for (int x = tid; x < N; x += n_thr) {
            float dx;
            if (x < H) {
                dx = result_at(x).k;
            } else {
                if (c_id[x - H] < 0) continue;
                dx = c_d[x - H];
            }
            if (!(dx >= 0.0f)) bad = true;
            const unsigned key = __float_as_uint(dx);
            if ((key & mask) == prefix) atomicAdd(&bins[(key >> shift) & 15u], 1);
        }
        __syncthreads();
        int before = 0, digit = 15;
        bool found = false;
#pragma unroll
        for (int b = 0; b < 16; ++b) {  // every thread, same result
            const int c = bins[b];
            if (!found) {
                if (before + c < want) {
                    before += c;
                } else {
                    digit = b;
                    found = true;
                }
            }
        }
        want -= before;
        at_T = bins[digit];
        prefix |= static_cast<unsigned>(digit) << shift;
        mask |= 15u << shift;
    }
    const unsigned T = prefix;  // `want` of the at_T entries equal to T are needed
    if (n_check >= H && at_T > want && T != __float_as_uint(CUDART_INF_F)) bad = true;
    if (bad) ctl->tie = 1;
    __syncthreads();
    if (ctl->tie != 0) return false;
    // (2) gather
    int P = 1;
    while (P < H) P <<= 1;  // P <= 2H - 1 entries fit
    for (int i = H + tid; i < P; i += n_thr) a[i] = HeapEntry{CUDART_INF_F, -1};
    for (int x = tid; x < N; x += n_thr) {
        HeapEntry e;
        if (x < H) {
            e = result_at(x);
        } else {
            e.v = c_id[x - H];
            if (e.v < 0) continue;
            e.k = c_d[x - H];
        }
        const unsigned key = __float_as_uint(e.k);
        bool take = key < T;
        if (key == T) take = atomicAdd(&ctl->n_equal, 1) < want;
        if (take) a[atomicAdd(&ctl->n_taken, 1)] = e;
    }
    __syncthreads();
    // (3) sort ascending
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = tid; t < (P >> 1); t += n_thr) {
                const int lo = 2 * t - (t & (stride - 1));  // index with bit `stride` clear
                const int hi = lo + stride;
                const bool up = (lo & size) == 0;
                const HeapEntry x = a[lo], y = a[hi];
                if ((x.k > y.k) == up) {
                    a[lo] = y;
                    a[hi] = x;
                }
            }
            __syncthreads();
        }
    }
    bool tie = kList && ctl->amb < CUDART_INF_F && ctl->amb <= a[n_check - 1].k;
    for (int i = tid; i < n_check && i + 1 < H; i += n_thr)
        if (a[i].k == a[i + 1].k && (a[i].v >= 0 || a[i + 1].v >= 0)) tie = true;
    if (tie) ctl->tie = 1;
    __syncthreads();
    if (ctl->tie != 0) return false;
    // (4)
    for (int r = tid; r < n_real; r += n_thr) {
        const HeapEntry e = a[r];
        S.c_id[k_out - n_real + r] = e.v;
        S.c_d[k_out - n_real + r] = e.k;
    }
    return true;
}

// The same end when the seeds ascend (full-graph stage): results and seeds are two
// sorted lists, an entry's place in the union is its own index plus the entries of
// the other list before it (a binary search).  Writes the first n_real.
__device__ __forceinline__ bool merge_sorted_output(const RefShared &S, const HeapEntry *list,
                                                    int H, int seed_lo, int n_seed, int n_real,
                                                    int k_out, RefCtl *ctl) {
    const int tid = threadIdx.x, n_thr = blockDim.x;
    const int ny = n_seed - seed_lo;
    HeapEntry *a = S.open;  // [n_real + 1], in front of `list`: the last one only to compare with
    if (tid == 0) {
        ctl->tie = 0;
        a[n_real] = HeapEntry{CUDART_INF_F, -1};  // should the union end before it
    }
    __syncthreads();
    for (int x = tid; x < H + ny; x += n_thr) {
        const bool res = x < H;
        const int own = res ? x : x - H;
        const HeapEntry e = res ? list[own] : HeapEntry{S.c_d[seed_lo + own], S.c_id[seed_lo + own]};
        if (own > n_real) continue;
        int lo = 0, hi = res ? ny : H;  // entries of the other list in front of e
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const float o = res ? S.c_d[seed_lo + mid] : list[mid].k;
            if (res ? o < e.k : o <= e.k) lo = mid + 1; else hi = mid;
        }
        if (own + lo <= n_real) a[own + lo] = e;
    }
    __syncthreads();
    bool tie = ctl->amb < CUDART_INF_F && ctl->amb <= a[n_real - 1].k;
    for (int i = tid; i < n_real; i += n_thr)
        if (a[i].k == a[i + 1].k && (a[i].v >= 0 || a[i + 1].v >= 0)) tie = true;
    if (tie) ctl->tie = 1;
    __syncthreads();
    if (ctl->tie != 0) return false;
    for (int r = tid; r < n_real; r += n_thr) {
        S.c_id[k_out - n_real + r] = a[r].v;
        S.c_d[k_out - n_real + r] = a[r].k;
    }
    return true;
}

__device__ __forceinline__ RefShared ref_shared(const RefineArgs &A, unsigned char *smem) {
    RefShared S;
    S.q = reinterpret_cast<float *>(smem);
    S.open = reinterpret_cast<HeapEntry *>(S.q + A.d);
    S.buf = S.open + 2 * A.H + 2;
    S.c_id = reinterpret_cast<int32_t *>(S.buf + A.H + 2);
    S.c_d = reinterpret_cast<float *>(S.c_id + A.n_cand);
    S.nb_id = reinterpret_cast<int32_t *>(S.c_d + A.n_cand);
    S.nb_d = reinterpret_cast<float *>(S.nb_id + 2 * kMaxDegree);
    S.stage = S.nb_d + 2 * kMaxDegree;
    return S;
}

extern __shared__ __align__(16) unsigned char ref_smem[];

// The heap warp's side of a stage: the result list (or the array heap, R = 0), the
// log, the counters.
template <int R, bool kList> struct HeapSide {
    TopList<R> top;
    float worst;
    int n_log;
    PathBits<R> larger;  // of the open heap

    __device__ __forceinline__ void clear(int H, int lane) {
        top.clear(H, lane);
        worst = CUDART_INF_F;
        n_log = 0;
    }
    // the open heap, once it holds its seeds
    __device__ __forceinline__ void open_filled(const RefShared &S, int n, int lane) {
        larger.build_larger(S.open, n, lane);
    }
    __device__ __forceinline__ void open_push(const RefShared &S, int n, float k, int32_t v,
                                              int lane, const WalkLane &) {
        bit_replace(S.open, n, k, v, larger, lane);
    }
    __device__ __forceinline__ HeapEntry open_pop(const RefShared &S, int n, int lane,
                                                  const WalkLane &WL) {
        return bit_pop(S.open, n, larger, lane, WL);
    }
    __device__ __forceinline__ float worst_of(const RefShared &) const { return worst; }
    // heap_update (:23-39) over the n_new neighbours in buffer nb: every distance below
    // the worst result is admitted, in row order; f(distance, id, index) follows.
    template <class F>
    __device__ __forceinline__ void admit(const RefShared &S, const int32_t *nb_id,
                                          const float *nb_d, int n_new, int log_room, int H,
                                          int lane, const WalkLane &, RefCtl *ctl, F f) {
        for (int c = 0; c < n_new; c += 32) {
            const bool in = c + lane < n_new;
            const float dist = in ? nb_d[c + lane] : CUDART_INF_F;
            const int32_t id = in ? nb_id[c + lane] : -1;
            if (!(dist >= 0.0f)) ctl->rerun = 1;  // NaN: see search_stage
            unsigned ahead = kAll;
            for (;;) {
                const unsigned m = __ballot_sync(kAll, dist < worst) & ahead;
                if (m == 0) break;
                const int j = __ffs(m) - 1;
                ahead = 0xfffffffeu << j;
                const float nk = __shfl_sync(kAll, dist, j);
                const int32_t nv = __shfl_sync(kAll, id, j);
                if (top.worst_twice(worst)) ctl->amb = fminf(ctl->amb, worst);  // all lanes alike
                top.insert(nk, nv, lane);
                worst = top.worst();
                if (lane == 0) {
                    if (n_log < min(H, log_room)) {
                        S.buf[1 + n_log] = HeapEntry{nk, nv};
                    } else if (n_log < log_room) {
                        S.c_id[n_log - H] = nv;
                        S.c_d[n_log - H] = nk;
                    }
                }
                ++n_log;
                f(nk, nv, c + j);
            }
        }
    }
    // after the last expansion: the list to shared memory, ascending
    __device__ __forceinline__ void finish(HeapEntry *list, int H, int lane, RefCtl *ctl) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = 32 * r + lane - (32 * R - H);
            if (i >= 0) list[i] = HeapEntry{top.k[r], top.v[r]};
        }
        ctl->n_log = n_log;
    }
};

// Array heaps with the comparison bits of both: a stage that will meet equal distances
// (finish_query).  (The bits follow the array as long as no key is NaN.)
template <int R> struct HeapSide<R, false> {
    float worst;
    PathBits<R> larger;                 // of the open heap
    PathBits<result_words(R)> smaller;  // of the result heap

    __device__ __forceinline__ void clear(int, int) {
        worst = CUDART_INF_F;
        smaller.clear();
    }
    __device__ __forceinline__ void open_filled(const RefShared &S, int n, int lane) {
        larger.build_larger(S.open, n, lane);
    }
    __device__ __forceinline__ void open_push(const RefShared &S, int n, float k, int32_t v,
                                              int lane, const WalkLane &) {
        bit_replace(S.open, n, k, v, larger, lane);
    }
    __device__ __forceinline__ HeapEntry open_pop(const RefShared &S, int n, int lane,
                                                  const WalkLane &WL) {
        return bit_pop(S.open, n, larger, lane, WL);
    }
    __device__ __forceinline__ float worst_of(const RefShared &) const { return worst; }
    template <class F>
    __device__ __forceinline__ void admit(const RefShared &S, const int32_t *nb_id,
                                          const float *nb_d, int n_new, int, int H, int lane,
                                          const WalkLane &, RefCtl *ctl, F f) {
        for (int c = 0; c < n_new; c += 32) {
            const bool in = c + lane < n_new;
            const float dist = in ? nb_d[c + lane] : CUDART_INF_F;
            const int32_t id = in ? nb_id[c + lane] : -1;
            if (!(dist >= 0.0f)) ctl->rerun = 1;  // NaN: see search_stage
            unsigned ahead = kAll;
            for (;;) {
                const unsigned m = __ballot_sync(kAll, dist < worst) & ahead;
                if (m == 0) break;
                const int j = __ffs(m) - 1;
                ahead = 0xfffffffeu << j;
                const float nk = __shfl_sync(kAll, dist, j);
                const int32_t nv = __shfl_sync(kAll, id, j);
                bit_sink(S.buf, H, HeapEntry{-nk, nv}, smaller, lane);
                worst = -S.buf[1].k;
                f(nk, nv, c + j);
            }
        }
    }
    __device__ __forceinline__ void finish(HeapEntry *, int, int, RefCtl *) {}
};

template <> struct HeapSide<0, false> {
    __device__ __forceinline__ void clear(int, int) {}
    __device__ __forceinline__ void open_filled(const RefShared &, int, int) {}
    __device__ __forceinline__ void open_push(const RefShared &S, int n, float k, int32_t v,
                                              int lane, const WalkLane &WL) {
        warp_replace(S.open, n, k, v, lane, WL);
    }
    __device__ __forceinline__ HeapEntry open_pop(const RefShared &S, int n, int lane,
                                                  const WalkLane &WL) {
        return warp_pop(S.open, n, lane, WL);
    }
    __device__ __forceinline__ float worst_of(const RefShared &S) const { return -S.buf[1].k; }
    template <class F>
    __device__ __forceinline__ void admit(const RefShared &S, const int32_t *nb_id,
                                          const float *nb_d, int n_new, int, int H, int lane,
                                          const WalkLane &WL, RefCtl *, F f) {
        for (int j = 0; j < n_new; ++j) {
            const float dist = nb_d[j];
            if (dist >= -S.buf[1].k) continue;
            warp_pushpop(S.buf, H, -dist, nb_id[j], lane, WL);
            f(dist, nb_id[j], j);
        }
    }
    __device__ __forceinline__ void finish(HeapEntry *, int, int, RefCtl *) {}
};

__device__ __forceinline__ void count_expansion(int *st, int n_new, int lane) {
    if (lane == 0) {
        ++st[0];
        st[1] += n_new;
    }
}

// A search of exactly two expansions (the sub-graph stage: REFINE_STEP = 2,
// traverse_cpu.cpp:317-326) without the open heap.  heap_replace only ever drops or
// evicts an entry that is no smaller than the leaf at the end of a larger-child
// walk, and at least four entries of a heap of 32 or more are no larger than that
// leaf (the root, its larger child and that child's sibling, the next node of the
// walk) -- so the two smallest keys ever offered are in the heap when they are
// popped, and with pairwise different keys the two pops are simply: the smallest
// seed, then the smaller of the second-smallest seed and the best neighbour
// admitted during the first expansion.  The results are kept exactly as
// upstream keeps them (the worst decides admissions and the stop test).
// Whenever the keys that matter are not pairwise different the layout of the open
// heap decides: with equal smallest seeds nothing is done and false is returned (the
// caller runs upstream's sequence); a tie met at the second pop is settled by
// building the open heap after all, in upstream's order, and popping it.
// Called by all threads after the seeds are marked; returns CTA-uniformly whether
// ctl->m1 .. c2 hold what brief_search needs.
__device__ __forceinline__ bool brief_prepare(const RefShared &S, int n_seed, RefCtl *ctl) {
    const int tid = threadIdx.x, n_thr = blockDim.x;
    constexpr unsigned long long kNone = ~0ull;
    if (tid == 0) {
        ctl->m1 = ctl->m2 = kNone;
        ctl->c1 = ctl->c2 = 0;
        ctl->tie = 0;
    }
    __syncthreads();
    bool bad = false;
    for (int i = tid; i < n_seed; i += n_thr) {
        if (S.c_id[i] < 0) continue;
        const float dist = S.c_d[i];
        if (!(dist >= 0.0f && dist < CUDART_INF_F)) bad = true;
        if (dist != dist) ctl->rerun = 1;  // NaN in the open heap: see search_stage
        atomicMin(&ctl->m1, (static_cast<unsigned long long>(__float_as_uint(dist)) << 32) | i);
    }
    if (bad) ctl->tie = 1;
    __syncthreads();
    const unsigned long long m1 = ctl->m1;
    const int i1 = static_cast<int>(m1 & 0xffffffffu);
    for (int i = tid; i < n_seed; i += n_thr) {
        if (S.c_id[i] < 0 || i == i1) continue;
        const unsigned key = __float_as_uint(S.c_d[i]);
        if (key == static_cast<unsigned>(m1 >> 32)) atomicAdd(&ctl->c1, 1);
        atomicMin(&ctl->m2, (static_cast<unsigned long long>(key) << 32) | i);
    }
    __syncthreads();
    if (ctl->tie != 0 || ctl->c1 != 0) return false;  // nothing has been changed
    const unsigned long long m2 = ctl->m2;
    const int i2 = static_cast<int>(m2 & 0xffffffffu);
    for (int i = tid; i < n_seed; i += n_thr) {
        if (S.c_id[i] < 0 || i == i1 || i == i2) continue;
        if (__float_as_uint(S.c_d[i]) == static_cast<unsigned>(m2 >> 32)) atomicAdd(&ctl->c2, 1);
    }
    __syncthreads();
    return true;
}

// The heap warp's half; the gather warps run the two expansions (search_stage).
template <int R, bool kList>
__device__ __forceinline__ void brief_search(const RefineArgs &A, const RefShared &S, int n_seed,
                                             RefCtl *ctl, HeapSide<R, kList> &side, const WalkLane &WL,
                                             int lane, int *st) {
    constexpr unsigned long long kNone = ~0ull;
    const int H = A.H;
    const unsigned long long m1 = ctl->m1, m2 = ctl->m2;
    if (m1 == kNone) return;  // no seed at all: the first pop ends the search
    const int i2 = static_cast<int>(m2 & 0xffffffffu);
    // first pop: the smallest seed; there is no result yet, the stop test passes
    cta_sync();  // its neighbours are in buffer 0
    const int n_new = ctl->n_new[0];
    count_expansion(st, n_new, lane);
    unsigned long long admitted = 0;
    float best = CUDART_INF_F;
    int best_j = -1;
    bool best_twice = false;
    side.admit(S, S.nb_id, S.nb_d, n_new, 0, H, lane, WL, ctl,
               [&](float dist, int32_t, int j) {  // heap_update without the open heap
                   admitted |= 1ull << j;
                   if (dist < best) {
                       best = dist;
                       best_j = j;
                       best_twice = false;
                   } else if (dist == best) {
                       best_twice = true;
                   }
               });
    // second pop
    const bool seed_left = m2 != kNone;
    const float seed_k = seed_left ? S.c_d[i2] : CUDART_INF_F;
    int u2 = -1;
    float k2 = CUDART_INF_F;
    bool unsure = false;
    if (best_j >= 0 && (!seed_left || best < seed_k)) {
        u2 = S.nb_id[best_j];
        k2 = best;
        unsure = best_twice;
    } else if (seed_left && (best_j < 0 || seed_k < best)) {
        u2 = S.c_id[i2];
        k2 = seed_k;
        unsure = ctl->c2 != 0;
    } else if (seed_left) {  // equal
        unsure = true;
    }
    if (unsure) {  // upstream's sequence on the open heap
        for (int i = 0; i < n_seed; ++i) {
            const int id = S.c_id[i];
            if (id >= 0) warp_replace(S.open, 2 * H, S.c_d[i], id, lane, WL);
        }
        warp_pop(S.open, 2 * H, lane, WL);
        for (int j = 0; j < n_new; ++j)
            if ((admitted >> j) & 1ull) warp_replace(S.open, 2 * H, S.nb_d[j], S.nb_id[j], lane, WL);
        const HeapEntry nx = warp_pop(S.open, 2 * H, lane, WL);
        u2 = nx.v;
        k2 = nx.k;
    }
    if (u2 >= 0 && k2 >= side.worst_of(S)) u2 = -1;  // :86-90
    if (lane == 0) ctl->pop_u[1] = u2;
    cta_sync();
    if (u2 < 0) return;
    cta_sync();  // the second expansion is in buffer 1
    count_expansion(st, ctl->n_new[1], lane);
    side.admit(S, S.nb_id + kMaxDegree, S.nb_d + kMaxDegree, ctl->n_new[1], 0, H, lane, WL, ctl,
               [](float, int32_t, int) {});
}

// The heap warp's half of the general search (:64-136).
template <int R, bool kList>
__device__ __forceinline__ void heap_loop(const RefineArgs &A, const RefShared &S, int n_seed,
                                          int seed_lo, int max_iter, bool closed_form, int log_room,
                                          RefCtl *ctl, HeapSide<R, kList> &side, const WalkLane &WL,
                                          int lane, int *st, int *prof, long long &prof_t) {
    (void)prof; (void)prof_t;
    const int H = A.H;
    if (closed_form) {
        // The real seeds are c[seed_lo ..] in ascending order, the first kSeedHead of them
        // strictly.  Every key offered to heap_replace is then no smaller than all keys in
        // the heap: it replaces a +inf leaf and climbs to just below a real entry, or meets
        // a real leaf and is dropped -- which of the two depends on the count of
        // seeds before it only.  Seed 0 ends at heap index 0, seeds 2t - 1 and 2t
        // at the two rightmost nodes of level t (2^(t+1) - 3 and 2^(t+1) - 2,
        // 0-based) while those exist; all later seeds are dropped.  Checked
        // against heap_replace for every heap size and seed count on the host.
        const int t = (lane + 1) >> 1;
        const int pos = lane == 0 ? 0 : (1 << (t + 1)) - 3 + ((lane & 1) ? 0 : 1);
        const int at = seed_lo + lane;
        // (heap_replace drops an infinite key)
        if (lane < 25 && pos < 2 * H && at < n_seed && S.c_id[at] >= 0 && S.c_d[at] < CUDART_INF_F)
            S.open[1 + pos] = HeapEntry{S.c_d[at], S.c_id[at]};
        __syncwarp();
    } else {
        for (int i = 0; i < n_seed; ++i) {
            const int id = S.c_id[i];
            if (id >= 0) warp_replace(S.open, 2 * H, S.c_d[i], id, lane, WL);
        }
    }
    side.open_filled(S, 2 * H, lane);
    PA_TICK(1);
    // :82-136.  Expansion i uses slot i & 1 of the control block and of the
    // neighbour buffers.  Per expansion one CTA-wide barrier: behind it the heap
    // warp has popped node i (or ended the search) and -- when speculating --
    // the gather warps have prepared the node they expected.
    {
        const HeapEntry u = side.open_pop(S, 2 * H, lane, WL);
        const bool stop = max_iter <= 0 || u.v < 0 || u.k >= side.worst_of(S);
        if (lane == 0) {
            ctl->pop_u[0] = stop ? -1 : u.v;
            ctl->root_k[0] = S.open[1].k;
            ctl->root_v[0] = S.open[1].v;
            ctl->guess[0] = ctl->guess[1] = -2;
        }
    }
    PA_TICK(2);
    for (int step = 0; step < max_iter; ++step) {
        const int p = step & 1;
        cta_sync();
        PA_TICK(4);
        const int u = ctl->pop_u[p];
        if (u < 0) break;
        if (u != ctl->guess[p]) cta_sync();  // the gather warps fetch node u now
        PA_TICK(3);
        // heap_update (:23-39) in row order, then the next pop (:84-90)
        const int n_new = ctl->n_new[p];
        count_expansion(st, n_new, lane);
        side.admit(S, S.nb_id + p * kMaxDegree, S.nb_d + p * kMaxDegree, n_new, log_room, H, lane,
                   WL, ctl, [&](float dist, int32_t id, int) {
                       side.open_push(S, 2 * H, dist, id, lane, WL);
#if PA_REFINE_PROFILE
                       if (PA_REFINE_PROFILE == 1 && threadIdx.x == 0) prof[7] += 1;
#endif
                   });
        PA_TICK(5);
        if (step + 1 < max_iter) {
            const HeapEntry nx = side.open_pop(S, 2 * H, lane, WL);
            const bool stop = nx.v < 0 || nx.k >= side.worst_of(S);
            if (lane == 0) {
                ctl->pop_u[p ^ 1] = stop ? -1 : nx.v;
                ctl->root_k[p ^ 1] = S.open[1].k;
                ctl->root_v[p ^ 1] = S.open[1].v;
            }
        }
        PA_TICK(2);
    }
}

// The heap warp's half of a stage.  Out of line: the registers of its heaps and those
// of the gather's row loads are never live together, and inlined they were allocated as
// if they were (rows spilled, 768 dimensions 17.8 instead of 16.1 ms per 8192 queries).
template <int R, bool kList>
__device__ __noinline__ void heap_side(const RefineArgs &A, RefCtl *ctl, int n_seed, int max_iter,
                                       bool second, bool brief, bool closed_form, int *st) {
    const RefShared S = ref_shared(A, ref_smem);
    const int lane = threadIdx.x & 31, H = A.H;
    const int seed_lo = second ? max(n_seed - H, 0) : 0;
    const WalkLane WL = walk_lane(lane);
    HeapSide<R, kList> side;
    side.clear(H, lane);
    ctl->amb = CUDART_INF_F;  // all lanes alike
    st[0] = st[1] = 0;
    __syncwarp();
    int prof[12] = {};
    long long prof_t = 0;
#if PA_REFINE_PROFILE
    prof_t = ctl->heap_clock;
#endif
    if (brief) {
        brief_search<R, kList>(A, S, n_seed, ctl, side, WL, lane, st);
        PA_TICK(1);
    } else {
        heap_loop<R, kList>(A, S, n_seed, seed_lo, max_iter, closed_form, second ? H + seed_lo : 0, ctl,
                     side, WL, lane, st, prof, prof_t);
    }
    side.finish(second ? S.open + H + 1 : S.buf + 1, H, lane, ctl);
#if PA_REFINE_PROFILE
    if (lane == 0) {
        for (int i = 0; i < 12; ++i) ctl->heap_prof[i] = prof[i];
        ctl->heap_clock = prof_t;
    }
#endif
}

// The gather warps' half of the general search.
__device__ __forceinline__ void gather_loop(const RefineArgs &A, const RefShared &S,
                                            const RefGraph &G, uint8_t *vis, uint8_t marker,
                                            int max_iter, bool speculate, RefCtl *ctl, int gw,
                                            int lane, int *prof, long long &prof_t) {
    for (int step = 0; step < max_iter; ++step) {
        const int p = step & 1;
        cta_sync();
        if (step == 0) { PA_GTICK(7); } else { PA_GTICK(6); }  // waiting for the heap warp: seed inserts / a pop
        const int u = ctl->pop_u[p];
        if (u < 0) break;
        if (u != ctl->guess[p]) {  // CTA-uniform: nothing, or something else, was prepared
            gather_node(A, S, G, vis, marker, ctl, u, p, gw, lane, prof, prof_t);
            cta_sync();
        }
        if (speculate && step + 1 < max_iter) {
            // the node the next pop returns unless it ends the search: the first
            // new neighbour with the smallest distance if that is below the root
            // the open heap had after this expansion's pop, else that root.
            // Distances are sums of squares: their bits order like their values.
            const int n_new = ctl->n_new[p];
            const float *nb_d = S.nb_d + p * kMaxDegree;
            unsigned best = __float_as_uint(CUDART_INF_F);
            int at = 0;
            for (int c = 0; c < n_new; c += 32) {
                const unsigned key = c + lane < n_new ? __float_as_uint(nb_d[c + lane]) : ~0u;
                const unsigned least = __reduce_min_sync(kAll, key);
                if (least < best) {
                    best = least;
                    at = c + __ffs(__ballot_sync(kAll, key == least)) - 1;
                }
            }
            const int guess = __uint_as_float(best) < ctl->root_k[p] ? S.nb_id[p * kMaxDegree + at]
                                                                     : ctl->root_v[p];
            if (gw == 0 && lane == 0) ctl->guess[p ^ 1] = guess;
            if (guess >= 0) gather_node(A, S, G, vis, marker, ctl, guess, p ^ 1, gw, lane, prof, prof_t);
        }
    }
}

// Upstream's sequence at the end of a stage (:139-162), by the heap warp.
template <int R, bool kList>
__device__ __noinline__ void upstream_output(const RefineArgs &A, const RefCtl *ctl, int n_seed,
                                             int n_real, int k_out, bool second) {
    const RefShared S = ref_shared(A, ref_smem);
    const int lane = threadIdx.x & 31, H = A.H;
    const int seed_lo = second ? max(n_seed - H, 0) : 0;
    PathBits<result_words(R)> smaller;
    const WalkLane WL = walk_lane(lane);
    auto push = [&](float dist, int32_t id) {
        if (R == 0) warp_pushpop(S.buf, H, -dist, id, lane, WL);
        else if (!(-dist <= S.buf[1].k))
            bit_sink(S.buf, H, HeapEntry{-dist, id}, smaller, lane);
    };
    auto pop = [&]() {
        if (R == 0) return warp_pop(S.buf, H, lane, WL);
        const HeapEntry out = S.buf[1];
        __syncwarp();
        bit_sink(S.buf, H, HeapEntry{CUDART_INF_F, -1}, smaller, lane);
        return out;
    };
    if (R > 0 && !kList) smaller.build_smaller(S.buf, H, lane);
    if (kList) {
        // the result heap as upstream's pushes leave it; the log's part in buf makes
        // room for it by going where the list was
        HeapEntry *moved = S.open;
        const int n_log = second ? ctl->n_log : 0, in_buf = min(n_log, H);
        for (int i = lane; i < in_buf; i += 32) moved[i] = S.buf[1 + i];
        __syncwarp();
        for (int i = lane; i < H + 2; i += 32) S.buf[i] = HeapEntry{-CUDART_INF_F, -1};
        smaller.clear();
        __syncwarp();
        for (int i = 0; i < n_log; ++i) {
            const HeapEntry e = i < H ? moved[i] : HeapEntry{S.c_d[i - H], S.c_id[i - H]};
            push(e.k, e.v);
        }
        for (int x = 0; !second && x < ctl->st[0]; ++x)  // the expansions of the first stage
            for (int j = 0; j < ctl->n_new[x]; ++j) {
                const float dist = S.nb_d[x * kMaxDegree + j];
                if (!(dist >= -S.buf[1].k)) push(dist, S.nb_id[x * kMaxDegree + j]);
            }
    }
    for (int i = seed_lo; i < n_seed; ++i) {
        const int id = S.c_id[i];
        if (id >= 0) push(S.c_d[i], id);
    }
    for (int i = k_out; i < H; ++i) pop();
    // what is left, worst first, into the open heap's memory: the seeds are in use
    for (int i = 0; i < n_real; ++i) {
        const HeapEntry e = pop();
        if (lane == 0) S.open[H + 1 - i] = HeapEntry{-e.k, e.v};
    }
    __syncwarp();
    for (int i = lane; i < n_real; i += 32) {
        const HeapEntry e = S.open[H + 2 - n_real + i];
        S.c_id[k_out - n_real + i] = e.v;
        S.c_d[k_out - n_real + i] = e.k;
    }
}

// One call of upstream's traverse_cpu_kernel: seeds in c_id / c_d (n_seed of
// them), the result (k_out entries, ascending behind (-1, -inf) pads) back into
// c_id / c_d.  `from` < d: the seeds' distances are first completed over dims
// [from, d).  `second`: the full-graph stage behind the sub-graph stage, whose seeds
// are that stage's output.  n_check: how many leading entries of the output have to be
// upstream's in the order of equal distances, too.  Returns expansions and
// evaluations through ctl->st, and false (CTA-uniform) if the query
// has to be run on the array heaps (R > 0 only: a NaN distance, of a neighbour or of a
// seed, which upstream's tests let into the heaps, or equal distances after more admissions than the log holds).
template <int R, bool kList>
__device__ __forceinline__ bool search_stage(const RefineArgs &A, const RefShared &S,
                                             const RefGraph &G, uint8_t *vis, uint8_t marker,
                                             int n_seed, int from, int max_iter, int k_out,
                                             bool second, int n_check, RefCtl *ctl, int *prof,
                                             long long &prof_t) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int d = A.d, H = A.H;
    const bool speculate = second;
    (void)prof; (void)prof_t;
    // distances completed over the trailing dims (:41-62), in place
    if (from < d) {
        float *stage = S.stage + w * d;
        const int n_w = static_cast<int>(blockDim.x >> 5);
        if (d - from <= 32) {
            short_residuals<8>(A.storage, S.q, S.c_id, S.c_d, n_seed, d, from, w, n_w, lane);
        } else if (d - from <= 64) {
            short_residuals<16>(A.storage, S.q, S.c_id, S.c_d, n_seed, d, from, w, n_w, lane);
        } else if (d - from > 384) {  // long rows: one round trip each, two rows per warp and trip
            for (int i = w; i < n_seed; i += 2 * n_w) {
                const int i1 = i + n_w;
                const int id0 = S.c_id[i], id1 = i1 < n_seed ? S.c_id[i1] : -1;
                if (id0 < 0 && id1 < 0) continue;  // warp-uniform
                if (id1 >= 0) row_to_stage(stage, A.storage + static_cast<int64_t>(id1) * d, d, from, lane);
                float r0 = 0.0f, r1 = 0.0f;
                if (id0 >= 0) r0 = one_row(A.storage + static_cast<int64_t>(id0) * d, S.q, d, from, lane);
                if (id1 >= 0) r1 = staged_row(stage, S.q, d, from, lane);
                if (lane == 0) {
                    if (id0 >= 0) S.c_d[i] = __fadd_rn(S.c_d[i], r0);
                    if (id1 >= 0) S.c_d[i1] = __fadd_rn(S.c_d[i1], r1);
                }
            }
        } else {
            for (int i = w; i < n_seed; i += 3 * n_w) {
                const int i1 = i + n_w, i2 = i + 2 * n_w;
                const int id0 = S.c_id[i], id1 = i1 < n_seed ? S.c_id[i1] : -1;
                const int id2 = i2 < n_seed ? S.c_id[i2] : -1;
                if (id0 < 0 && id1 < 0 && id2 < 0) continue;  // warp-uniform
                if (id2 >= 0) row_to_stage(stage, A.storage + static_cast<int64_t>(id2) * d, d, from, lane);
                float r0, r1;
                two_rows(A.storage + static_cast<int64_t>(max(id0, 0)) * d,
                         A.storage + static_cast<int64_t>(max(id1, 0)) * d, S.q, d, from, lane, r0, r1);
                float r2 = 0.0f;
                if (id2 >= 0) r2 = staged_row(stage, S.q, d, from, lane);
                if (lane == 0) {
                    if (id0 >= 0) S.c_d[i] = __fadd_rn(S.c_d[i], r0);
                    if (id1 >= 0) S.c_d[i1] = __fadd_rn(S.c_d[i1], r1);
                    if (id2 >= 0) S.c_d[i2] = __fadd_rn(S.c_d[i2], r2);
                }
            }
        }
    }
    PA_GTICK(4);  // residual distances of the seeds
    // :65-68
    if (!kList)
        for (int i = tid; i < H + 2; i += blockDim.x) S.buf[i] = HeapEntry{-CUDART_INF_F, -1};
    for (int i = tid; i < 2 * H + 2; i += blockDim.x) S.open[i] = HeapEntry{CUDART_INF_F, -1};
    // :69-79, the marks (their order does not matter; the heap inserts below keep it)
    for (int i = tid; i < n_seed; i += blockDim.x) {
        const int id = S.c_id[i];
        if (id >= 0) vis[id] = marker;
    }
    __syncthreads();
    PA_TICK(0);
    // seeds of the second stage: behind the pads the first stage left
    const int seed_lo = second ? max(n_seed - H, 0) : 0;
    // Log of the second stage: H entries in buf, the others where its pads were; the list
    // then goes behind the part of the open heap that the merge writes.  The first stage
    // has no log: its neighbours are still in their buffers.
    const int log_room = second ? H + seed_lo : 0;
    HeapEntry *list = second ? S.open + H + 1 : S.buf + 1;
    const int sorted = second ? ctl->sorted : 0;
    const bool brief = max_iter == 2 && !speculate && 2 * H >= 32 && G.degree <= 64 &&
                       brief_prepare(S, n_seed, ctl);
    if (w == 0) {
#if PA_REFINE_PROFILE
        if (lane == 0) ctl->heap_clock = prof_t;
        __syncwarp();
#endif
        heap_side<R, kList>(A, ctl, n_seed, max_iter, second, brief,
                     sorted == (kAscending | kHeadStrict) && n_seed >= H, ctl->st + (second ? 2 : 0));
#if PA_REFINE_PROFILE
        if (lane == 0) {
            for (int i = 0; i < 12; ++i) prof[i] += ctl->heap_prof[i];
            prof_t = ctl->heap_clock;
        }
#endif
    } else if (brief) {
        if (ctl->m1 != ~0ull) {
            gather_node(A, S, G, vis, marker, ctl, S.c_id[ctl->m1 & 0xffffffffu], 0, w - 1, lane, prof, prof_t);
            cta_sync();
            cta_sync();  // the heap warp has the second node
            const int u2 = ctl->pop_u[1];
            if (u2 >= 0) {
                gather_node(A, S, G, vis, marker, ctl, u2, 1, w - 1, lane, prof, prof_t);
                cta_sync();
            }
        }
    } else {
        gather_loop(A, S, G, vis, marker, max_iter, speculate, ctl, w - 1, lane, prof, prof_t);
    }
    __syncthreads();
    if (R > 0 && (ctl->rerun != 0 || (second && (sorted & kAscending) == 0))) return false;
    PA_TICK(5);
    // :139-162: the seeds join the results; all but k_out are dropped; what is
    // left comes out worst first and is stored ascending
    const int n_real = min(k_out, H);
    const bool done =  // CTA-uniform
        kList && second
            ? merge_sorted_output(S, list, H, seed_lo, n_seed, n_real, k_out, ctl)
            : select_sort_output<kList>(S, H, seed_lo, n_seed, n_real, k_out, min(n_check, n_real), ctl);
    if (tid == 0) {
        ctl->sorted = kAscending | kHeadStrict;  // select_sort_output has seen to it
        if (!second) ctl->tied = 0;
    }
    if (!done) {
        if (kList && second && ctl->n_log > log_room) return false;
        if (w == 0) upstream_output<R, kList>(A, ctl, n_seed, n_real, k_out, second);
        __syncthreads();
        // NaN distances may come out in any order; equal ones near the front forbid the
        // closed form of the next stage's seeding (pads are not seeded)
        for (int i = tid; i + 1 < n_real; i += blockDim.x) {
            const int at = k_out - n_real + i;
            if (!(S.c_d[at] <= S.c_d[at + 1])) ctl->sorted = 0;
            else if (S.c_d[at] == S.c_d[at + 1] && (S.c_id[at] >= 0 || S.c_id[at + 1] >= 0)) {
                if (i < kSeedHead) atomicAnd(&ctl->sorted, kAscending);
                if (!second) atomicAdd(&ctl->tied, 1);
            }
        }
    }
    // pops of an exhausted heap give (-1, key +inf): the leading pads
    for (int i = tid; i < k_out - n_real; i += blockDim.x) {
        S.c_id[i] = -1;
        S.c_d[i] = -CUDART_INF_F;
    }
    __syncthreads();
    PA_TICK(6);
    PA_GTICK(8);  // merge and output
    return true;
}

// A stage of the running query, with the arguments that go with it.
template <int R, bool kList>
__device__ __forceinline__ bool query_stage(const RefineArgs &A, const RefShared &S, uint8_t *vis,
                                            int marker, bool second, RefCtl *ctl, int *prof,
                                            long long &prof_t) {
    // sub-graph, REFINE_STEP expansions (traverse_cpu.cpp:317-326); full graph, same marker
    // (:327-336)
    return search_stage<R, kList>(
        A, S, second ? A.full : A.sub, vis, static_cast<uint8_t>(marker), A.n_cand, second ? A.d : A.d_p,
        min(second ? 1024 : 2, 2 * A.ef), second ? A.k : A.n_cand, second,
        second ? A.k : A.stages >= 3 ? max(A.k, kSeedHead) : A.H, ctl, prof, prof_t);
}

// Query b is loaded and gets a marker of its own.
__device__ __forceinline__ int begin_query(const RefineArgs &A, const RefShared &S, int64_t b,
                                           int slot, uint8_t *vis, RefCtl *ctl) {
    const int tid = threadIdx.x;
    // next marker of this slot; the array is wiped when the markers run out
    // (bitmask.hpp:17-36 does the same on wrap-around)
    if (tid == 0) {
        ctl->marker = A.epoch[slot] + 1;
        ctl->rerun = ctl->half = 0;
        ctl->st[2] = ctl->st[3] = 0;
    }
    __syncthreads();
    int marker = ctl->marker;
    if (marker > 254) {
        uint4 *p = reinterpret_cast<uint4 *>(vis);
        for (int64_t i = tid; i < A.slot_stride / 16; i += blockDim.x)
            p[i] = make_uint4(0, 0, 0, 0);
        marker = 1;
    }
    __syncthreads();
    if (tid == 0) A.epoch[slot] = ctl->marker = marker;

    for (int i = tid; i < A.d; i += blockDim.x) S.q[i] = A.query[b * A.ldq + i];
    for (int i = tid; i < A.n_cand; i += blockDim.x) {
        const int64_t id = A.cand_I[b * A.n_cand + i];
        S.c_id[i] = (id < 0 || id >= A.n_nodes) ? -1 : static_cast<int32_t>(id);
        S.c_d[i] = A.cand_D[b * A.n_cand + i];
    }
    __syncthreads();
    return marker;
}

__device__ __forceinline__ void end_query(const RefineArgs &A, const RefShared &S, int64_t b,
                                          const RefCtl *ctl, const int *prof) {
    (void)prof;
    const int tid = threadIdx.x;
    const int k_last = A.stages >= 3 ? A.k : A.n_cand;
    for (int i = tid; i < k_last; i += blockDim.x) {
        A.out_I[b * k_last + i] = S.c_id[i];
        A.out_D[b * k_last + i] = S.c_d[i];
    }
#if PA_REFINE_PROFILE
    if (A.stats != nullptr && tid == 32)
        for (int i = 0; i < 12; ++i) A.stats[b * 24 + 12 + i] = prof[i];
#endif
    if (A.stats != nullptr && tid == 0) {
#if PA_REFINE_PROFILE
        for (int i = 0; i < 4; ++i) A.stats[b * 24 + i] = ctl->st[i];
        for (int i = 0; i < 8; ++i) A.stats[b * 24 + 4 + i] = prof[i];
#else
#pragma unroll
        for (int i = 0; i < 4; ++i) A.stats[b * 4 + i] = ctl->st[i];
#endif
    }
}

// Query b from its candidates to its output.  False: finish_query has to.
template <int R>
__device__ __forceinline__ bool run_query(const RefineArgs &A, const RefShared &S, int64_t b,
                                          int slot, uint8_t *vis, RefCtl *ctl) {
    const int marker = begin_query(A, S, b, slot, vis, ctl);
    int prof[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    long long prof_t = 0;
#if PA_REFINE_PROFILE
    prof_t = pinned_clock();
#endif
    if (!query_stage<R, (R > 0)>(A, S, vis, marker, false, ctl, prof, prof_t)) return false;
    if (A.stages >= 3) {
        if (R > 0 && ctl->tied >= kManyTied) {
#if PA_REFINE_PROFILE
            if (threadIdx.x == 0 || threadIdx.x == 32) {
                ctl->clock[threadIdx.x / 32] = prof_t;
                for (int i = 0; i < 12; ++i) ctl->phases[threadIdx.x / 32][i] = prof[i];
            }
#endif
            if (threadIdx.x == 0) ctl->half = 1;
            return false;
        }
        if (!query_stage<R, (R > 0)>(A, S, vis, marker, true, ctl, prof, prof_t)) return false;
    }
    end_query(A, S, b, ctl, prof);
    return true;
}

// What is left of a query for the array heaps in a kernel that has the list, out of line: few
// queries need it.  With comparison bits the second stage of a query whose first stage met
// several equal distances, since the second will meet more of them, and with the list each tie
// ends in a replay of the log by one warp or, when the log is full, in a second run of the
// query.  (One equal pair is chance as a rule and stays with the list: 1024 queries at ef 128 and
// k 100 in 300 k different vectors of 200 dimensions 2180 us, with every tied one here 2330.)
// Without: both stages of a query that met a NaN or overflowed the log.  The whole search where
// every vector is there twice (300 k), us, heaps only / list only / now: 1024 queries of 96
// dimensions at ef 256 3379 / 5418 / 2820, 8192 at ef 128 8934 / 11392 / 8325; of 200 dimensions
// 1024 at ef 128 2665 / 3736 / 2521, 8192 at ef 32 5768 / 9144 / 6164.  (Called from one place, at
// the end of the query: a call between the stages cost a lone query 2 % in spills around it.)
template <int R>
__device__ __noinline__ void finish_query(const RefineArgs &A, int64_t b, RefCtl *ctl) {
    __syncthreads();
    const RefShared S = ref_shared(A, ref_smem);
    const int slot = A.slot_begin + blockIdx.x;
    uint8_t *vis = A.marks + static_cast<int64_t>(slot) * A.slot_stride;
    if (ctl->half != 0) {
        int prof[12] = {};
        long long prof_t = 0;
#if PA_REFINE_PROFILE
        if (threadIdx.x == 0 || threadIdx.x == 32) {
            prof_t = ctl->clock[threadIdx.x / 32];
            for (int i = 0; i < 12; ++i) prof[i] = ctl->phases[threadIdx.x / 32][i];
        }
#endif
        if (query_stage<R, false>(A, S, vis, ctl->marker, true, ctl, prof, prof_t)) {
            end_query(A, S, b, ctl, prof);
            return;
        }
        __syncthreads();
    }
    run_query<0>(A, S, b, slot, vis, ctl);
}

template <int R, int kMaxThreads, int kMinCtas>
__global__ void __launch_bounds__(kMaxThreads, kMinCtas) refine_kernel(const __grid_constant__ RefineArgs A) {
    __shared__ RefCtl ctl_s;
    RefCtl *ctl = &ctl_s;
    const RefShared S = ref_shared(A, ref_smem);
    const int tid = threadIdx.x;
    const int slot = A.slot_begin + blockIdx.x;
    uint8_t *vis = A.marks + static_cast<int64_t>(slot) * A.slot_stride;

    // CTA i starts on query i; whoever finishes claims the next unclaimed query (queries
    // differ several-fold in length, and a launch is over when its last CTA is)
    for (int64_t b = blockIdx.x; b < A.batch;) {
        if (!run_query<R>(A, S, b, slot, vis, ctl)) finish_query<R>(A, b, ctl);
        if (tid == 0) ctl->next = atomicAdd(A.claim, 1u);
        __syncthreads();
        b = static_cast<int64_t>(gridDim.x) + ctl->next;
    }
}

// traverse_cpu.cpp:228-254
static int cpu_heap_size_for(int ef) {
    static const int sizes[] = {16, 32, 48, 64, 96, 128, 192, 256, 384, 512, 1024, 2048};
    for (int s : sizes)
        if (ef <= s) return s;
    return -1;
}

// Refinement CTAs one SM holds at ef_search 128 (registers and shared memory): the
// number of visited slots worth having per SM.
int refine_ctas_per_sm(int d_model) {
    const int by_registers = (64 * 1024) / (56 * ref_threads_for(d_model));
    return by_registers < 12 ? by_registers : 12;  // shared memory: about 17 KB per CTA
}

// one staged row per warp
static size_t refine_smem_bytes(int d, int H, int n_cand, int warps) {
    return sizeof(float) * d * (1 + warps) + sizeof(HeapEntry) * (3 * H + 4) +
           8 * static_cast<size_t>(n_cand) + 16 * kMaxDegree;
}
// what a call is accepted by: a narrow CTA may be launched with up to four warps
static size_t refine_smem_bytes(int d, int H, int n_cand) {
    return refine_smem_bytes(d, H, n_cand, max(ref_threads_for(d), 128) / 32);
}
constexpr size_t kRefMaxSmem = 200 * 1024;

template <int R, int kMaxThreads, int kMinCtas>
static int refine_launch_with(const RefineArgs &A, unsigned grid, int threads, int dev,
                              cudaStream_t stream) {
    const size_t smem = refine_smem_bytes(A.d, A.H, A.n_cand, max(threads, 128) / 32);
    static size_t configured[64] = {};
    if (smem > 48 * 1024 && dev >= 0 && dev < 64 && configured[dev] < smem) {
        PA_CUDA_TRY(cudaFuncSetAttribute(refine_kernel<R, kMaxThreads, kMinCtas>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem)));
        configured[dev] = smem;
    }
    refine_kernel<R, kMaxThreads, kMinCtas><<<grid, threads, smem, stream>>>(A);
    count_launch();
    PA_CUDA_TRY(cudaGetLastError());
    return PA_OK;
}

// The CTA for a launch of `grid` queries at a time on a device of `sms` SMs.  A query
// alone waits for its rows' round trips and for nothing else, so as long as the SMs
// have room a query gets the warps to fetch an expansion in one trip: 16 warps up to two
// queries per SM, 8 up to four.  One query of 768 dimensions at ef 128: 0.86 -> 0.54 ms;
// seven of 96 dimensions at ef 96: 0.32 -> 0.28; 333 of 384 dimensions at ef 48 (8 warps):
// 0.47 -> 0.385.  At the limits, ef 32 to 256, time over that of three or five warps: 16 warps
// at two queries per SM 0.65 to 0.84 (96 dimensions up to 0.97, where 8 are as fast), 8 warps at four
// 0.83 to 0.96, sub-graph stage alone included.
template <int R>
static int refine_launch_for(const RefineArgs &A, unsigned grid, unsigned sms, int dev,
                             cudaStream_t stream) {
    auto fits = [&](int threads, unsigned per_sm) {
        return grid <= per_sm * sms &&
               refine_smem_bytes(A.d, A.H, A.n_cand, threads / 32) <= kRefMaxSmem / per_sm;
    };
    if (fits(512, 2)) return refine_launch_with<R, 512, 2>(A, grid, 512, dev, stream);
    if (fits(256, 4)) return refine_launch_with<R, 256, 4>(A, grid, 256, dev, stream);
    int threads = ref_threads_for(A.d);
    if (threads == kRefThreadsNarrow && kRefThreadsNarrow == 96 && grid <= 9 * sms) threads = 128;
    return refine_launch_with<R, kRefThreads, PA_REFINE_MIN_CTAS>(A, grid, threads, dev, stream);
}

static int refine_launch(const RefineArgs &A, int n_slots, cudaStream_t stream) {
    if (A.batch == 0) return PA_OK;
    int dev = 0;
    PA_CUDA_TRY(cudaGetDevice(&dev));
    const unsigned grid = static_cast<unsigned>(min(static_cast<int64_t>(A.batch),
                                                    static_cast<int64_t>(n_slots)));
    static int sm_count[64] = {};
    int sms = 0;
    if (dev >= 0 && dev < 64) {
        if (sm_count[dev] == 0)
            PA_CUDA_TRY(cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev));
        sms = sm_count[dev];
    }
    switch (list_regs_for(A.H)) {
        case 2: return refine_launch_for<2>(A, grid, sms, dev, stream);
        case 4: return refine_launch_for<4>(A, grid, sms, dev, stream);
        case 8: return refine_launch_for<8>(A, grid, sms, dev, stream);
        default: {
            int threads = ref_threads_for(A.d);
            if (threads == kRefThreadsNarrow && kRefThreadsNarrow == 96 && grid <= 9u * sms)
                threads = 128;
            return refine_launch_with<0, kRefThreads, PA_REFINE_MIN_CTAS>(A, grid, threads, dev, stream);
        }
    }
}

static int refine_check(const void *out_I, const void *out_D, const void *cand_I, const void *cand_D,
                 const float *query, int64_t ldq, const float *storage, const int32_t *packed_nbr,
                 const int32_t *row_of, int n_neighbors, const int32_t *full_nbr, int full_degree,
                 int64_t batch, int64_t n_nodes, int d, int d_p, int n_cand, int ef, int k,
                 int stages) {
    PA_REQUIRE(batch >= 0 && batch <= 0x7fffffff, "batch out of range");
    PA_REQUIRE(stages == 2 || stages == 3, "stages must be 2 (sub-graph stage) or 3 (both)");
    PA_REQUIRE(ef > 0 && cpu_heap_size_for(ef) > 0, "ef_search must be in (0, 2048]");
    PA_REQUIRE(d > 0 && d % 4 == 0 && d_p > 0 && d_p % 4 == 0 && d_p <= d,
               "d_model / d_principle must be multiples of 4 with d_principle <= d_model");
    PA_REQUIRE(ldq >= d && ldq % 4 == 0, "query row stride must be a multiple of 4");
    PA_REQUIRE(n_cand > 0 && n_cand % 4 == 0, "the candidate row must be a positive multiple of 4");
    PA_REQUIRE(n_nodes > 0 && n_nodes < 0x7fffffff, "node ids must fit int32");
    PA_REQUIRE(n_neighbors > 0 && n_neighbors <= kMaxDegree, "n_neighbors must be in (0, 64]");
    if (stages >= 3) {
        PA_REQUIRE(k > 0 && k <= n_cand, "k must be in (0, candidates per query]");
        PA_REQUIRE(full_degree > 0 && full_degree <= kMaxDegree, "full-graph degree must be in (0, 64]");
    }
    PA_REQUIRE(refine_smem_bytes(d, cpu_heap_size_for(ef), n_cand) <= kRefMaxSmem,
               "d_model, ef_search and the candidate row together exceed the shared memory of a CTA");
    if (batch == 0) return PA_OK;
    PA_REQUIRE(out_I && out_D && cand_I && cand_D && query && storage && packed_nbr && row_of,
               "null pointer");
    PA_REQUIRE(stages < 3 || full_nbr != nullptr, "stage 3 needs the packed full graph");
    PA_REQUIRE(aligned16(query) && aligned16(storage), "query / storage must be 16-byte aligned");
    return PA_OK;
}

static RefineArgs refine_args(int64_t *out_I, float *out_D, const int64_t *cand_I, const float *cand_D,
                       const float *query, int64_t ldq, const float *storage,
                       const int32_t *packed_nbr, const int32_t *row_of, int n_neighbors,
                       const int32_t *full_nbr, int full_degree, int64_t batch, int64_t n_nodes,
                       int d, int d_p, int n_cand, int ef, int k, int stages, uint8_t *marks,
                       int32_t *epoch, int64_t slot_stride, int slot_begin, int32_t *stats) {
    RefineArgs A;
    A.cand_I = cand_I; A.cand_D = cand_D; A.query = query; A.ldq = ldq; A.storage = storage;
    A.n_nodes = n_nodes; A.d = d; A.d_p = d_p;
    A.sub = RefGraph{packed_nbr, row_of, 4 * static_cast<int64_t>(n_neighbors), 4, n_neighbors};
    A.full = RefGraph{full_nbr, nullptr, full_degree, 1, full_degree};
    A.n_cand = n_cand; A.ef = ef; A.H = cpu_heap_size_for(ef); A.k = k; A.stages = stages;
    A.batch = static_cast<int>(batch);
    A.out_I = out_I; A.out_D = out_D; A.marks = marks; A.epoch = epoch;
    A.slot_stride = slot_stride; A.slot_begin = slot_begin; A.stats = stats;
    return A;
}

// ---- full graph, packed: int32 [n_nodes, degree], -1 padded ----------------------
// One thread per node.  A row stops at its first negative id (as the search
// does); an id that repeats an earlier id of the row is dropped (the search would
// find it visited), so rows hold distinct ids.
__global__ void pack_full_kernel(int32_t *__restrict__ out, const int64_t *__restrict__ indptr,
                                 const int64_t *__restrict__ indices, int64_t n_nodes, int degree,
                                 int *__restrict__ error) {
    const int64_t u = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (u >= n_nodes) return;
    const int64_t lo = indptr[u], hi = indptr[u + 1];
    int32_t *row = out + u * degree;
    int n = 0;
    for (int64_t i = lo; i < hi; ++i) {
        const int64_t v = indices[i];
        if (v < 0) break;
        if (v >= n_nodes) { atomicMax(error, 2); break; }
        bool dup = false;
        for (int j = 0; j < n; ++j) dup = dup || row[j] == static_cast<int32_t>(v);
        if (dup) continue;
        if (n == degree) { atomicMax(error, 1); break; }
        row[n++] = static_cast<int32_t>(v);
    }
    for (; n < degree; ++n) row[n] = -1;
}

}  // namespace pa

extern "C" int pa_cpu_heap_size_for(int ef_search) { return pa::cpu_heap_size_for(ef_search); }

extern "C" int pa_refine_ctas_per_sm(int d_model) { return pa::refine_ctas_per_sm(d_model); }

namespace pa {

// Checks, then one launch on `stream` whose CTAs own pool slots
// [slot_begin, slot_begin + slot_count).
int refine_enqueue(int64_t *out_I, float *out_D, const int64_t *cand_I, const float *cand_D,
                   const float *query, int64_t ldq, const float *storage_full,
                   const int32_t *packed_nbr, const int32_t *row_of, int n_neighbors,
                   const int32_t *full_nbr, int full_degree, int64_t batch, int64_t n_nodes,
                   int d_model, int d_principle, int n_cand, int ef_search, int k, int stages,
                   const pa_visited_pool *pool, int slot_begin, int slot_count, int32_t *stats,
                   cudaStream_t stream) {
    int rc = refine_check(out_I, out_D, cand_I, cand_D, query, ldq, storage_full, packed_nbr,
                          row_of, n_neighbors, full_nbr, full_degree, batch, n_nodes, d_model,
                          d_principle, n_cand, ef_search, k, stages);
    if (rc != PA_OK || batch == 0) return rc;
    if (pool == nullptr) return fail(PA_ERR_STATE, "visited pool is null");
    uint8_t *marks; int32_t *epoch; int64_t slot_stride, pool_nodes; int n_slots;
    pool_view(pool, &marks, &epoch, &slot_stride, &n_slots, &pool_nodes);
    PA_REQUIRE(pool_nodes >= n_nodes, "the visited pool was created for fewer nodes");
    PA_REQUIRE(slot_begin >= 0 && slot_count > 0 && slot_begin + slot_count <= n_slots,
               "slot range outside the visited pool");
    RefineArgs A = refine_args(out_I, out_D, cand_I, cand_D, query, ldq, storage_full, packed_nbr,
                               row_of, n_neighbors, full_nbr, full_degree, batch, n_nodes, d_model,
                               d_principle, n_cand, ef_search, k, stages, marks, epoch, slot_stride,
                               slot_begin, stats);
    A.claim = reinterpret_cast<unsigned *>(epoch + n_slots + slot_begin);
    PA_CUDA_TRY(cudaMemsetAsync(A.claim, 0, sizeof(unsigned), stream));
    return refine_launch(A, slot_count, stream);
}

}  // namespace pa

extern "C" int pa_refine(int64_t *out_I, float *out_D, const int64_t *cand_I, const float *cand_D,
                         const float *query, const float *storage_full, const int32_t *packed_nbr,
                         const int32_t *row_of, int n_neighbors, const int32_t *full_nbr,
                         int full_degree, int64_t batch, int64_t n_nodes, int d_model,
                         int d_principle, int n_cand, int ef_search, int k, int stages,
                         pa_visited_pool *pool, int32_t *stats, void *stream) {
    return pa::refine_enqueue(out_I, out_D, cand_I, cand_D, query, d_model, storage_full,
                              packed_nbr, row_of, n_neighbors, full_nbr, full_degree, batch,
                              n_nodes, d_model, d_principle, n_cand, ef_search, k, stages, pool, 0,
                              pa_visited_pool_slots(pool), stats, static_cast<cudaStream_t>(stream));
}

extern "C" int pa_pack_fullgraph(int32_t *full_nbr, const int64_t *indptr, const int64_t *indices,
                                 int64_t n_nodes, int degree, void *stream_) {
    using namespace pa;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    PA_REQUIRE(n_nodes >= 0 && n_nodes < 0x7fffffff, "node ids must fit int32");
    PA_REQUIRE(degree > 0 && degree <= kMaxDegree, "degree must be in (0, 64]");
    if (n_nodes == 0) return PA_OK;
    PA_REQUIRE(full_nbr && indptr && indices, "null pointer");
    struct ErrorWord {
        int *p = nullptr;
        cudaStream_t s;
        ~ErrorWord() { if (p != nullptr) cudaFreeAsync(p, s); }
    } word;
    word.s = stream;
    PA_CUDA_TRY(cudaMallocAsync(&word.p, sizeof(int), stream));
    PA_CUDA_TRY(cudaMemsetAsync(word.p, 0, sizeof(int), stream));
    pack_full_kernel<<<static_cast<unsigned>((n_nodes + 127) / 128), 128, 0, stream>>>(
        full_nbr, indptr, indices, n_nodes, degree, word.p);
    count_launch();
    PA_CUDA_TRY(cudaGetLastError());
    int host_error = 0;
    PA_CUDA_TRY(cudaMemcpyAsync(&host_error, word.p, sizeof(int), cudaMemcpyDeviceToHost, stream));
    PA_CUDA_TRY(cudaStreamSynchronize(stream));
    if (host_error == 1)
        return fail(PA_ERR_UNPACKABLE, "a row holds more than `degree` distinct neighbours");
    if (host_error == 2) return fail(PA_ERR_UNPACKABLE, "a neighbour id is out of range");
    return PA_OK;
}
