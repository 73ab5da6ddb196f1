// PageRank over an EBV-partitioned graph: the propagation step is the same sparse
// aggregation as GraphSum at feature width 1.
//
// Two schedules share the kernels below:
//  * DRONE's delta PageRank (PR_PEVal / PR_IncEVal, DRONE/src/cuda/algorithm/pr.cu:375-488):
//    pr starts at 1, a vertex whose value moved by at least eps pushes (new-old)/outDegree
//    to its out-neighbours, boundary vertices are reconciled mirror -> master (add) and
//    master -> mirror (assign), dangling mass goes through a one-element all-reduce.
//  * synchronous power iteration (damping d, fixed iteration count, start 1/|V|).
//
// Where the reference pushes along out-edges with atomicAdd (pr.cu:14-87), this
// implementation pulls along in-edges of the transposed local graph: every vertex
// publishes its delta once (-0.0 for "did not push") and every vertex sums what its
// in-neighbours published.  Same arithmetic, no atomics on values, fixed summation order.
// Parts held by one process run all their supersteps in one launch (pr_run_kernel); between
// processes the boundary exchange is static and dense (all mirrors of a peer in one
// message, ordered by global id), each entry carrying the flag that the
// reference expresses by sending or not sending the vertex.  Either way the counts the
// caller uses to detect termination (Response, common.h:23-27) are reproduced.
#include "exchange.cuh"
#include "grid_sync.cuh"
#include "plan.cuh"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdlib>
#include <new>
#include <vector>

namespace drone {
int xplan_ensure_device(drone_xplan *x);
}

struct drone_pr {
    unsigned long long uid = 0;       // number of this handle in the process (addresses are reused, this is not)
    int device = 0, n_local = 0, global_v = 0, nnz = 0;
    bool dbl = false;
    double eps = 1e-6;
    drone_plan *plan = nullptr;       // owned: transposed local graph + chunk lists (values unused)
    drone_xplan *xplan = nullptr;     // borrowed
    drone_comm *comm = nullptr;       // borrowed (may be NULL for a single part)
    int *out_degree = nullptr, *mirror2worker = nullptr;
    void *pr = nullptr, *acc = nullptr, *diff = nullptr, *push = nullptr;   // real[n] each
    void *push2 = nullptr;            // real[n] second buffer of the published values (pr_resident_kernel)
    // Where vertex i publishes its delta.  The deltas lie in the order of how often they are gathered (most gathered
    // first) and the pull lists' columns are renumbered to match, so that a prefix of the array, small enough for
    // shared memory, serves most gathers.  NULL (few vertices): delta i lies at i.
    int *place = nullptr;
    int *active = nullptr, *ubm = nullptr;
    void *scalars = nullptr;          // real[4]: globalDiff, globalAcc, dangling (power mode), isolated value
    void *block_sums = nullptr;       // real[kReduceBlocks]
    void *partials = nullptr;         // Partial[n_partials]
    int *slot_split = nullptr;        // [n_partials] split row a partial slot belongs to
    int *arrived = nullptr;           // [n_split_rows] slots written so far in this pull (0 between pulls)
    void *send = nullptr, *recv = nullptr;   // real2[max(up, down)]
    int *counters = nullptr;          // [0..3] exchange counts, [4] active count
    // parts held by one process: {part, row} of every contribution a master row takes, in m_pos order, {place, out
    // degree} of that row in its part, and the plans these were filled in for
    int2 *pairs = nullptr, *targets = nullptr;
    std::vector<unsigned long long> pairs_for;
    int *role = nullptr;              // [n_local] kOwnRow, kMirrorRow, or the number of the master row
    // [b - 1]: {rows, edges} of the largest slice when this part's rows are dealt to b blocks; empty: too large for that
    std::vector<int2> slices;
    char *control = nullptr;          // RunControl + superstep counts of the persistent kernel (part 0 of a run)
    drone::RowStream stream;                 // one part too large for slices: its rows in the order of place
    int *stream_od = nullptr;
    void *stream_tails = nullptr;
    drone::DeviceBlock stream_block;         // what the stream's arrays are pieces of
    drone::DeviceBlock block;                // what the other arrays made at creation are pieces of
    int sms = 0;
    bool separate_steps = false;      // parts in one process take the kernels of one process per GPU (local_parts_run_separately)
    unsigned barrier_start = 0, barrier_polls = 0;   // what the grid barrier's count starts at, and when its waits run out
    unsigned run = 0;                 // number (in the process) of the launch that made the values; 0: the separate kernels did
    unsigned *unfinished = nullptr;   // device: number of the last launch that gave up
    bool started = false;
    long long n_isolated = 0;         // vertex ids that occur in no part (power iteration treats them as dangling)
};

namespace drone {

static const int kReduceBlocks = 1024;

template <typename R> struct alignas(2 * sizeof(R)) Pair { R val, flag; };          // one boundary entry of a message
template <typename R> struct alignas(2 * sizeof(R)) Partial { R sum; int pushed; };   // one chunk of a split row
template <typename R> struct NcclType;
template <> struct NcclType<float> { static constexpr ncclDataType_t value = ncclFloat; };
template <> struct NcclType<double> { static constexpr ncclDataType_t value = ncclDouble; };

template <typename R> __device__ __forceinline__ R fma_r(R a, R b, R c);
template <> __device__ __forceinline__ float fma_r<float>(float a, float b, float c) { return fmaf(a, b, c); }
template <> __device__ __forceinline__ double fma_r<double>(double a, double b, double c) { return fma(a, b, c); }

// What a vertex that does not push publishes: -0.0.  A pushed delta is never -0.0 ((new - old) / outDegree gives +0.0
// when nothing moved), and adding -0.0 changes no sum, so one word per vertex carries both the delta and the flag.
__device__ __forceinline__ bool is_pushed(float v) { return __float_as_uint(v) != 0x80000000u; }
__device__ __forceinline__ bool is_pushed(double v) { return __double_as_longlong(v) != (long long)0x8000000000000000ULL; }
template <typename R> __device__ __forceinline__ R not_pushed() { return (R)-0.0; }

constexpr int kOwnRow = -1, kMirrorRow = -2;      // roles of a row that no other part holds, and of one whose master is elsewhere

// Device view of one part.
template <typename R>
struct PartView {
    int n, global_v, n_chunks, n_ranges, n_masters, table_n;
    const Chunk *chunks;
    const int *col, *s_range_row, *s_rowptr, *s_rows, *s_col;
    const SplitRow *split;
    const int *slot_split;
    int *arrived;
    Partial<R> *partials;
    R *pr, *acc, *diff, *push, *scalars;
    int *active, *ubm;
    const int *out_degree, *mirror2worker, *place;
    const int *m_rows, *m_off;
    const int2 *pairs, *targets;
    unsigned *unfinished;
    const int *rowptr;
    R *push2;
    const int *role;                       // runs over several parts: kOwnRow, kMirrorRow, or the number of the master row
};

// Sum of v over the block in a fixed order (tree over warps), result in thread 0.
template <typename R>
__device__ R block_sum(R v) {
    __shared__ double sm[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sm[w] = (double)v;
    __syncthreads();
    R tot = 0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += (R)sm[i];
    return tot;
}

// ---- per-vertex steps, shared by the kernels of one superstep and the persistent kernel.  `first` / `stride`: the
// thread's share of the vertices, four of them at a time so that their loads are in flight together (a store between
// two vertices' loads would keep the compiler from doing that itself).  Each returns the dangling mass it met. ----
constexpr int kVertexBatch = 4;

// pr = start, acc = diff = 0, flags cleared; publish start/outDegree.
// (pr_init, DRONE/src/cuda/algorithm/pr.cu:14-37, plus the fills of PR_PEVal :391-394.)
template <typename R>
__device__ __forceinline__ R init_vertices(const PartView<R> &p, R start, bool power, int first, int stride) {
    R dangling = 0;
#pragma unroll 1
    for (int i0 = first; i0 < p.n; i0 += kVertexBatch * stride) {
        int od[kVertexBatch], at[kVertexBatch];
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) {
            const int i = i0 + b * stride;
            od[b] = i < p.n ? __ldg(p.out_degree + i) : 1;
            at[b] = i < p.n && p.place ? __ldg(p.place + i) : i;
        }
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) {
            const int i = i0 + b * stride;
            if (i >= p.n) break;
            p.pr[i] = start;
            p.acc[i] = 0;
            p.diff[i] = 0;
            p.active[i] = 0;
            p.ubm[i] = 0;
            if (od[b] == 0 && __ldg(p.mirror2worker + i) == -1) dangling += power ? start : start / p.global_v;
            p.push[at[b]] = od[b] == 0 ? not_pushed<R>() : start / od[b];
        }
    }
    return dangling;
}

// pr_process_messages (pr.cu:430-448) fused with pr_increment (pr.cu:51-87).
template <typename R>
__device__ __forceinline__ R increment_vertices(const PartView<R> &p, R eps, R gacc, int first, int stride) {
    const R alpha = (R)0.85f;                // pr.cu:12 declares a float constant
    const R one_minus_alpha = (R)1 - alpha;
    R dangling = 0;
#pragma unroll 1
    for (int i0 = first; i0 < p.n; i0 += kVertexBatch * stride) {
        R a[kVertexBatch], old[kVertexBatch];
        int od[kVertexBatch], at[kVertexBatch];
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) {
            const int i = i0 + b * stride;
            a[b] = i < p.n ? p.acc[i] + p.diff[i] : (R)0;
            old[b] = i < p.n ? p.pr[i] : (R)0;
            od[b] = i < p.n ? __ldg(p.out_degree + i) : 1;
            at[b] = i < p.n && p.place ? __ldg(p.place + i) : i;
        }
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) {
            const int i = i0 + b * stride;
            if (i >= p.n) break;
            p.ubm[i] = 0;
            p.acc[i] = a[b];                 // the pull that follows writes diff and active of every vertex
            const R now = fma_r<R>(alpha, a[b] + gacc, one_minus_alpha);
            R d = now - old[b];
            if (d < 0) d = -d;
            R out = not_pushed<R>();
            if (!(d < eps)) {
                if (od[b] == 0) {
                    if (__ldg(p.mirror2worker + i) == -1) dangling += (now - old[b]) / p.global_v;
                } else {
                    out = (now - old[b]) / od[b];
                }
                p.pr[i] = now;
            }
            p.push[at[b]] = out;
        }
    }
    return dangling;
}

// pr' = (1-d)/V + d * (sum over in-edges + dangling/V), published as pr'/outDegree for the next iteration; after the
// last one (`last`) the value itself is stored instead: before that nobody can see it.  Leaves out the vertices that
// other parts hold too (SHARED).
template <typename R, bool SHARED>
__device__ __forceinline__ R power_vertices(const PartView<R> &p, R damping, R dang, bool last, int first, int stride) {
    const R base = ((R)1 - damping) / p.global_v;
    const R share = dang / p.global_v;
    R dangling = 0;
#pragma unroll 1
    for (int i0 = first; i0 < p.n; i0 += kVertexBatch * stride) {
        R d[kVertexBatch];
        int od[kVertexBatch], at[kVertexBatch], skip[kVertexBatch];
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) {
            const int i = i0 + b * stride;
            skip[b] = i >= p.n ? 1 : SHARED && p.role ? __ldg(p.role + i) != kOwnRow : 0;
            d[b] = i < p.n ? p.diff[i] : (R)0;
            od[b] = i < p.n && !last ? __ldg(p.out_degree + i) : 1;
            at[b] = i < p.n && !last && p.place ? __ldg(p.place + i) : i;
        }
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) {
            const int i = i0 + b * stride;
            if (skip[b]) continue;
            const R now = base + damping * (d[b] + share);
            if (last) {
                p.pr[i] = now;
                continue;
            }
            if (od[b] == 0 && __ldg(p.mirror2worker + i) == -1) dangling += now;
            p.push[at[b]] = od[b] == 0 ? not_pushed<R>() : now / od[b];
        }
    }
    return dangling;
}

// ---- pull along in-edges: diff[v] = sum of published deltas, active[v] = any in-neighbour pushed ----
//
// Bound: one scattered gather per edge.  A load of 32 scattered words from L2 costs the LSU 32 wavefronts whatever
// its hit rate, which caps the whole part at about 2.9e11 gathers per second; a shared-memory load of 32 scattered
// words costs 3 to 4.  So every block first copies the most gathered part of the array (a prefix, see `place`) into
// shared memory and gathers from global memory only what lies behind it (R-MAT-22: 56 % of the gathers hit 40,960
// floats).  Measured, R-MAT-22 float: 0.323 -> 0.256 ms per power iteration.
//
// `table`: the first p.table_n published values, in shared memory.  `warp` of `n_warps`: this warp's share of the work.

// The value published at place c.  Both loads are predicated instead of branched around, so that the gathers of a batch
// stay in flight together.  `table` is a shared-memory address.
__device__ __forceinline__ float published(unsigned table, int table_n, const float *push, int c) {
    float v;
    asm volatile("{\n\t.reg .pred n;\n\t.reg .u32 s;\n\t.reg .u64 g;\n\t.reg .f32 a, b;\n\t"
                 "setp.lt.s32 n, %1, %2;\n\t"
                 "mad.lo.u32 s, %1, 4, %3;\n\t"
                 "mad.wide.s32 g, %1, 4, %4;\n\t"
                 "@n ld.shared.f32 a, [s];\n\t"
                 "@!n ld.global.f32 b, [g];\n\t"
                 "selp.f32 %0, a, b, n;\n\t}"
                 : "=f"(v) : "r"(c), "r"(table_n), "r"(table), "l"(push) : "memory");
    return v;
}
__device__ __forceinline__ double published(unsigned table, int table_n, const double *push, int c) {
    double v;
    asm volatile("{\n\t.reg .pred n;\n\t.reg .u32 s;\n\t.reg .u64 g;\n\t.reg .f64 a, b;\n\t"
                 "setp.lt.s32 n, %1, %2;\n\t"
                 "mad.lo.u32 s, %1, 8, %3;\n\t"
                 "mad.wide.s32 g, %1, 8, %4;\n\t"
                 "@n ld.shared.f64 a, [s];\n\t"
                 "@!n ld.global.f64 b, [g];\n\t"
                 "selp.f64 %0, a, b, n;\n\t}"
                 : "=d"(v) : "r"(c), "r"(table_n), "r"(table), "l"(push) : "memory");
    return v;
}

// 16 bytes a load and four loads in flight: the table is filled once per pull by every block.
template <typename R>
__device__ __forceinline__ void load_table(const PartView<R> &p, R *table) {
    constexpr int W = 16 / sizeof(R);
    const int n4 = p.table_n / W;
    const float4 *src = reinterpret_cast<const float4 *>(p.push);
    float4 *dst = reinterpret_cast<float4 *>(table);
    int i = threadIdx.x;
#pragma unroll 1
    for (; i + 3 * (int)blockDim.x < n4; i += 4 * blockDim.x) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = src[i + u * blockDim.x];
#pragma unroll
        for (int u = 0; u < 4; ++u) dst[i + u * blockDim.x] = v[u];
    }
    for (; i < n4; i += blockDim.x) dst[i] = src[i];
    for (i = n4 * W + threadIdx.x; i < p.table_n; i += blockDim.x) table[i] = p.push[i];
}

// Split rows: the warps note the slots they filled and, 32 chunks at a time, make them visible with one fence and count
// them in; the warp that counts in a row's last slot adds the row's slots, in slot order.  (Waiting at fences is 1.4 %
// of the stall cycles this way; with a fence per chunk it was 11 %.)  `slot`: lane l's l-th noted slot, -1 for none.
template <typename R, bool FLAGS>
__device__ __forceinline__ void close_slots(const PartView<R> &p, int slot) {
    const int lane = threadIdx.x & 31;
    if (!__any_sync(0xffffffffu, slot >= 0)) return;
    int at = 0, first = 0, n_slots = 0;
    bool last = false;
    __threadfence();
    __syncwarp();
    if (slot >= 0) {
        at = __ldg(p.slot_split + slot);
        const int4 sr = __ldg(reinterpret_cast<const int4 *>(p.split) + at);      // row, first slot, slots
        first = sr.y;
        n_slots = sr.z;
        last = atomicAdd(p.arrived + at, 1) == n_slots - 1;
    }
    unsigned todo = __ballot_sync(0xffffffffu, last);
    if (todo) __threadfence();
#pragma unroll 1
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const int f = __shfl_sync(0xffffffffu, first, src), n = __shfl_sync(0xffffffffu, n_slots, src);
        R sum = 0;
        bool pushed = false;
#pragma unroll 1
        for (int k = lane; k < n; k += 32) {
            const Partial<R> *q = p.partials + f + k;
            sum += __ldcg(&q->sum);
            if (FLAGS) pushed = pushed || __ldcg(&q->pushed) != 0;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (FLAGS) pushed = __any_sync(0xffffffffu, pushed);
        if (lane == src) {
            const int row = __ldg(&p.split[at].row);
            p.arrived[at] = 0;
            p.diff[row] = sum;
            if (FLAGS) p.active[row] = pushed ? 1 : 0;
        }
    }
}

template <typename R, bool FLAGS, int UN, int US>
__device__ void pull_rows(const PartView<R> &p, const R *table_ptr, int warp, int n_warps) {
    const int lane = threadIdx.x & 31;
    // in registers: the gathers below are opaque to the compiler, which would fetch the view's fields again after each
    const unsigned table = (unsigned)__cvta_generic_to_shared(table_ptr);
    const int table_n = p.table_n, n_chunks = p.n_chunks;
    const R *push = p.push;
    // Long rows: one warp per chunk, UN gathers per lane in flight.  The next chunk's first columns and the descriptor of
    // the one after it are requested before the gathers of the current one.  (The loops are kept rolled: unrolled by the
    // compiler they spilled, which cost more than the loop.)
    const int4 *chunks = reinterpret_cast<const int4 *>(p.chunks);
    const int *cols = p.col + lane;
    const int4 none = make_int4(0, 0, 0, -1);
    int noted = 0, my_slot = -1;
    int4 ch = warp < n_chunks ? __ldg(chunks + warp) : none;
    int4 ahead = warp + n_warps < n_chunks ? __ldg(chunks + warp + n_warps) : none;
    int c[UN];
#pragma unroll
    for (int u = 0; u < UN; ++u) c[u] = u * 32 + lane < ch.z ? __ldcs(cols + ch.y + u * 32) : 0;
#pragma unroll 1
    for (int i = warp; i < n_chunks; i += n_warps) {
        int cn[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) cn[u] = u * 32 + lane < ahead.z ? __ldcs(cols + ahead.y + u * 32) : 0;
        const int4 after = i + 2 * n_warps < n_chunks ? __ldg(chunks + i + 2 * n_warps) : none;
        R sum = 0;
        bool pushed = false;
#pragma unroll 1
        for (int k = 0; k < ch.z; k += UN * 32) {
            R v[UN];
            if (k > 0) {
#pragma unroll
                for (int u = 0; u < UN; ++u) c[u] = k + u * 32 + lane < ch.z ? __ldcs(cols + ch.y + k + u * 32) : 0;
            }
#pragma unroll
            for (int u = 0; u < UN; ++u) {      // lanes beyond the chunk read place 0 and count as not pushed
                v[u] = published(table, table_n, push, c[u]);
                if (k + u * 32 + lane >= ch.z) v[u] = not_pushed<R>();
            }
#pragma unroll
            for (int u = 0; u < UN; ++u) {
                sum += v[u];
                if (FLAGS) pushed = pushed || is_pushed(v[u]);
            }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (FLAGS) pushed = __any_sync(0xffffffffu, pushed);
        if (ch.w < 0) {
            if (lane == 0) {
                p.diff[ch.x] = sum;
                if (FLAGS) p.active[ch.x] = pushed ? 1 : 0;
            }
        } else {
            if (lane == 0) {
                Partial<R> q;
                q.sum = sum;
                q.pushed = pushed ? 1 : 0;
                p.partials[ch.w] = q;
            }
            if (lane == noted) my_slot = ch.w;
            if (++noted == 32) {
                close_slots<R, FLAGS>(p, my_slot);
                noted = 0;
                my_slot = -1;
            }
        }
        ch = ahead;
        ahead = after;
#pragma unroll
        for (int u = 0; u < UN; ++u) c[u] = cn[u];
    }
    close_slots<R, FLAGS>(p, my_slot);
    // Short rows through the plan's stream (columns with an end-of-row flag, ranges of whole rows): a warp takes up to
    // eight neighbouring ranges, one lane per entry and four entries per lane in flight, so the column reads are
    // coalesced; the sums of the rows inside 32 entries come from a segmented scan (fixed tree order), a row that
    // continues into the next 32 carries its sum over.  The warps go on where the chunks left off.
    const int n_ranges = p.n_ranges, per_item = min(8, max(1, n_ranges / n_warps));
    const int n_items = (n_ranges + per_item - 1) / per_item;
    const int *range_row = p.s_range_row, *s_rowptr = p.s_rowptr, *s_rows = p.s_rows, *s_col = p.s_col;
    R *diff = p.diff;
    int *active = p.active;
    int item = (warp - n_chunks) % n_warps;
    if (item < 0) item += n_warps;
#pragma unroll 1
    for (; item < n_items; item += n_warps) {
        int ri = __ldg(range_row + item * per_item);
        const int k0 = __ldg(s_rowptr + ri), k1 = __ldg(s_rowptr + __ldg(range_row + min((item + 1) * per_item, n_ranges)));
        R carry = 0;
        bool carry_pushed = false;
        unsigned e[US];
#pragma unroll
        for (int u = 0; u < US; ++u) e[u] = k0 + u * 32 + lane < k1 ? (unsigned)__ldcs(s_col + k0 + u * 32 + lane) : 0u;
#pragma unroll 1
        for (int base = k0; base < k1; base += US * 32) {
            unsigned en[US];
            R v[US];
#pragma unroll
            for (int u = 0; u < US; ++u) {
                const int k = base + (US + u) * 32 + lane;
                en[u] = k < k1 ? (unsigned)__ldcs(s_col + k) : 0u;
            }
#pragma unroll
            for (int u = 0; u < US; ++u) {
                const bool live = base + u * 32 + lane < k1 && !(e[u] & kPlaceholder);
                v[u] = published(table, table_n, push, live ? (int)(e[u] & kColMask) : 0);
                if (!live) v[u] = not_pushed<R>();
            }
#pragma unroll
            for (int u = 0; u < US; ++u) {
                const bool end = base + u * 32 + lane < k1 && (e[u] & kLastInRow);
                const unsigned ends = __ballot_sync(0xffffffffu, end);
                const unsigned heads = (ends << 1) | 1u;                   // lane starts a row if the lane before ended one
                const int start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
                const unsigned pushers = FLAGS ? __ballot_sync(0xffffffffu, is_pushed(v[u])) : 0u;
                R s = v[u];
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const R t = __shfl_up_sync(0xffffffffu, s, d);
                    if (lane - d >= start) s += t;
                }
                bool pushed = FLAGS && (pushers & (0xffffffffu >> (31 - lane)) & (0xffffffffu << start)) != 0;
                if (start == 0) {                                          // the row open at the start of this batch
                    s += carry;
                    if (FLAGS) pushed = pushed || carry_pushed;
                }
                if (end) {
                    const int row = __ldg(s_rows + ri + __popc(ends & ((1u << lane) - 1u)));
                    diff[row] = s;
                    if (FLAGS) active[row] = pushed ? 1 : 0;
                }
                const R last = __shfl_sync(0xffffffffu, s, 31);
                const bool open = !(ends >> 31);
                carry = open ? last : (R)0;
                if (FLAGS) {
                    const int last_pushed = __shfl_sync(0xffffffffu, (int)pushed, 31);
                    carry_pushed = open && last_pushed != 0;
                }
                ri += __popc(ends);
                e[u] = en[u];
            }
        }
    }
}

// ---- the steps as kernels of their own, for one process per GPU (the exchange between them is the transport's) ----

constexpr int kPullThreads = 768;      // most threads a block of the kernels below has

template <typename R, bool FLAGS>
__global__ void __launch_bounds__(kPullThreads, 1) pr_pull_kernel(PartView<R> p) {
    extern __shared__ __align__(16) char table_bytes[];
    R *table = reinterpret_cast<R *>(table_bytes);
    load_table(p, table);
    __syncthreads();
    // warps numbered across the blocks first: neighbours in the work list go to different SMs
    pull_rows<R, FLAGS, sizeof(R) == 4 ? 8 : 4, 4>(p, table, (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x),
                                                   (int)((blockDim.x >> 5) * gridDim.x));
}

template <typename R>
__global__ void pr_init_kernel(PartView<R> p, R start, int power, R *block_sums) {
    const R tot = block_sum<R>(init_vertices(p, start, power != 0, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x));
    if (threadIdx.x == 0) block_sums[blockIdx.x] = tot;
}

template <typename R>
__global__ void pr_increment_kernel(PartView<R> p, R eps, R *block_sums) {
    const R tot = block_sum<R>(increment_vertices(p, eps, p.scalars[1], blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x));
    if (threadIdx.x == 0) block_sums[blockIdx.x] = tot;
}

template <typename R>
__global__ void pr_power_apply_kernel(PartView<R> p, R damping, int store, R *block_sums) {
    const R dang = p.scalars[2];
    const R tot = block_sum<R>(power_vertices<R, false>(p, damping, dang, store != 0, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x));
    if (threadIdx.x == 0) block_sums[blockIdx.x] = tot;
    if (blockIdx.x == 0 && threadIdx.x == 0) p.scalars[3] = ((R)1 - damping) / p.global_v + damping * (dang / p.global_v);
}

// scalars[slot] += sum of block sums, lane by lane, then a fixed tree.
template <typename R>
__global__ void pr_fold_block_sums_kernel(const R *block_sums, int n_blocks, R *scalars, int slot) {
    if (blockIdx.x != 0 || threadIdx.x >= 32) return;
    R s = 0;
    for (int i = threadIdx.x; i < n_blocks; i += 32) s += block_sums[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) scalars[slot] += s;
}

// globalAcc += globalDiff; globalDiff = 0   (pr_process_messages, pr.cu:435-438)
template <typename R>
__global__ void pr_roll_scalars_kernel(R *scalars) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        scalars[1] += scalars[0];
        scalars[0] = 0;
    }
}

// ---- boundary exchange (Mirror2MasterSend pr.cu:215-297, Master2MirrorSend :299-373) ----

// every mirror row, in plan order; active mirrors carry their diff (pr_generate_sendBuff_mirror :125-148)
template <typename R>
__global__ void pr_pack_up_kernel(const int *__restrict__ up_rows, int n_up, const R *diff, const int *active,
                                  Pair<R> *send, int *counters) {
    int cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_up; i += gridDim.x * blockDim.x) {
        const int row = up_rows[i];
        Pair<R> p;
        const int a = active[row];
        p.val = a ? diff[row] : (R)0;
        p.flag = (R)a;
        send[i] = p;
        cnt += a;
    }
    if (cnt) atomicAdd(counters + 0, cnt);
}

// master rows add what their mirrors sent, ascending rank order (pr_process_recvBuff_Add :167-187)
template <typename R>
__global__ void pr_apply_up_kernel(const int *__restrict__ m_rows, const int *__restrict__ m_off,
                                   const int *__restrict__ m_pos, int n_masters, const Pair<R> *recv, R *diff, int *ubm,
                                   int *counters) {
    int cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_masters; i += gridDim.x * blockDim.x) {
        const int row = m_rows[i];
        R d = diff[row];
        int got = 0;
        for (int k = m_off[i]; k < m_off[i + 1]; ++k) {
            const Pair<R> p = recv[m_pos[k]];
            if (p.flag > 0) {
                d += p.val;
                ++got;
            }
        }
        if (got) {
            diff[row] = d;
            ubm[row] = 1;
            cnt += got;
        }
    }
    if (cnt) atomicAdd(counters + 1, cnt);
}

// masters that changed publish their total to every mirror (pr_generate_sendBuff_master :150-172)
template <typename R>
__global__ void pr_pack_down_kernel(const int *__restrict__ down_rows, int n_down, const R *diff, const int *active,
                                    const int *ubm, Pair<R> *send, int *counters) {
    int cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_down; i += gridDim.x * blockDim.x) {
        const int row = down_rows[i];
        const int f = (active[row] != 0 || ubm[row] != 0) ? 1 : 0;
        Pair<R> p;
        p.val = diff[row];
        p.flag = (R)f;
        send[i] = p;
        cnt += f;
    }
    if (cnt) atomicAdd(counters + 2, cnt);
}

// mirrors take the master's total (pr_process_recvBuff_Exch :189-213)
template <typename R>
__global__ void pr_apply_down_kernel(const int *__restrict__ up_rows, int n_up, const Pair<R> *recv, R *diff, int *ubm,
                                     int *counters) {
    int cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_up; i += gridDim.x * blockDim.x) {
        const Pair<R> p = recv[i];
        if (p.flag > 0) {
            const int row = up_rows[i];
            diff[row] = p.val;
            ubm[row] = 1;
            ++cnt;
        }
    }
    if (cnt) atomicAdd(counters + 3, cnt);
}

__global__ void pr_count_active_kernel(const int *active, int n, int *counters) {
    int cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) cnt += active[i] != 0;
    if (cnt) atomicAdd(counters + 4, cnt);
}

// scalars[2] += n_isolated * (common value of the isolated vertices): ids that occur in no part have no
// edges at all, so they are dangling and all hold scalars[3]; one rank adds their mass.
template <typename R>
__global__ void pr_power_isolated_kernel(R *scalars, long long n_isolated) {
    if (threadIdx.x == 0 && blockIdx.x == 0) scalars[2] += (R)n_isolated * scalars[3];
}

template <typename R>
__global__ void pr_set_scalar_kernel(R *scalars, int slot, R value) {
    if (threadIdx.x == 0 && blockIdx.x == 0) scalars[slot] = value;
}

// ---- all supersteps in one launch, for parts that one process holds on one device ----
//
// A superstep of a small graph is a few microseconds of work, so launches, copies between the parts and the host's
// look at the counts used to be nearly all of its time (R-MAT-16, four parts: 310 us per superstep of the job, two
// parts: 117 us per power iteration).  Here one cooperative launch, one block per SM, runs supersteps back to back
// with a grid barrier between their phases; every block works for one part, blocks are dealt to the parts by their
// number of edges, and boundary vertices are read and written where they lie instead of being packed and copied.
// Measured on the same graphs: 29 us per superstep of the job, 20 us per power iteration.

constexpr int kMaxLocalParts = 64;
constexpr int kHistorySteps = 128;         // supersteps of the job per launch

struct RunControl {
    GridBarrier barrier;
    int steps, done;                       // supersteps run; 1 when the last one exchanged nothing
    unsigned long long t_start, t_pull, t_end;   // nanoseconds: start, end of the first pull, end
    int visited[kMaxLocalParts];
};

template <typename R, int MAXP>
struct RunArgs {
    int n_parts;
    int first_block[MAXP + 1];             // part q's blocks: first_block[q] .. first_block[q + 1]
    PartView<R> part[MAXP];
    R *block_sums;
    RunControl *control;
    unsigned barrier_start, barrier_polls, run;
    int *history;                          // [max_steps][n_parts][4], zero at the start
    // job
    R eps;
    int peval, max_steps, count_visited;
    // power iteration
    R damping;
    int iterations;
    long long n_isolated;
};

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Sum of the blocks' sums in a fixed order, the same value in every thread.
template <typename R>
__device__ R fold_blocks(const R *block_sums) {
    __shared__ double total;
    if (threadIdx.x < 32) {
        R s = 0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += 32) s += block_sums[i];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) total = (double)s;
    }
    __syncthreads();
    return (R)total;
}

// One entry that travelled from (which = 0) or to (3) part q: in registers for few parts, up in the low and down in the
// high half (atomics of a whole warp on one word of shared memory took longer than the exchange itself).
template <int MAXP>
__device__ __forceinline__ void note_moved(unsigned *moved, int *counts, int q, int which) {
    if (MAXP <= 8) {
#pragma unroll
        for (int i = 0; i < (MAXP <= 8 ? MAXP : 1); ++i) moved[i] += i == q ? (which == 0 ? 1u : 0x10000u) : 0u;
    } else {
        atomicAdd(counts + 4 * q + which, 1);
    }
}

// The other parts' arrays, by part.
template <typename R, int MAXP>
struct PartArrays {
    R *diff[MAXP], *push[MAXP], *pr[MAXP], *acc[MAXP];
    int *active[MAXP], *ubm[MAXP];
};

// power_vertices for the vertices that several parts hold, exchange included: a master adds what its mirrors' parts summed
// (ascending rank order), and publishes the new value in every part that holds the vertex.  The mirrors' sums are only
// read and the published values only written between two barriers, so that the exchange needs none of its own (us per
// iteration with / without one; R-MAT-16: two parts, double 20.4 / 20.1, four, float 22.6 / 20.8, eight, double 27.7 / 27.0;
// R-MAT-18, two parts, float 36.7 / 34.3).  Where a mirror publishes lies beside its row in a list of its own: looked up in
// the mirror's part it was one scattered load more and made eight parts slower (28.4).
template <typename R, int MAXP>
__device__ __noinline__ R power_shared_vertices(const PartView<R> &p, const PartArrays<R, MAXP> &of, R damping, R dang, bool last,
                                                   int first, int stride) {
    const R base = ((R)1 - damping) / p.global_v;
    const R share = dang / p.global_v;
    R dangling = 0;
#pragma unroll 1
    for (int m = first; m < p.n_masters; m += stride) {
        const int row = __ldg(p.m_rows + m), k0 = __ldg(p.m_off + m), k1 = __ldg(p.m_off + m + 1);
        R d = p.diff[row];
        const int od = last ? 1 : __ldg(p.out_degree + row), at = !last && p.place ? __ldg(p.place + row) : row;
        // four mirrors at a time, their loads in flight together (most masters have fewer); the last four stay in registers
        int2 to[4], where[4];
        int k = k0;
        while (true) {
            R v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                to[u] = k + u < k1 ? p.pairs[k + u] : make_int2(-1, 0);
                where[u] = k + u < k1 ? p.targets[k + u] : make_int2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = to[u].x < 0 ? (R)0 : of.diff[to[u].x][to[u].y];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (to[u].x >= 0) d += v[u];
            if (k + 4 >= k1) break;
            k += 4;
        }
        const R now = base + damping * (d + share);
        if (last) {
            p.pr[row] = now;
        } else {
            if (od == 0 && __ldg(p.mirror2worker + row) == -1) dangling += now;
            p.push[at] = od == 0 ? not_pushed<R>() : now / od;
        }
        while (true) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int q = to[u].x;
                if (q < 0) continue;
                if (last) of.pr[q][to[u].y] = now;
                else of.push[q][where[u].x] = where[u].y == 0 ? not_pushed<R>() : now / where[u].y;
            }
            k -= 4;
            if (k < k0) break;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                to[u] = p.pairs[k + u];
                where[u] = p.targets[k + u];
            }
        }
    }
    return dangling;
}

// A block whose wait at a barrier ran out: the run is marked as unfinished in every part, since any of them may lack what this
// block would have stored, and the block's share of the values becomes NaN, so that nobody takes the start values, or those
// of some superstep, for a result.
template <typename R, int MAXP>
__device__ __noinline__ void give_up(const RunArgs<R, MAXP> &a, R *pr, int n, int first, int stride) {
    for (int q = threadIdx.x; q < a.n_parts; q += blockDim.x) *a.part[q].unfinished = a.run;
    for (int i = first; i < n; i += stride) pr[i] = (R)NAN;
}

template <typename R, int MAXP, bool JOB, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) pr_run_kernel(const __grid_constant__ RunArgs<R, MAXP> a) {
    extern __shared__ __align__(16) char table_bytes[];
    R *table = reinterpret_cast<R *>(table_bytes);
    __shared__ PartView<R> p;
    __shared__ PartArrays<R, MAXP> of;
    __shared__ int counts[MAXP * 4];
    __shared__ int me_shared;
    if (threadIdx.x == 0) {
        int q = 0;
        while (q + 1 < a.n_parts && (int)blockIdx.x >= a.first_block[q + 1]) ++q;
        me_shared = q;
        p = a.part[q];
    }
    for (int q = threadIdx.x; q < a.n_parts; q += blockDim.x) {
        of.diff[q] = a.part[q].diff;
        of.push[q] = a.part[q].push;
        of.pr[q] = a.part[q].pr;
        of.active[q] = a.part[q].active;
        of.ubm[q] = a.part[q].ubm;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.control->t_start = now_ns();
    __syncthreads();
    const int me = me_shared;
    const int block = (int)blockIdx.x - a.first_block[me], blocks = a.first_block[me + 1] - a.first_block[me];
    const int first = block * blockDim.x + threadIdx.x, stride = blocks * blockDim.x;
    const int warp = (threadIdx.x >> 5) * blocks + block, n_warps = (blockDim.x >> 5) * blocks;
    unsigned phase = a.barrier_start;

    R gdiff = 0, gacc = 0, iso = 0, dangling = 0;
    if (JOB) {
        if (!a.peval) {
            gdiff = p.scalars[0];
            gacc = p.scalars[1];
        }
    } else {
        iso = (R)1 / (R)p.global_v;
        dangling = init_vertices(p, iso, true, first, stride);
    }
    const int n_steps = JOB ? a.max_steps : a.iterations;
    for (int step = 0; step < n_steps; ++step) {
        if (JOB) {
            if (a.peval && step == 0) {
                dangling = init_vertices(p, (R)1, false, first, stride);
            } else {
                gacc += gdiff;
                dangling = increment_vertices(p, a.eps, gacc, first, stride);
            }
        }
        const R mine = block_sum<R>(dangling);
        if (threadIdx.x == 0) a.block_sums[blockIdx.x] = mine;
        if (!grid_barrier(&a.control->barrier, phase, a.barrier_polls)) return give_up(a, p.pr, p.n, first, stride);
        load_table(p, table);
        const R dang = fold_blocks<R>(a.block_sums);      // its barrier also closes the table
        pull_rows<R, JOB, sizeof(R) == 4 || THREADS <= 512 ? 8 : 4, 4>(p, table, warp, n_warps);
        if (JOB) gdiff = dang;
        if (!grid_barrier(&a.control->barrier, phase, a.barrier_polls)) return give_up(a, p.pr, p.n, first, stride);
        if (JOB && step == 0 && blockIdx.x == 0 && threadIdx.x == 0) a.control->t_pull = now_ns();
        if (JOB && a.n_parts > 1) {
            // a master takes what its mirrors hold, in ascending rank order, and hands the total back (Mirror2MasterSend,
            // pr.cu:215-297, Master2MirrorSend, :299-373); only flagged entries travel, and they are counted
            for (int q = threadIdx.x; q < a.n_parts * 4; q += blockDim.x) counts[q] = 0;
            __syncthreads();
            int received = 0, sent = 0;
            unsigned moved[MAXP <= 8 ? MAXP : 1] = {0};
#pragma unroll 1
            for (int m = first; m < p.n_masters; m += stride) {
                const int row = __ldg(p.m_rows + m), k0 = __ldg(p.m_off + m), k1 = __ldg(p.m_off + m + 1);
                R d = p.diff[row];
                const int own = p.active[row];
                int got = 0;
                // four mirrors at a time, their loads in flight together (most masters have fewer)
                for (int k = k0; k < k1; k += 4) {
                    int2 from[4];
                    int flag[4];
                    R v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) from[u] = k + u < k1 ? p.pairs[k + u] : make_int2(-1, 0);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        flag[u] = from[u].x < 0 ? 0 : of.active[from[u].x][from[u].y];
                        v[u] = from[u].x < 0 ? (R)0 : of.diff[from[u].x][from[u].y];
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (flag[u] == 0) continue;
                        d += v[u];
                        ++got;
                        note_moved<MAXP>(moved, counts, from[u].x, 0);
                    }
                }
                received += got;
                if (got) {
                    p.diff[row] = d;
                    p.ubm[row] = 1;
                }
                if (!got && own == 0) continue;
                sent += k1 - k0;
                for (int k = k0; k < k1; ++k) {
                    const int2 to = p.pairs[k];
                    of.diff[to.x][to.y] = d;
                    of.ubm[to.x][to.y] = 1;
                    note_moved<MAXP>(moved, counts, to.x, 3);
                }
            }
            received = __reduce_add_sync(0xffffffffu, received);
            sent = __reduce_add_sync(0xffffffffu, sent);
            if ((threadIdx.x & 31) == 0) {
                if (received) atomicAdd(&counts[4 * me + 1], received);
                if (sent) atomicAdd(&counts[4 * me + 2], sent);
            }
            if (MAXP <= 8) {
#pragma unroll
                for (int q = 0; q < (MAXP <= 8 ? MAXP : 1); ++q) {
                    const unsigned up = __reduce_add_sync(0xffffffffu, moved[q] & 0xffffu);
                    const unsigned down = __reduce_add_sync(0xffffffffu, moved[q] >> 16);
                    if ((threadIdx.x & 31) == 0 && up) atomicAdd(&counts[4 * q], (int)up);
                    if ((threadIdx.x & 31) == 0 && down) atomicAdd(&counts[4 * q + 3], (int)down);
                }
            }
            __syncthreads();
            int *h = a.history + (long long)step * a.n_parts * 4;
            for (int q = threadIdx.x; q < a.n_parts * 4; q += blockDim.x)
                if (counts[q]) atomicAdd(h + q, counts[q]);
            if (!grid_barrier(&a.control->barrier, phase, a.barrier_polls)) return give_up(a, p.pr, p.n, first, stride);
        }
        if (JOB) {
            int sent = 0;      // every block looks at the counts of all parts
            if (a.n_parts > 1)
                for (int q = threadIdx.x; q < a.n_parts * 4; q += blockDim.x) sent |= __ldcg(a.history + (long long)step * a.n_parts * 4 + q);
            const bool done = __syncthreads_or(sent) == 0;
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                a.control->steps = step + 1;
                a.control->done = done ? 1 : 0;
            }
            if (done) break;
        } else {
            const R all = dang + (R)a.n_isolated * iso;
            const bool last = step + 1 == n_steps;
            dangling = power_vertices<R, (MAXP > 1)>(p, a.damping, all, last, first, stride);
            if (MAXP > 1) dangling += power_shared_vertices<R, MAXP>(p, of, a.damping, all, last, first, stride);
            iso = ((R)1 - a.damping) / p.global_v + a.damping * (all / p.global_v);
        }
    }
    if (JOB) {
        if (block == 0 && threadIdx.x == 0) {
            p.scalars[0] = gdiff;
            p.scalars[1] = gacc;
        }
        if (a.count_visited) {      // VisitedSize: the barrier after the pull made every block's flags visible
            int seen = 0;
            for (int i = first; i < p.n; i += stride) seen += p.active[i] != 0;
            seen = __reduce_add_sync(0xffffffffu, seen);
            if ((threadIdx.x & 31) == 0 && seen) atomicAdd(&a.control->visited[me], seen);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.control->t_end = now_ns();
}

}  // namespace drone

#include "pagerank_resident.cuh"
#include "pagerank_stream.cuh"

namespace drone {

// pairs[k] = {part, row} (and targets[k] = {place, out degree} of that row) behind position m_pos[k] of part q's receive
// buffer: peer p's entries start at down_off[p] there and are, in the same order, peer p's up list for q.
struct PeerLists {
    int down_off[kMaxLocalParts + 1];
    const int *up_rows[kMaxLocalParts];    // start of each peer's list for this part
    const int *place[kMaxLocalParts], *out_degree[kMaxLocalParts];
};

__global__ void pr_pairs_kernel(const int *__restrict__ m_pos, int n, const __grid_constant__ PeerLists peers, int n_parts,
                                int2 *pairs, int2 *targets) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int pos = m_pos[k];
        int q = 0;
        while (q + 1 < n_parts && pos >= peers.down_off[q + 1]) ++q;
        const int row = peers.up_rows[q][pos - peers.down_off[q]];
        pairs[k] = make_int2(q, row);
        targets[k] = make_int2(peers.place[q] ? peers.place[q][row] : row, peers.out_degree[q][row]);
    }
}

// role[rows[i]]: that of a mirror, or the row's number in the list of masters.
__global__ void pr_roles_kernel(const int *__restrict__ rows, int n, bool masters, int *role) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) role[rows[i]] = masters ? i : kMirrorRow;
}

// ---- host side ----

static inline int grid1d(long long n, int cap = 148 * 16) {
    long long g = (n + 255) / 256;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

// Fewer vertices than this lie in local-id order: all their published values fit the table in either type, so ordering
// them by how often they are gathered (a sort at creation) would gain nothing.
constexpr long long kOrderMinRows = 16 << 10;
constexpr int kTableBytes = 160 * 1024;        // shared memory for the table; the rest of the SM serves as L1, whose lines are
                                               // what gathers in flight wait in (R-MAT-22: 5.3 ms with 64 to 160 KB, 7.0 with 200)

// View of part p for a pull by `blocks` blocks.  The table holds no more values than a block has edges to gather for
// (filling it costs a read per value, which a small graph's gathers would not pay back), and is left out where the
// published values lie in no particular order and do not all fit.
template <typename R>
static PartView<R> part_view(const drone_pr *p, int blocks) {
    const Side &s = p->plan->side[DRONE_OP_AT];
    const drone_xplan *x = p->xplan;
    PartView<R> v;
    v.n = p->n_local;
    v.global_v = p->global_v;
    v.chunks = s.chunks;
    v.n_chunks = s.n_chunks;
    v.col = s.col;
    v.s_range_row = s.ranges.row;
    v.n_ranges = s.ranges.n;
    v.s_rowptr = s.s_rowptr;
    v.s_rows = s.s_rows;
    v.s_col = s.s_col;
    v.split = s.split;
    v.slot_split = p->slot_split;
    v.arrived = p->arrived;
    v.partials = (Partial<R> *)p->partials;
    v.pr = (R *)p->pr;
    v.acc = (R *)p->acc;
    v.diff = (R *)p->diff;
    v.push = (R *)p->push;
    v.scalars = (R *)p->scalars;
    v.active = p->active;
    v.ubm = p->ubm;
    v.out_degree = p->out_degree;
    v.mirror2worker = p->mirror2worker;
    v.place = p->place;
    v.m_rows = x->d_m_rows;
    v.m_off = x->d_m_off;
    v.n_masters = (int)x->m_rows.size();
    v.pairs = p->pairs;
    v.targets = p->targets;
    v.unfinished = p->unfinished;
    v.rowptr = s.rowptr;
    v.push2 = (R *)p->push2;
    v.role = p->role;
    const long long capacity = kTableBytes / (long long)sizeof(R);
    long long t = std::min<long long>(capacity, p->n_local);
    if (!p->place && p->n_local > capacity) t = 0;
    v.table_n = (int)std::min<long long>(t, p->nnz / std::max(blocks, 1));
    return v;
}

template <typename Kernel>
static int allow_table(Kernel kernel) {
    DRONE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes));
    return DRONE_OK;
}

template <typename R, bool FLAGS>
static int pull(drone_pr *p, cudaStream_t st) {
    if (p->n_local == 0) return DRONE_OK;
    const PartView<R> v = part_view<R>(p, p->sms);
    const int rc = allow_table(pr_pull_kernel<R, FLAGS>);
    if (rc) return rc;
    pr_pull_kernel<R, FLAGS><<<p->sms, kPullThreads, (size_t)v.table_n * sizeof(R), st>>>(v);
    DRONE_LAUNCH_CHECK("pr_pull_kernel");
    return DRONE_OK;
}

// Moves the packed boundary entries of the parts this process steps (one, with one process per GPU): up == true sends their
// `up` slices and receives `down` slices.
struct Transport {
    virtual int move(std::vector<drone_pr *> &parts, bool up, size_t pair_bytes, cudaStream_t st) = 0;
    // where the entries sent to part p lie after move(): its receive buffer unless the transport delivers elsewhere
    virtual const void *received(drone_pr *p) { return p->recv; }
    virtual int allreduce(std::vector<drone_pr *> &parts, int slot, cudaStream_t st) = 0;
    virtual ~Transport() {}
};

struct NcclTransport : Transport {
    int move(std::vector<drone_pr *> &parts, bool up, size_t pair_bytes, cudaStream_t st) override {
        drone_pr *p = parts[0];
        const drone_xplan *x = p->xplan;
        if (x->nranks == 1) return DRONE_OK;
        const std::vector<int> &s_off = up ? x->up_off : x->down_off;
        const std::vector<int> &r_off = up ? x->down_off : x->up_off;
        const ncclDataType_t ty = p->dbl ? ncclDouble : ncclFloat;
        DRONE_NCCL(ncclGroupStart());
        for (int q = 0; q < x->nranks; ++q) {
            if (q == x->rank) continue;
            const size_t ns = (size_t)(s_off[q + 1] - s_off[q]) * 2, nr = (size_t)(r_off[q + 1] - r_off[q]) * 2;
            if (ns) DRONE_NCCL(ncclSend((char *)p->send + (size_t)s_off[q] * pair_bytes, ns, ty, q, p->comm->comm, st));
            if (nr) DRONE_NCCL(ncclRecv((char *)p->recv + (size_t)r_off[q] * pair_bytes, nr, ty, q, p->comm->comm, st));
        }
        DRONE_NCCL(ncclGroupEnd());
        return DRONE_OK;
    }
    int allreduce(std::vector<drone_pr *> &parts, int slot, cudaStream_t st) override {
        drone_pr *p = parts[0];
        if (!p->comm || p->comm->nranks == 1) return DRONE_OK;
        char *ptr = (char *)p->scalars + (size_t)slot * (p->dbl ? 8 : 4);
        DRONE_NCCL(ncclAllReduce(ptr, ptr, 1, p->dbl ? ncclDouble : ncclFloat, ncclSum, p->comm->comm, st));
        return DRONE_OK;
    }
};

// One process per GPU on one NVLink domain: entries are stored straight into the receiver's memory
// (the exchange plan's peer-memory transport, exchange_p2p.cu); the scalar sums stay on NCCL.
struct PeerTransport : NcclTransport {
    const void *landed = nullptr;
    int move(std::vector<drone_pr *> &parts, bool up, size_t pair_bytes, cudaStream_t st) override {
        drone_pr *p = parts[0];
        if (p->xplan->nranks == 1) return DRONE_OK;
        return p2p_move_elements(p->xplan, p->send, pair_bytes, up, st, &landed);
    }
    const void *received(drone_pr *p) override { return p->xplan->nranks == 1 ? p->recv : landed; }
};

// All parts in one process: device-to-device copies, and a kernel that adds the parts' scalars in rank order.
struct ScalarLists {
    void *of[kMaxLocalParts];
};

template <typename R>
__global__ void pr_sum_scalars_kernel(const __grid_constant__ ScalarLists scalars, int n_parts, int slot) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    R s = 0;
    for (int p = 0; p < n_parts; ++p) s += ((R *)scalars.of[p])[slot];
    for (int p = 0; p < n_parts; ++p) ((R *)scalars.of[p])[slot] = s;
}

struct LocalTransport : Transport {
    int move(std::vector<drone_pr *> &parts, bool up, size_t pair_bytes, cudaStream_t st) override {
        const int P = (int)parts.size();
        for (int p = 0; p < P; ++p)
            for (int q = 0; q < P; ++q) {
                if (p == q) continue;
                const std::vector<int> &s_off = up ? parts[p]->xplan->up_off : parts[p]->xplan->down_off;
                const std::vector<int> &r_off = up ? parts[q]->xplan->down_off : parts[q]->xplan->up_off;
                const size_t ns = (size_t)(s_off[q + 1] - s_off[q]), nr = (size_t)(r_off[p + 1] - r_off[p]);
                if (ns != nr)
                    return set_error(DRONE_E_STATE, "exchange plans disagree between parts %d and %d (%zu vs %zu rows)", p, q, ns, nr);
                if (ns)
                    DRONE_CUDA(cudaMemcpyAsync((char *)parts[q]->recv + (size_t)r_off[p] * pair_bytes,
                                               (char *)parts[p]->send + (size_t)s_off[q] * pair_bytes, ns * pair_bytes,
                                               cudaMemcpyDeviceToDevice, st));
            }
        return DRONE_OK;
    }
    int allreduce(std::vector<drone_pr *> &parts, int slot, cudaStream_t st) override {
        ScalarLists lists;
        for (size_t p = 0; p < parts.size(); ++p) lists.of[p] = parts[p]->scalars;
        if (parts[0]->dbl) pr_sum_scalars_kernel<double><<<1, 32, 0, st>>>(lists, (int)parts.size(), slot);
        else pr_sum_scalars_kernel<float><<<1, 32, 0, st>>>(lists, (int)parts.size(), slot);
        DRONE_LAUNCH_CHECK("pr_sum_scalars_kernel");
        return DRONE_OK;
    }
};

// The transport of a job that runs as one process per GPU: peer memory when the exchange plan has it enabled and its
// receive areas are wide enough for a {value, flag} pair, grouped send/recv otherwise.
static bool use_peer_transport(const drone_pr *p) {
    return p->xplan->p2p != nullptr && (size_t)p->xplan->max_features * 4 >= (p->dbl ? 16u : 8u);
}

// mirror -> master (add), master -> mirror (assign)
template <typename R>
static int exchange(std::vector<drone_pr *> &parts, Transport &tr, cudaStream_t st) {
    int rc;
    for (drone_pr *p : parts) {
        const drone_xplan *x = p->xplan;
        const int n_up = (int)x->up_rows.size();
        if (n_up) {
            pr_pack_up_kernel<R><<<grid1d(n_up), 256, 0, st>>>(x->d_up_rows, n_up, (const R *)p->diff, p->active,
                                                              (Pair<R> *)p->send, p->counters);
            DRONE_LAUNCH_CHECK("pr_pack_up_kernel");
        }
    }
    if ((rc = tr.move(parts, true, sizeof(Pair<R>), st))) return rc;
    for (drone_pr *p : parts) {
        const drone_xplan *x = p->xplan;
        const int n_m = (int)x->m_rows.size(), n_down = (int)x->down_rows.size();
        if (n_m) {
            pr_apply_up_kernel<R><<<grid1d(n_m), 256, 0, st>>>(x->d_m_rows, x->d_m_off, x->d_m_pos, n_m,
                                                              (const Pair<R> *)tr.received(p), (R *)p->diff, p->ubm, p->counters);
            DRONE_LAUNCH_CHECK("pr_apply_up_kernel");
        }
        if (n_down) {
            pr_pack_down_kernel<R><<<grid1d(n_down), 256, 0, st>>>(x->d_down_rows, n_down, (const R *)p->diff, p->active,
                                                                  p->ubm, (Pair<R> *)p->send, p->counters);
            DRONE_LAUNCH_CHECK("pr_pack_down_kernel");
        }
    }
    if ((rc = tr.move(parts, false, sizeof(Pair<R>), st))) return rc;
    for (drone_pr *p : parts) {
        const drone_xplan *x = p->xplan;
        const int n_up = (int)x->up_rows.size();
        if (n_up) {
            pr_apply_down_kernel<R><<<grid1d(n_up), 256, 0, st>>>(x->d_up_rows, n_up, (const Pair<R> *)tr.received(p), (R *)p->diff,
                                                                 p->ubm, p->counters);
            DRONE_LAUNCH_CHECK("pr_apply_down_kernel");
        }
    }
    return DRONE_OK;
}

// One superstep of the job, its steps as kernels of their own: the part of a rank whose boundary entries travel between GPUs.
template <typename R>
static int delta_step(std::vector<drone_pr *> &parts, bool peval, Transport &tr, drone_pr_response *res, cudaStream_t st) {
    using clock = std::chrono::steady_clock;
    const auto t0 = clock::now();
    int rc;
    for (drone_pr *p : parts) {
        DRONE_CUDA(cudaMemsetAsync(p->counters, 0, sizeof(int) * 8, st));
        p->run = 0;
        const PartView<R> v = part_view<R>(p, p->sms);
        const int grid = grid1d(p->n_local, kReduceBlocks);
        if (peval) {
            DRONE_CUDA(cudaMemsetAsync(p->scalars, 0, sizeof(R) * 4, st));
            pr_init_kernel<R><<<grid, 256, 0, st>>>(v, (R)1, 0, (R *)p->block_sums);
            DRONE_LAUNCH_CHECK("pr_init_kernel");
        } else {
            pr_roll_scalars_kernel<R><<<1, 32, 0, st>>>((R *)p->scalars);
            DRONE_LAUNCH_CHECK("pr_roll_scalars_kernel");
            pr_increment_kernel<R><<<grid, 256, 0, st>>>(v, (R)p->eps, (R *)p->block_sums);
            DRONE_LAUNCH_CHECK("pr_increment_kernel");
        }
        pr_fold_block_sums_kernel<R><<<1, 32, 0, st>>>((const R *)p->block_sums, grid, (R *)p->scalars, 0);
        DRONE_LAUNCH_CHECK("pr_fold_block_sums_kernel");
        if ((rc = pull<R, true>(p, st))) return rc;
        p->started = true;
    }
    DRONE_CUDA(cudaStreamSynchronize(st));
    const auto t1 = clock::now();
    if ((rc = exchange<R>(parts, tr, st))) return rc;
    if ((rc = tr.allreduce(parts, 0, st))) return rc;
    std::vector<int> h(8 * parts.size());
    for (size_t i = 0; i < parts.size(); ++i) {
        drone_pr *p = parts[i];
        if (p->n_local > 0) {
            pr_count_active_kernel<<<grid1d(p->n_local), 256, 0, st>>>(p->active, p->n_local, p->counters);
            DRONE_LAUNCH_CHECK("pr_count_active_kernel");
        }
        DRONE_CUDA(cudaMemcpyAsync(h.data() + 8 * i, p->counters, sizeof(int) * 8, cudaMemcpyDeviceToHost, st));
    }
    DRONE_CUDA(cudaStreamSynchronize(st));
    const auto t2 = clock::now();
    for (size_t i = 0; i < parts.size(); ++i) {
        drone_pr_response &r = res[i];
        r.Mirror2MasterSendSize = h[8 * i + 0];
        r.Mirror2MasterRecvSize = h[8 * i + 1];
        r.Master2MirrorSendSize = h[8 * i + 2];
        r.Master2MirrorRecvSize = h[8 * i + 3];
        r.VisitedSize = h[8 * i + 4];
        r.LocalVertexSize = parts[i]->n_local;
        r.CalTime = std::chrono::duration<float>(t1 - t0).count();
        r.SendTime = std::chrono::duration<float>(t2 - t1).count();
    }
    return DRONE_OK;
}

template <typename R>
static int power_iterations(std::vector<drone_pr *> &parts, int iterations, double damping, Transport &tr, cudaStream_t st) {
    int rc;
    for (drone_pr *p : parts) {
        const R start = (R)1 / (R)p->global_v;
        DRONE_CUDA(cudaMemsetAsync(p->scalars, 0, sizeof(R) * 4, st));
        pr_init_kernel<R><<<grid1d(p->n_local, kReduceBlocks), 256, 0, st>>>(part_view<R>(p, p->sms), start, 1, (R *)p->block_sums);
        DRONE_LAUNCH_CHECK("pr_init_kernel");
        pr_set_scalar_kernel<R><<<1, 32, 0, st>>>((R *)p->scalars, 3, start);
        DRONE_LAUNCH_CHECK("pr_set_scalar_kernel");
        p->started = false;
        p->run = 0;
    }
    for (int it = 0; it < iterations; ++it) {
        for (drone_pr *p : parts) {
            DRONE_CUDA(cudaMemsetAsync((char *)p->scalars + 2 * sizeof(R), 0, sizeof(R), st));
            pr_fold_block_sums_kernel<R><<<1, 32, 0, st>>>((const R *)p->block_sums, grid1d(p->n_local, kReduceBlocks), (R *)p->scalars, 2);
            DRONE_LAUNCH_CHECK("pr_fold_block_sums_kernel");
            if (p->xplan->rank == 0 && p->n_isolated > 0) {
                pr_power_isolated_kernel<R><<<1, 32, 0, st>>>((R *)p->scalars, p->n_isolated);
                DRONE_LAUNCH_CHECK("pr_power_isolated_kernel");
            }
            // with flags: the exchange's pack kernels send the rows that have some in-neighbour
            if ((rc = pull<R, true>(p, st))) return rc;
        }
        if ((rc = exchange<R>(parts, tr, st))) return rc;
        if ((rc = tr.allreduce(parts, 2, st))) return rc;
        for (drone_pr *p : parts) {
            // new values, and what they publish for the next iteration, in one pass
            pr_power_apply_kernel<R><<<grid1d(p->n_local, kReduceBlocks), 256, 0, st>>>(part_view<R>(p, p->sms), (R)damping,
                                                                                       it + 1 == iterations, (R *)p->block_sums);
            DRONE_LAUNCH_CHECK("pr_power_apply_kernel");
        }
    }
    return DRONE_OK;
}

static int prepare_parts(std::vector<drone_pr *> &parts) {
    for (drone_pr *p : parts) {
        if (!p) return set_error(DRONE_E_INVALID, "PageRank handle is NULL");
        const int rc = xplan_ensure_device(p->xplan);
        if (rc) return rc;
    }
    return DRONE_OK;
}

// Where every part's master rows find their mirrors in the other parts' arrays; made once per set of handles.
static int prepare_pairs(std::vector<drone_pr *> &parts, cudaStream_t st) {
    const int P = (int)parts.size();
    std::vector<unsigned long long> key;
    for (drone_pr *p : parts) {
        key.push_back(p->xplan->uid);
        key.push_back(p->uid);
    }
    for (int q = 0; q < P; ++q) {
        drone_pr *me = parts[q];
        const drone_xplan *x = me->xplan;
        if (me->pairs_for == key || P == 1) continue;
        PeerLists lists;
        for (int p = 0; p <= P; ++p) lists.down_off[p] = x->down_off[p];
        for (int p = 0; p < P; ++p) {
            const drone_xplan *y = parts[p]->xplan;
            const int ns = y->up_off[q + 1] - y->up_off[q], nr = x->down_off[p + 1] - x->down_off[p];
            if (p != q && ns != nr)
                return set_error(DRONE_E_STATE, "exchange plans disagree between parts %d and %d (%d vs %d rows)", p, q, ns, nr);
            lists.up_rows[p] = y->d_up_rows + y->up_off[q];
            lists.place[p] = parts[p]->place;
            lists.out_degree[p] = parts[p]->out_degree;
        }
        const int n = (int)x->m_pos.size();
        if (n > 0) {
            pr_pairs_kernel<<<grid1d(n), 256, 0, st>>>(x->d_m_pos, n, lists, P, me->pairs, me->targets);
            DRONE_LAUNCH_CHECK("pr_pairs_kernel");
        }
        if (me->n_local > 0) {
            DRONE_CUDA(cudaMemsetAsync(me->role, 0xff, sizeof(int) * (size_t)me->n_local, st));      // kOwnRow
            const int up = (int)x->up_rows.size(), masters = (int)x->m_rows.size();
            if (up > 0) {
                pr_roles_kernel<<<grid1d(up), 256, 0, st>>>(x->d_up_rows, up, false, me->role);
                DRONE_LAUNCH_CHECK("pr_roles_kernel");
            }
            if (masters > 0) {
                pr_roles_kernel<<<grid1d(masters), 256, 0, st>>>(x->d_m_rows, masters, true, me->role);
                DRONE_LAUNCH_CHECK("pr_roles_kernel");
            }
        }
        me->pairs_for = key;
    }
    return DRONE_OK;
}

// Number of a launch in the process, never 0.
static unsigned next_run() {
    static std::atomic<unsigned> runs{0};
    unsigned run;
    do run = ++runs;
    while (run == 0);
    return run;
}

// What one persistent launch is asked to do.
struct RunRequest {
    bool job = false;              // supersteps of the job; otherwise the power iteration
    bool peval = false, count_visited = false;
    int max_steps = 0;
    int iterations = 0;
    double damping = 0;
};

// Whether the parts' edges and rows fit the shared memory of the blocks they are dealt to, and how that is divided.  The table
// takes what is left, up to a value for every 8 bytes of which a block has an edge; with less than a quarter of that the kernel
// that leaves the columns in global memory has the better table.
constexpr size_t kSliceBytes = 216 * 1024;
constexpr long long kSliceEdges = kSliceBytes / sizeof(unsigned);      // more edges per SM than this never fit

static bool all_values_or_order(const drone_pr *p, size_t value) { return p->place || p->n_local <= kTableBytes / (int)value; }

// How many edges the largest slice may have above the average: a row lies in one block, and the others wait for it.  An iteration of
// balanced slices is at least 4 us shorter than one of the other kernels, which cut long rows (R-MAT-12 to R-MAT-17, 65,536 vertices
// with 524,000 edges: 3.4 to 7 us); what an edge costs the largest slice, in ns, depends on how much of the published values its table
// and L1 hold.  Measured with one vertex of many in-edges, us of 20 iterations on 65,536 vertices, other kernels / slices: float 16,000
// in-edges 219 / 201, 24,000 206 / 265, 48,000 217 / 866; double 8,000 221 / 182, 16,000 223 / 251; two parts, double, 24,000 332 /
// 300, 48,000 333 / 401; 131,072 vertices, double, 24,000 344 / 568 (1.3 ns; R-MAT-17, whose gathers the table serves, 0.3: 318 / 269
// with 5,400 edges above the average); 16,384 vertices, float, 16,000 191 / 159.
static long long edges_above_average(size_t value, long long n_local) {
    const double ns[2][3] = {{0.20, 0.32, 0.45}, {0.29, 0.44, 0.6}};
    const long long published = (long long)value * n_local;
    return (long long)(4000 / ns[value == 8][published <= 128 << 10 ? 0 : published <= 512 << 10 ? 1 : 2]);
}

static bool slices_fit(int n_parts, drone_pr *const *parts, const int *first_block, size_t value, bool job, SliceRoom *room, size_t *bytes) {
    *room = SliceRoom{0, 0, 0};
    long long table = 0;
    for (int q = 0; q < n_parts; ++q) {
        const drone_pr *p = parts[q];
        const int blocks = first_block[q + 1] - first_block[q];
        if (p->n_local == 0 || blocks > (int)p->slices.size()) return false;
        const int2 most = p->slices[blocks - 1];
        if (most.y - p->nnz / blocks > edges_above_average(value, p->n_local)) return false;
        room->rows = std::max(room->rows, (most.x + 3) & ~3);
        room->edges = std::max(room->edges, most.y);
        if (!all_values_or_order(p, value)) continue;
        const long long worth = (long long)p->nnz / blocks * 8 / (long long)value;
        table = std::max(table, std::min<long long>(worth, std::min<long long>(kTableBytes / (long long)value, p->n_local)));
    }
    const size_t used = slice_row_bytes(value, job, n_parts > 1) * (size_t)room->rows + sizeof(unsigned) * (size_t)room->edges;
    if (used > kSliceBytes) return false;
    const long long left = (long long)((kSliceBytes - used) / value) & ~3LL;
    if (left < table / 4) return false;
    room->table = (int)std::min<long long>((table + 3) & ~3LL, left);
    *bytes = used + value * (size_t)room->table;
    return true;
}

// A block has at least about 1024 edges and vertices to work through; more blocks only make the barriers longer.
static int run_blocks(long long edges, int n_parts, int sms) {
    return std::max(n_parts, (int)std::min<long long>(sms, (edges + 1023) / 1024));
}

static bool slices_fit_alone(drone_pr *p) {
    const int first_block[2] = {0, run_blocks((long long)p->nnz + p->n_local, 1, p->sms)};
    SliceRoom room;
    size_t bytes = 0;
    return slices_fit(1, &p, first_block, p->dbl ? 8 : 4, false, &room, &bytes);
}

// How large the blocks' slices would be, for the runs that keep them in shared memory.
static int measure_slices(drone_pr *p, const Side &side) {
    pr_slice_sizes_kernel<<<p->sms, 256>>>(side.rowptr, p->n_local, (int2 *)p->block_sums);
    DRONE_LAUNCH_CHECK("pr_slice_sizes_kernel");
    p->slices.resize((size_t)p->sms);
    DRONE_CUDA(cudaMemcpy(p->slices.data(), p->block_sums, sizeof(int2) * p->slices.size(), cudaMemcpyDeviceToHost));
    return DRONE_OK;
}

// The edges as one stream; where the device has no room for it power iterations do without (pr_run_kernel).
static int make_stream(drone_pr *p) {
    p->stream_block.add(&p->stream_od, sizeof(int) * (size_t)p->n_local);
    const int warps = p->sms * (p->dbl ? stream_threads<double>() : stream_threads<float>()) / 32;
    p->stream_block.add(&p->stream_tails, (p->dbl ? 8 : 4) * 4 * (size_t)warps);      // a piece each
    const int rc = plan_rows_in_order(p->plan, DRONE_OP_AT, p->place, warps, &p->stream, &p->stream_block, nullptr);
    if (rc == kNoRoom) {
        p->stream_block.release();
        p->stream = RowStream();
        return DRONE_OK;
    }
    if (rc) return rc;
    pr_stream_degrees_kernel<<<grid1d(p->n_local), 256>>>(p->stream.row_of, p->out_degree, p->mirror2worker, p->n_local, p->stream_od);
    DRONE_LAUNCH_CHECK("pr_stream_degrees_kernel");
    DRONE_CUDA(cudaDeviceSynchronize());
    return DRONE_OK;
}

template <typename R, int MAXP, bool JOB>
static int launch_run(std::vector<drone_pr *> &parts, const RunRequest &rq, cudaStream_t st) {
    const int P = (int)parts.size();
    drone_pr *lead = parts[0];
    long long edges = 0;
    for (drone_pr *p : parts) edges += (long long)p->nnz + p->n_local;
    const int grid = run_blocks(edges, P, lead->sms);
    // More warps hide more of a chunk's latencies (R-MAT-22: 6.5 ms with 512 threads, 5.3 with 768); fewer meet sooner at
    // a barrier and have the registers for more gathers each (R-MAT-16, two parts: 0.40 against 0.46 ms).
    const int threads = edges / grid > 32768 ? kPullThreads : 512;
    RunArgs<R, MAXP> a;
    a.n_parts = P;
    // blocks dealt to the parts by their share of the work, at least one each
    long long before = 0;
    a.first_block[0] = 0;
    for (int q = 0; q < P; ++q) {
        before += (long long)parts[q]->nnz + parts[q]->n_local;
        int end = edges > 0 ? (int)((before * grid + edges / 2) / edges) : q + 1;
        end = std::max(end, a.first_block[q] + 1);
        end = std::min(end, grid - (P - 1 - q));
        a.first_block[q + 1] = q + 1 == P ? grid : end;
    }
    size_t table = 0;
    for (int q = 0; q < P; ++q) {
        a.part[q] = part_view<R>(parts[q], a.first_block[q + 1] - a.first_block[q]);
        table = std::max(table, (size_t)a.part[q].table_n * sizeof(R));
    }
    a.block_sums = (R *)lead->block_sums;
    a.control = (RunControl *)lead->control;
    a.run = next_run();
    a.barrier_start = lead->barrier_start;
    a.barrier_polls = lead->barrier_polls;
    a.history = (int *)(lead->control + sizeof(RunControl));
    a.eps = (R)lead->eps;
    a.peval = rq.peval;
    a.max_steps = rq.max_steps;
    a.count_visited = rq.count_visited;
    a.damping = (R)rq.damping;
    a.iterations = rq.iterations;
    a.n_isolated = lead->n_isolated;
    DRONE_CUDA(cudaMemsetAsync(lead->control, 0, sizeof(RunControl) + (JOB ? sizeof(int) * 4 * (size_t)P * rq.max_steps : 0), st));
    if (lead->barrier_start != 0)
        DRONE_CUDA(cudaMemcpyAsync(&a.control->barrier.arrived, &lead->barrier_start, sizeof(unsigned), cudaMemcpyHostToDevice, st));
    SliceRoom room;
    size_t bytes = 0;
    // The job of one part is a single superstep, which does not repay filling the slices (float, R-MAT-16 61 / 69 us a call, R-MAT-17
    // 68 / 82).  With several parts a superstep by itself (R-MAT-16 in two parts, double, 66 / 78) takes the kernel that the whole job
    // takes, so that the bits are the same.
    if ((!JOB || P > 1) && slices_fit(P, parts.data(), a.first_block, sizeof(R), JOB, &room, &bytes)) {
        for (int q = 0; q < P; ++q) a.part[q].table_n = all_values_or_order(parts[q], sizeof(R)) ? std::min(room.table, parts[q]->n_local) : 0;
        auto kernel = pr_resident_kernel<R, MAXP, JOB>;
        DRONE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSliceBytes));
        void *args[] = {&a, &room};
        DRONE_CUDA(cudaLaunchCooperativeKernel((const void *)kernel, dim3(grid), dim3(kSliceThreads), args, bytes, st));
    } else if constexpr (MAXP == 1) {
        return launch_run<R, 8, JOB>(parts, rq, st);      // few vertices with very many edges, in no order (part_view)
    } else {
        auto kernel = threads == 512 ? pr_run_kernel<R, MAXP, JOB, 512> : pr_run_kernel<R, MAXP, JOB, kPullThreads>;
        const int rc = allow_table(kernel);
        if (rc) return rc;
        void *args[] = {&a};
        DRONE_CUDA(cudaLaunchCooperativeKernel((const void *)kernel, dim3(grid), dim3(threads), args, table, st));
    }
    count_launch();
    for (drone_pr *p : parts) {
        p->started = JOB;
        p->run = a.run;
    }
    return DRONE_OK;
}

template <typename R>
static int launch_stream(drone_pr *p, const RunRequest &rq, cudaStream_t st) {
    StreamArgs<R> a;
    a.part = part_view<R>(p, p->sms);
    a.part.table_n = std::min<int>(a.part.table_n, kStreamTableBytes / (int)sizeof(R));
    a.rows = p->stream;
    a.od = p->stream_od;
    a.sum = (R *)p->push2;
    a.tails = (R *)p->stream_tails;
    a.block_sums = (R *)p->block_sums;
    a.control = (RunControl *)p->control;
    a.barrier_start = p->barrier_start;
    a.barrier_polls = p->barrier_polls;
    a.run = p->run = next_run();
    a.damping = (R)rq.damping;
    a.iterations = rq.iterations;
    a.n_isolated = p->n_isolated;
    p->started = false;
    DRONE_CUDA(cudaMemsetAsync(p->control, 0, sizeof(RunControl), st));
    if (p->barrier_start != 0)
        DRONE_CUDA(cudaMemcpyAsync(&a.control->barrier.arrived, &p->barrier_start, sizeof(unsigned), cudaMemcpyHostToDevice, st));
    auto kernel = p->stream.most_spanned > kSerialPieces ? pr_stream_kernel<R, true> : pr_stream_kernel<R, false>;
    const int rc = allow_table(kernel);
    if (rc) return rc;
    void *args[] = {&a};
    DRONE_CUDA(cudaLaunchCooperativeKernel((const void *)kernel, dim3(p->sms), dim3(stream_threads<R>()), args, (size_t)a.part.table_n * sizeof(R),
                                           st));
    count_launch();
    return DRONE_OK;
}

static int run_local(std::vector<drone_pr *> &parts, const RunRequest &rq, cudaStream_t st) {
    const drone_pr *lead = parts[0];
    const int rc = prepare_pairs(parts, st);
    if (rc) return rc;
    const bool few = parts.size() <= 8;
    if (!rq.job && lead->stream.col) return lead->dbl ? launch_stream<double>(parts[0], rq, st) : launch_stream<float>(parts[0], rq, st);
    if (lead->dbl) {
        if (rq.job) return few ? launch_run<double, 8, true>(parts, rq, st) : launch_run<double, kMaxLocalParts, true>(parts, rq, st);
        if (parts.size() == 1) return launch_run<double, 1, false>(parts, rq, st);
        return few ? launch_run<double, 8, false>(parts, rq, st) : launch_run<double, kMaxLocalParts, false>(parts, rq, st);
    }
    if (rq.job) return few ? launch_run<float, 8, true>(parts, rq, st) : launch_run<float, kMaxLocalParts, true>(parts, rq, st);
    if (parts.size() == 1) return launch_run<float, 1, false>(parts, rq, st);
    return few ? launch_run<float, 8, false>(parts, rq, st) : launch_run<float, kMaxLocalParts, false>(parts, rq, st);
}

// What the persistent launch left: its control block and the counts of `steps` supersteps.
static int read_control(std::vector<drone_pr *> &parts, int steps, RunControl *c, int *history, cudaStream_t st) {
    const drone_pr *lead = parts[0];
    DRONE_CUDA(cudaMemcpyAsync(c, lead->control, sizeof(RunControl), cudaMemcpyDeviceToHost, st));
    if (history)
        DRONE_CUDA(cudaMemcpyAsync(history, lead->control + sizeof(RunControl), sizeof(int) * 4 * parts.size() * steps,
                                   cudaMemcpyDeviceToHost, st));
    DRONE_CUDA(cudaStreamSynchronize(st));
    if (!c->barrier.failed) return DRONE_OK;
    for (drone_pr *p : parts) p->started = false;
    return set_error(DRONE_E_STATE, "PageRank: a wait between the blocks of a superstep ran out");
}

// Parts in one process usually run in the persistent kernel.  Handles made with DRONE_PR_SEPARATE_STEPS=1 take the kernels and
// the order of one process per GPU instead, with copies for messages: so that those can be tested on one GPU.
static bool local_parts_run_separately(const std::vector<drone_pr *> &parts) {
    for (const drone_pr *p : parts)
        if (!p->separate_steps) return false;
    return true;
}

// One superstep of all given parts.
static int step_parts(std::vector<drone_pr *> &parts, bool peval, drone_pr_response *res, cudaStream_t st) {
    for (drone_pr *p : parts)
        if (!peval && !p->started) return set_error(DRONE_E_STATE, "PR_IncEVal called before PR_PEVal");
    if (local_parts_run_separately(parts)) {
        LocalTransport copies;
        return parts[0]->dbl ? delta_step<double>(parts, peval, copies, res, st) : delta_step<float>(parts, peval, copies, res, st);
    }
    RunRequest rq;
    rq.job = true;
    rq.peval = peval;
    rq.max_steps = 1;
    rq.count_visited = true;
    int rc = run_local(parts, rq, st);
    if (rc) return rc;
    RunControl c;
    std::vector<int> h(4 * parts.size());
    if ((rc = read_control(parts, 1, &c, h.data(), st))) return rc;
    for (size_t i = 0; i < parts.size(); ++i) {
        drone_pr_response &r = res[i];
        r.Mirror2MasterSendSize = h[4 * i + 0];
        r.Mirror2MasterRecvSize = h[4 * i + 1];
        r.Master2MirrorSendSize = h[4 * i + 2];
        r.Master2MirrorRecvSize = h[4 * i + 3];
        r.VisitedSize = c.visited[i];
        r.LocalVertexSize = parts[i]->n_local;
        r.CalTime = (float)((c.t_pull - c.t_start) * 1e-9);
        r.SendTime = (float)((c.t_end - c.t_pull) * 1e-9);
    }
    return DRONE_OK;
}

}  // namespace drone

using namespace drone;

extern "C" {

int drone_pr_destroy(drone_pr *p);

int drone_pr_create(drone_pr **out, int n_local, int global_v, int nnz, const int *d_index, const int *d_dst,
                    const int *d_out_degree, const int *d_mirror2worker, drone_xplan *xplan, drone_comm *comm,
                    int use_double, double eps) {
    DRONE_REQUIRE(out != nullptr, "drone_pr_create: out is NULL");
    *out = nullptr;
    DRONE_REQUIRE(n_local >= 0 && global_v > 0 && nnz >= 0, "drone_pr_create: bad sizes");
    DRONE_REQUIRE(xplan != nullptr, "drone_pr_create: exchange plan is NULL");
    DRONE_REQUIRE(xplan->n_local == n_local, "drone_pr_create: exchange plan has %d rows, graph has %d", xplan->n_local,
                  n_local);
    DRONE_REQUIRE(xplan->nranks == 1 || comm == nullptr || (comm->nranks == xplan->nranks && comm->rank == xplan->rank),
                  "drone_pr_create: communicator and exchange plan disagree on rank");
    DRONE_REQUIRE(n_local == 0 || (d_index && d_out_degree && d_mirror2worker), "drone_pr_create: NULL device array");
    DRONE_REQUIRE(eps >= 0, "drone_pr_create: eps=%g is negative", eps);
    drone_pr *p = new (std::nothrow) drone_pr();
    if (!p) return set_error(DRONE_E_INVALID, "drone_pr_create: out of host memory");
    static std::atomic<unsigned long long> created{0};
    p->uid = ++created;
    p->n_local = n_local;
    p->global_v = global_v;
    p->nnz = nnz;
    p->dbl = use_double != 0;
    p->eps = eps;
    p->xplan = xplan;
    p->comm = comm;
    p->barrier_start = barrier_start();
    p->barrier_polls = barrier_polls();
    const char *separate = getenv("DRONE_PR_SEPARATE_STEPS");
    p->separate_steps = separate && separate[0] == '1';
    cudaGetDevice(&p->device);
    const size_t rs = p->dbl ? 8 : 4;
    const size_t n1 = (size_t)(n_local > 0 ? n_local : 1);
    int rc = DRONE_OK;
    do {
        // transposed graph and the split of long rows: reuse the aggregation plan, whose coefficients are never read here, so
        // any nnz words do
        rc = plan_create_untagged(&p->plan, n_local, nnz, d_index, d_dst, reinterpret_cast<const float *>(d_dst), nullptr, nullptr,
                                  DRONE_PLAN_AT, nullptr);
        if (rc) break;
        {
            const char *v = getenv("DRONE_PR_ORDER_MIN_ROWS");
            const long long min_rows = (v && *v) ? atoll(v) : kOrderMinRows;
            if (min_rows > 0 && n_local >= min_rows && nnz > 0) {
                rc = plan_order_columns_by_frequency(p->plan, DRONE_OP_AT, d_index, &p->place, nullptr);
                if (rc) break;
            }
        }
        cudaError_t e = cudaSuccess;
        p->block.add(&p->out_degree, sizeof(int) * n1);
        p->block.add(&p->mirror2worker, sizeof(int) * n1);
        p->block.add(&p->pr, rs * n1);
        p->block.add(&p->acc, rs * n1);
        p->block.add(&p->diff, rs * n1);
        p->block.add(&p->push, rs * n1);
        p->block.add(&p->push2, rs * n1);
        p->block.add(&p->active, sizeof(int) * n1);
        p->block.add(&p->ubm, sizeof(int) * n1);
        p->block.add(&p->scalars, 8 * 4);
        p->block.add(&p->block_sums, 8 * kReduceBlocks);
        const Side &side = p->plan->side[DRONE_OP_AT];
        p->block.add(&p->partials, 2 * rs * (size_t)side.n_partials);
        p->block.add(&p->slot_split, sizeof(int) * (size_t)side.n_partials);
        p->block.add(&p->arrived, sizeof(int) * (size_t)side.n_split_rows);
        const size_t nb = std::max(xplan->up_rows.size(), xplan->down_rows.size());
        p->block.add(&p->send, 2 * rs * nb);
        p->block.add(&p->recv, 2 * rs * nb);
        p->block.add(&p->counters, sizeof(int) * 8);
        p->block.add(&p->unfinished, sizeof(unsigned));
        if (xplan->nranks > 1 && xplan->nranks <= kMaxLocalParts) {      // for runs over all parts in one process
            p->block.add(&p->pairs, sizeof(int2) * xplan->m_pos.size());
            p->block.add(&p->targets, sizeof(int2) * xplan->m_pos.size());
            p->block.add(&p->role, sizeof(int) * n1);
        }
        const size_t control_bytes = sizeof(RunControl) + sizeof(int) * 4 * (size_t)xplan->nranks * kHistorySteps;
        p->block.add(&p->control, control_bytes);
        if (e == cudaSuccess) e = p->block.make();
        if (e == cudaSuccess) e = cudaMemset(p->control, 0, control_bytes);
        if (e == cudaSuccess) e = cudaMemset(p->unfinished, 0, sizeof(unsigned));
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, p->device);
        if (e == cudaSuccess && side.n_split_rows > 0) {
            e = cudaMemset(p->arrived, 0, sizeof(int) * (size_t)side.n_split_rows);
            if (e == cudaSuccess && (rc = fill_slot_split(side, p->slot_split, nullptr))) break;
        }
        if (e != cudaSuccess) { rc = set_error(DRONE_E_CUDA, "drone_pr_create: cudaMalloc failed: %s", cudaGetErrorString(e)); break; }
        // (DRONE_PR_SLICES=0: no run keeps its rows in shared memory)
        const char *slices = getenv("DRONE_PR_SLICES");
        const bool may_slice = !(slices && slices[0] == '0') && (xplan->nranks == 1 || !comm);
        if (may_slice && n_local > 0 && nnz <= (long long)p->sms * kSliceEdges && p->sms <= kBlockSums && (rc = measure_slices(p, side))) break;
        if (n_local > 0) {
            e = cudaMemcpy(p->out_degree, d_out_degree, sizeof(int) * (size_t)n_local, cudaMemcpyDeviceToDevice);
            if (e == cudaSuccess) e = cudaMemcpy(p->mirror2worker, d_mirror2worker, sizeof(int) * (size_t)n_local, cudaMemcpyDeviceToDevice);
            if (e != cudaSuccess) { rc = set_error(DRONE_E_CUDA, "drone_pr_create: copy failed: %s", cudaGetErrorString(e)); break; }
        }
        // one part whose slices do not fit: its edges as one stream
        if (xplan->nranks == 1 && p->place && nnz > 0 && !slices_fit_alone(p) && (rc = make_stream(p))) break;
    } while (0);
    if (rc) {
        drone_pr_destroy(p);
        return rc;
    }
    *out = p;
    return DRONE_OK;
}

int drone_pr_destroy(drone_pr *p) {
    if (!p) return DRONE_OK;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(p->device);
    drone_plan_destroy(p->plan);
    cudaFree(p->place);
    p->block.release();
    p->stream_block.release();
    if (prev >= 0) cudaSetDevice(prev);
    delete p;
    return DRONE_OK;
}

static int run_step(drone_pr *p, bool peval, drone_pr_response *res, void *stream) {
    std::vector<drone_pr *> parts{p};
    OnDevice dev;
    int rc = dev.enter(p->device);
    if (rc) return rc;
    if ((rc = prepare_parts(parts))) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (p->xplan->nranks == 1) return step_parts(parts, peval, res, st);
    if (!peval && !p->started) return set_error(DRONE_E_STATE, "PR_IncEVal called before PR_PEVal");
    PeerTransport peer;
    NcclTransport nccl;
    NcclTransport &tr = use_peer_transport(p) ? peer : nccl;
    return p->dbl ? delta_step<double>(parts, peval, tr, res, st) : delta_step<float>(parts, peval, tr, res, st);
}

int drone_pr_peval(drone_pr *p, drone_pr_response *res, void *stream) {
    DRONE_REQUIRE(p && res, "drone_pr_peval: NULL argument");
    DRONE_REQUIRE(p->xplan->nranks == 1 || p->comm, "drone_pr_peval: %d ranks but no communicator", p->xplan->nranks);
    return run_step(p, true, res, stream);
}

int drone_pr_inceval(drone_pr *p, drone_pr_response *res, void *stream) {
    DRONE_REQUIRE(p && res, "drone_pr_inceval: NULL argument");
    DRONE_REQUIRE(p->xplan->nranks == 1 || p->comm, "drone_pr_inceval: %d ranks but no communicator", p->xplan->nranks);
    return run_step(p, false, res, stream);
}

// The handles of all parts of one partition, as the *_local entry points take them.
static int local_parts(const char *who, int n_parts, drone_pr **prs, std::vector<drone_pr *> *parts) {
    DRONE_REQUIRE(n_parts >= 1 && n_parts <= kMaxLocalParts && prs, "%s: bad arguments", who);
    parts->assign(prs, prs + n_parts);
    for (int i = 0; i < n_parts; ++i) {
        const drone_pr *p = (*parts)[i];
        DRONE_REQUIRE(p && p->xplan->nranks == n_parts && p->xplan->rank == i && p->dbl == prs[0]->dbl && p->device == prs[0]->device,
                      "%s: handle %d is not part %d of %d", who, i, i, n_parts);
    }
    return DRONE_OK;
}

int drone_pr_step_local(int n_parts, drone_pr **prs, int is_peval, drone_pr_response *res, void *stream) {
    std::vector<drone_pr *> parts;
    int rc = local_parts("drone_pr_step_local", n_parts, prs, &parts);
    if (rc) return rc;
    DRONE_REQUIRE(res != nullptr, "drone_pr_step_local: bad arguments");
    OnDevice dev;
    if ((rc = dev.enter(prs[0]->device)) || (rc = prepare_parts(parts))) return rc;
    return step_parts(parts, is_peval != 0, res, (cudaStream_t)stream);
}

int drone_pr_job_local(int n_parts, drone_pr **prs, int max_steps, int *n_steps, int *sizes, void *stream) {
    std::vector<drone_pr *> parts;
    int rc = local_parts("drone_pr_job_local", n_parts, prs, &parts);
    if (rc) return rc;
    DRONE_REQUIRE(n_steps != nullptr && max_steps >= 1, "drone_pr_job_local: max_steps=%d, or a NULL step count", max_steps);
    OnDevice dev;
    if ((rc = dev.enter(prs[0]->device)) || (rc = prepare_parts(parts))) return rc;
    RunRequest rq;
    rq.job = true;
    std::vector<int> h((size_t)kHistorySteps * n_parts * 4);
    int total = 0;
    if (local_parts_run_separately(parts)) {
        std::vector<drone_pr_response> res((size_t)n_parts);
        for (bool sent = true; sent && total < max_steps; ++total) {
            if ((rc = step_parts(parts, total == 0, res.data(), (cudaStream_t)stream))) return rc;
            sent = false;
            for (int i = 0; i < n_parts; ++i) {
                const int four[4] = {res[i].Mirror2MasterSendSize, res[i].Mirror2MasterRecvSize, res[i].Master2MirrorSendSize,
                                     res[i].Master2MirrorRecvSize};
                for (int k = 0; k < 4; ++k) sent = sent || four[k] != 0;
                if (sizes) memcpy(sizes + ((size_t)total * n_parts + i) * 4, four, sizeof(four));
            }
        }
        *n_steps = total;
        return DRONE_OK;
    }
    for (RunControl c{}; !c.done && total < max_steps; total += c.steps) {
        rq.peval = total == 0;
        rq.max_steps = std::min(kHistorySteps, max_steps - total);
        if ((rc = run_local(parts, rq, (cudaStream_t)stream))) return rc;
        if ((rc = read_control(parts, rq.max_steps, &c, h.data(), (cudaStream_t)stream))) return rc;
        if (sizes) memcpy(sizes + (size_t)total * n_parts * 4, h.data(), sizeof(int) * 4 * (size_t)n_parts * c.steps);
    }
    *n_steps = total;
    return DRONE_OK;
}

static int run_power(std::vector<drone_pr *> &parts, int iterations, double damping, cudaStream_t st) {
    if (local_parts_run_separately(parts)) {
        LocalTransport copies;
        return parts[0]->dbl ? power_iterations<double>(parts, iterations, damping, copies, st)
                             : power_iterations<float>(parts, iterations, damping, copies, st);
    }
    RunRequest rq;
    rq.iterations = iterations;
    rq.damping = damping;
    return run_local(parts, rq, st);
}

int drone_pr_power_iterate(drone_pr *p, int iterations, double damping, void *stream) {
    DRONE_REQUIRE(p != nullptr, "drone_pr_power_iterate: handle is NULL");
    DRONE_REQUIRE(iterations >= 0 && damping >= 0 && damping <= 1, "drone_pr_power_iterate: iterations=%d damping=%g",
                  iterations, damping);
    DRONE_REQUIRE(p->xplan->nranks == 1 || p->comm, "drone_pr_power_iterate: %d ranks but no communicator",
                  p->xplan->nranks);
    std::vector<drone_pr *> parts{p};
    OnDevice dev;
    int rc = dev.enter(p->device);
    if (rc || (rc = prepare_parts(parts))) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (p->xplan->nranks == 1) return run_power(parts, iterations, damping, st);
    PeerTransport peer;
    NcclTransport nccl;
    NcclTransport &tr = use_peer_transport(p) ? peer : nccl;
    return p->dbl ? power_iterations<double>(parts, iterations, damping, tr, st)
                  : power_iterations<float>(parts, iterations, damping, tr, st);
}

int drone_pr_power_iterate_local(int n_parts, drone_pr **prs, int iterations, double damping, void *stream) {
    std::vector<drone_pr *> parts;
    int rc = local_parts("drone_pr_power_iterate_local", n_parts, prs, &parts);
    if (rc) return rc;
    DRONE_REQUIRE(iterations >= 0 && damping >= 0 && damping <= 1, "drone_pr_power_iterate_local: iterations=%d damping=%g",
                  iterations, damping);
    OnDevice dev;
    if ((rc = dev.enter(prs[0]->device)) || (rc = prepare_parts(parts))) return rc;
    return run_power(parts, iterations, damping, (cudaStream_t)stream);
}

int drone_pr_set_isolated_count(drone_pr *p, long long n_isolated) {
    DRONE_REQUIRE(p != nullptr && n_isolated >= 0, "drone_pr_set_isolated_count: bad argument");
    p->n_isolated = n_isolated;
    return DRONE_OK;
}

int drone_pr_device_arrays(drone_pr *p, void **d_pr, void **d_acc, void **d_diff, int **d_active,
                           int **d_update_by_message) {
    DRONE_REQUIRE(p != nullptr, "drone_pr_device_arrays: handle is NULL");
    if (d_pr) *d_pr = p->pr;
    if (d_acc) *d_acc = p->acc;
    if (d_diff) *d_diff = p->diff;
    if (d_active) *d_active = p->active;
    if (d_update_by_message) *d_update_by_message = p->ubm;
    return DRONE_OK;
}

int drone_pr_values(drone_pr *p, void *h_out, void *stream) {
    DRONE_REQUIRE(p && (h_out || p->n_local == 0), "drone_pr_values: NULL argument");
    if (p->n_local == 0) return DRONE_OK;
    unsigned unfinished = 0;
    DRONE_CUDA(cudaMemcpyAsync(h_out, p->pr, (p->dbl ? 8 : 4) * (size_t)p->n_local, cudaMemcpyDeviceToHost,
                               (cudaStream_t)stream));
    DRONE_CUDA(cudaMemcpyAsync(&unfinished, p->unfinished, sizeof(unsigned), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    DRONE_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    if (p->run != 0 && unfinished == p->run)
        return set_error(DRONE_E_STATE, "drone_pr_values: a wait between the blocks of the run that should have made the values ran out");
    return DRONE_OK;
}

}  // extern "C"
