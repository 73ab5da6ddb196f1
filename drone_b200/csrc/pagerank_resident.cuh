// All supersteps in one launch, for graphs whose edges fit the shared memory of the GPU's SMs (about 4 million of them).
//
// The columns of the pull do not change from one superstep to the next, and neither does who owns which row: every block
// keeps a contiguous run of its part's rows in shared memory for the whole launch, with their columns, degrees, places and
// (in the job) state.  What a superstep reads from global memory is then only what the other blocks published.  Rows are
// whole inside a block, so that no partial sums travel between blocks, and the thread that owns a row goes on with it as soon
// as it is summed; the published values have two buffers, so that this needs no barrier of its own: one grid barrier a
// power iteration with a single part, two with several and in the job (pr_run_kernel: two and three).
//
// Bound: latency.  R-MAT-16, two parts, double, us an iteration: two barriers 1.7 and 1.3 (what the slowest block takes longer
// included), the table 1.4, the sums 2.7 (of these 1.7 are wavefronts of the LSU), the rows 1.5, the masters 1.3.  Whole runs
// against pr_run_kernel, us: power iterations, 20, R-MAT-12 two parts double 257 / 165, R-MAT-16 one part float 287 / 121, two
// parts double 402 / 229, eight parts float 490 / 321; the job, R-MAT-12 four parts 1416 / 817, R-MAT-16 four parts 2451 / 1142.
#pragma once

namespace drone {

constexpr int kSliceThreads = 512;
constexpr int kBlockSums = kReduceBlocks / 2;         // blocks of a launch at most: their sums of dangling mass have two buffers
constexpr int kRowWeight = 4;                        // what a row weighs beside its edges when rows are dealt to blocks (2: the same, 10: to 4 % slower)
constexpr int kPlaceMask = 0x3fffffff, kGotSome = 0x40000000, kToldMirrors = (int)0x80000000;   // job: a master's last exchange, on its place

// First row of block `index` of `blocks` (index == blocks: n): rowptr[r] + kRowWeight * r grows with every row.
__device__ __forceinline__ long long slice_target(const int *rowptr, int n, int index, int blocks) {
    const long long total = __ldg(rowptr + n) + (long long)kRowWeight * n;
    return (total * index + blocks - 1) / blocks;
}
__device__ __forceinline__ int slice_start(const int *rowptr, int n, int index, int blocks) {
    const long long target = slice_target(rowptr, n, index, blocks);
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if (__ldg(rowptr + mid) + (long long)kRowWeight * mid < target) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
// The same by one warp, 32 probes at a time: a chain of four loads instead of eighteen.
__device__ __forceinline__ int slice_start_warp(const int *rowptr, int n, int index, int blocks) {
    const long long target = slice_target(rowptr, n, index, blocks);
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32, at = lo + lane * step;
        const bool below = at < hi && __ldg(rowptr + at) + (long long)kRowWeight * at < target;
        const int count = __popc(__ballot_sync(0xffffffffu, below));
        if (count == 0) break;
        hi = min(lo + count * step, hi);
        lo += (count - 1) * step + 1;
    }
    return lo;
}

// most[b - 1] = {rows, edges} of the largest slices when the rows are dealt to b blocks.
__global__ void pr_slice_sizes_kernel(const int *__restrict__ rowptr, int n, int2 *most) {
    __shared__ int rows, edges;
    if (threadIdx.x == 0) rows = edges = 0;
    __syncthreads();
    const int blocks = (int)blockIdx.x + 1;
    for (int i = threadIdx.x; i < blocks; i += blockDim.x) {
        const int a = slice_start(rowptr, n, i, blocks), b = slice_start(rowptr, n, i + 1, blocks);
        atomicMax(&rows, b - a);
        atomicMax(&edges, __ldg(rowptr + b) - __ldg(rowptr + a));
    }
    __syncthreads();
    if (threadIdx.x == 0) most[blockIdx.x] = make_int2(rows, edges);
}

// A block's rows in shared memory, those with edges first (in order), then those without.
struct SliceRoom {
    int table, rows, edges;      // capacities: values, rows, edges
};
template <typename R>
struct Slice {
    R *table, *sum;              // published values; sum of a row's edges, -0.0 where none of them was pushed
    R *acc, *pr, *total;         // job: state after the superstep before, and what the last one added
    int *row, *od, *place;       // row: a master's number in the list of masters; od: 0 dangling, -1 neither pushes nor counts
    int *order;                  // several parts: the rows by kind, masters, mirrors, those that no other part holds
    unsigned *col;
    int n_rows, n_edges, n_masters, n_mirrors;
};
inline size_t slice_row_bytes(size_t value, bool job, bool several) { return value * (job ? 4 : 1) + sizeof(int) * (several ? 4 : 3); }

template <typename R, bool JOB>
__device__ __forceinline__ Slice<R> place_slice(char *at, const SliceRoom &room, bool several) {
    Slice<R> s;
    s.table = reinterpret_cast<R *>(at);
    s.sum = s.table + room.table;
    s.acc = s.sum + room.rows;
    s.pr = s.acc + (JOB ? room.rows : 0);
    s.total = s.pr + (JOB ? room.rows : 0);
    s.row = reinterpret_cast<int *>(s.total + (JOB ? room.rows : 0));
    s.od = s.row + room.rows;
    s.place = s.od + room.rows;
    s.order = s.place + room.rows;
    s.col = reinterpret_cast<unsigned *>(s.order + (several ? room.rows : 0));
    return s;
}

// Exclusive sum of v over the block's threads.  `warps`: 32 words of shared memory, free again when the call returns.
__device__ __forceinline__ int block_exclusive_sum(int v, int *warps, int *total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int upto = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += t;
    }
    if (lane == 31) warps[w] = upto;
    __syncthreads();
    int before = 0, all = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
        if (i < w) before += warps[i];
        all += warps[i];
    }
    __syncthreads();
    *total = all;
    return before + upto - v;
}

// Fills the slice with rows [r0, r1) of the part; returns the row (place in the slice) in which this thread's edges start.
template <typename R, bool JOB, int THREADS>
__device__ int fill_slice(Slice<R> &s, const PartView<R> &p, int r0, int r1, bool several, int *warps) {
    const int tid = threadIdx.x;
    const int e0 = __ldg(p.rowptr + r0);
    s.n_rows = r1 - r0;
    s.n_edges = __ldg(p.rowptr + r1) - e0;
    for (int e = tid; e < s.n_edges; e += THREADS) s.col[e] = (unsigned)__ldcs(p.col + e0 + e);
    const int per = (s.n_rows + THREADS - 1) / THREADS, first = min(tid * per, s.n_rows), end = min(first + per, s.n_rows);
    int filled = 0, kinds = 0, all_filled, all_kinds = 0;       // kinds: masters, and mirrors in the upper half
    for (int i = first; i < end; ++i) {
        filled += __ldg(p.rowptr + r0 + i + 1) > __ldg(p.rowptr + r0 + i);
        const int role = several ? __ldg(p.role + r0 + i) : kOwnRow;
        kinds += role >= 0 ? 1 : role == kMirrorRow ? 0x10000 : 0;
    }
    int at = block_exclusive_sum(filled, warps, &all_filled);      // its barriers also order the columns before the flags
    int at_empty = all_filled + first - at;
    if (several) kinds = block_exclusive_sum(kinds, warps, &all_kinds);
    s.n_masters = all_kinds & 0xffff;
    s.n_mirrors = all_kinds >> 16;
    int at_master = kinds & 0xffff, at_mirror = s.n_masters + (kinds >> 16);
    int at_own = s.n_masters + s.n_mirrors + first - (kinds & 0xffff) - (kinds >> 16);
    for (int i = first; i < end; ++i) {
        const int row = r0 + i, b = __ldg(p.rowptr + row), e = __ldg(p.rowptr + row + 1);
        const int to = e > b ? at++ : at_empty++;
        if (e > b) s.col[e - 1 - e0] |= kRowEnd;
        const int od = __ldg(p.out_degree + row);
        s.od[to] = od == 0 && __ldg(p.mirror2worker + row) != -1 ? -1 : od;
        s.place[to] = p.place ? __ldg(p.place + row) : row;
        const int role = several ? __ldg(p.role + row) : kOwnRow;
        s.row[to] = role >= 0 ? role : row;
        if (several) s.order[role >= 0 ? at_master++ : role == kMirrorRow ? at_mirror++ : at_own++] = to;
        s.sum[to] = not_pushed<R>();
        if (JOB) s.total[to] = 0;
    }
    __syncthreads();
    const int share = ((s.n_edges + THREADS - 1) / THREADS) | 1;
    int ends = 0, unused;
    for (int e = min(tid * share, s.n_edges); e < min((tid + 1) * share, s.n_edges); ++e) ends += s.col[e] >> 31;
    return block_exclusive_sum(ends, warps, &unused);
}

// load_table with eight loads in flight, the last ones as well: with small tables a round trip to L2 is most of its time.
template <typename R>
__device__ __forceinline__ void load_slice_table(const R *push, int table_n, R *table) {
    constexpr int W = 16 / sizeof(R), DEPTH = 8;
    const int n4 = table_n / W;
    const float4 *src = reinterpret_cast<const float4 *>(push);
    float4 *dst = reinterpret_cast<float4 *>(table);
#pragma unroll 1
    for (int i = threadIdx.x; i < n4; i += DEPTH * kSliceThreads) {
        float4 v[DEPTH];
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) v[u] = src[min(i + u * kSliceThreads, n4 - 1)];      // beyond the end: its last vector
#pragma unroll
        for (int u = 0; u < DEPTH; ++u)
            if (i + u * kSliceThreads < n4) dst[i + u * kSliceThreads] = v[u];
    }
    for (int i = n4 * W + threadIdx.x; i < table_n; i += kSliceThreads) table[i] = push[i];
}

// sum[i] = what the in-edges of row i published.  Every thread adds an equal run of edges (an odd number, so that the
// threads' columns lie in different banks); what it has of rows that other threads finish is handed on by a segmented scan.
// Ends with the block's threads together.
template <typename R, int UN>
__device__ __forceinline__ void slice_sums(const Slice<R> &s, const R *push, int table_n, int first_row, R *tails, int *closes) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned table = (unsigned)__cvta_generic_to_shared(s.table);
    const int share = ((s.n_edges + (int)blockDim.x - 1) / (int)blockDim.x) | 1;
    const int begin = min((int)threadIdx.x * share, s.n_edges), end = min(begin + share, s.n_edges);
    R acc = not_pushed<R>();
    int at = first_row;
#pragma unroll 1
    for (int e = begin; e < end; e += UN) {
        unsigned c[UN];
        R v[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) c[u] = e + u < end ? s.col[e + u] : 0u;
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            v[u] = published(table, table_n, push, (int)(c[u] & ~kRowEnd));
            if (e + u >= end) v[u] = not_pushed<R>();
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            acc += v[u];
            if (c[u] & kRowEnd) {
                s.sum[at++] = acc;
                acc = not_pushed<R>();
            }
        }
    }
    // (tail, closed a row) of the threads up to this one, a closed row starting the sum anew
    R upto = acc;
    int closed = at > first_row;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const R t = __shfl_up_sync(0xffffffffu, upto, d);
        const int c = __shfl_up_sync(0xffffffffu, closed, d);
        if (lane >= d) {
            if (!closed) upto = t + upto;
            closed |= c;
        }
    }
    if (lane == 31) {
        tails[w] = upto;
        closes[w] = closed;
    }
    R before = __shfl_up_sync(0xffffffffu, upto, 1);
    int before_closed = __shfl_up_sync(0xffffffffu, closed, 1);
    if (lane == 0) {
        before = not_pushed<R>();
        before_closed = 0;
    }
    __syncthreads();
    const unsigned closed_warps = __ballot_sync(0xffffffffu, lane < w && closes[lane]);
    if (!before_closed) {
        R carry = not_pushed<R>();      // the warps since the last one that closed a row
        for (int i = closed_warps ? 31 - __clz(closed_warps) : 0; i < w; ++i) carry += tails[i];
        before = carry + before;
    }
    if (at > first_row) s.sum[first_row] = before + s.sum[first_row];      // only the thread that closed the row touches its sum
    __syncthreads();
}

// A master row's mirrors: the first four {part, row} and {place, out degree}, part -1 for none.
struct Mirrors {
    int k0, k1;
    int2 at[4], target[4];
};
template <typename R>
__device__ __forceinline__ Mirrors mirrors_of(const PartView<R> &p, int master) {
    Mirrors m;
    m.k0 = __ldg(p.m_off + master);
    m.k1 = __ldg(p.m_off + master + 1);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        m.at[u] = m.k0 + u < m.k1 ? __ldg(p.pairs + m.k0 + u) : make_int2(-1, 0);
        m.target[u] = m.k0 + u < m.k1 ? __ldg(p.targets + m.k0 + u) : make_int2(0, 0);
    }
    return m;
}

// Calls visit(part, row, place, out degree) for every mirror, in ascending rank order.
template <typename R, typename Visit>
__device__ __forceinline__ void for_each_mirror(const PartView<R> &p, const Mirrors &m, Visit visit) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (m.at[u].x >= 0) visit(m.at[u].x, m.at[u].y, m.target[u].x, m.target[u].y);
#pragma unroll 1
    for (int k = m.k0 + 4; k < m.k1; ++k) {
        const int2 at = __ldg(p.pairs + k), target = __ldg(p.targets + k);
        visit(at.x, at.y, target.x, target.y);
    }
}

// One step of a row of the job: pr_process_messages and pr_increment (increment_vertices), on state in shared memory.
template <typename R>
__device__ __forceinline__ bool next_value(R acc, R gacc, R old, R eps, R *now) {
    const R alpha = (R)0.85f;
    *now = fma_r<R>(alpha, acc + gacc, (R)1 - alpha);
    R d = *now - old;
    if (d < 0) d = -d;
    return !(d < eps);
}

template <typename R, int MAXP, bool JOB>
__global__ void __launch_bounds__(kSliceThreads, 1)
pr_resident_kernel(const __grid_constant__ RunArgs<R, MAXP> a, const SliceRoom room) {
    extern __shared__ __align__(16) char room_bytes[];
    __shared__ PartView<R> p;
    __shared__ PartArrays<R, MAXP> of;
    __shared__ R *push2_of[MAXP];
    __shared__ int counts[MAXP * 4];
    __shared__ R tails[32], folded[32];
    __shared__ int closes[32];
    __shared__ int me_shared, bounds[2];
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) {
        int q = 0;
        while (q + 1 < a.n_parts && (int)blockIdx.x >= a.first_block[q + 1]) ++q;
        me_shared = q;
        p = a.part[q];
    }
    for (int q = tid; q < a.n_parts; q += kSliceThreads) {
        of.diff[q] = a.part[q].diff;
        of.push[q] = a.part[q].push;
        push2_of[q] = a.part[q].push2;
        of.pr[q] = a.part[q].pr;
        of.acc[q] = a.part[q].acc;
        of.ubm[q] = a.part[q].ubm;
    }
    if (blockIdx.x == 0 && tid == 0) a.control->t_start = now_ns();
    __syncthreads();
    const int me = me_shared;
    const int block = (int)blockIdx.x - a.first_block[me], blocks = a.first_block[me + 1] - a.first_block[me];
    const int first = block * kSliceThreads + tid, stride = blocks * kSliceThreads;
    const bool several = MAXP > 1 && a.n_parts > 1;
    unsigned phase = a.barrier_start;

    if (tid < 64) {
        const int r = slice_start_warp(p.rowptr, p.n, block + (tid >> 5), blocks);
        if (lane == 0) bounds[tid >> 5] = r;
    }
    R gdiff = 0, gacc = 0, iso = 0, dangling = 0;
    if (JOB) {
        if (a.peval) {
            dangling = init_vertices(p, (R)1, false, first, stride);
        } else {
            gdiff = p.scalars[0];
            gacc = p.scalars[1] + gdiff;
            dangling = increment_vertices(p, a.eps, gacc, first, stride);
        }
    } else {
        iso = (R)1 / (R)p.global_v;
        dangling = init_vertices(p, iso, true, first, stride);
    }
    __syncthreads();
    Slice<R> s = place_slice<R, JOB>(room_bytes, room, several);
    const int first_row = fill_slice<R, JOB, kSliceThreads>(s, p, bounds[0], bounds[1], several, closes);
    Mirrors kept;      // those of this thread's first master row stay in registers
    if (tid < s.n_masters) kept = mirrors_of(p, s.row[s.order[tid]]);

    const int n_steps = JOB ? a.max_steps : a.iterations;
    bool done = false;
    int step = 0;
    for (;; ++step) {
        for (int o = 16; o > 0; o >>= 1) dangling += __shfl_down_sync(0xffffffffu, dangling, o);
        if (lane == 0) tails[tid >> 5] = dangling;
        __syncthreads();
        if (tid == 0) {
            R sum = 0;
#pragma unroll
            for (int i = 0; i < kSliceThreads / 32; ++i) sum += tails[i];
            a.block_sums[(step & 1) * kBlockSums + blockIdx.x] = sum;      // blocks may still read the step's before
            if (JOB || step < n_steps) grid_arrive(&a.control->barrier);
        }
        if (!JOB && step == n_steps) break;      // nobody looks at what follows the last iteration
        if (!grid_wait(&a.control->barrier, phase, a.barrier_polls)) return give_up(a, p.pr, p.n, first, stride);
        int sent = 0;      // in the superstep before; every block looks at the counts of all parts
        if (JOB && several && step > 0)
            for (int q = tid; q < a.n_parts * 4; q += kSliceThreads) sent |= __ldcg(a.history + (long long)(step - 1) * a.n_parts * 4 + q);
        // what the blocks met of dangling vertices (fixed tree order), and the table
        const R *push = step & 1 ? p.push2 : p.push;
        R part_sum = 0;
        for (int i = tid; i < (int)gridDim.x; i += kSliceThreads) part_sum += __ldcg(a.block_sums + (step & 1) * kBlockSums + i);
        load_slice_table(push, p.table_n, s.table);
        for (int o = 16; o > 0; o >>= 1) part_sum += __shfl_down_sync(0xffffffffu, part_sum, o);
        if (lane == 0) folded[tid >> 5] = part_sum;
        if (JOB && several)
            for (int q = tid; q < a.n_parts * 4; q += kSliceThreads) counts[q] = 0;
        if (JOB && step == 0)
            for (int j = tid; j < s.n_rows; j += kSliceThreads) {
                const int i = several ? s.order[j] : j, row = j < s.n_masters ? __ldg(p.m_rows + s.row[i]) : s.row[i];
                s.acc[i] = p.acc[row];
                s.pr[i] = p.pr[row];
            }
        const bool exchanged = __syncthreads_or(sent) != 0;
        if (JOB && step > 0) {
            done = !exchanged;
            if (done || step == n_steps) break;
            gacc += gdiff;
        }
        R dang = 0;
#pragma unroll
        for (int i = 0; i < kSliceThreads / 32; ++i) dang += folded[i];
        slice_sums<R, 8>(s, push, p.table_n, first_row, tails, closes);
        if (JOB) gdiff = dang;
        dangling = 0;
        R *publish = step & 1 ? p.push : p.push2;
        R *const *publish_of = step & 1 ? of.push : push2_of;
        const R all = dang + (R)a.n_isolated * iso;
        const R base = ((R)1 - a.damping) / p.global_v, share = all / p.global_v;
        const bool last = step + 1 == n_steps;
        const R gacc_next = gacc + gdiff;

        // a row's own step: the value before the last superstep's sum (commit), then what it publishes after this one's
        auto commit = [&](int i) {
            if (step == 0) return;
            const R acc = s.acc[i] + s.total[i];
            R now;
            if (next_value<R>(acc, gacc, s.pr[i], a.eps, &now)) s.pr[i] = now;
            s.acc[i] = acc;
        };
        auto delta_of = [&](int i, R total, R *moved_by) {      // whether the row will push, and how far it moves
            s.total[i] = total;
            R now;
            const bool push_it = next_value<R>(s.acc[i] + total, gacc_next, s.pr[i], a.eps, &now);
            *moved_by = now - s.pr[i];
            return push_it;
        };
        if (several) {
            for (int j = s.n_masters + tid; j < s.n_masters + s.n_mirrors; j += kSliceThreads) {
                const int i = s.order[j];
                p.diff[s.row[i]] = JOB ? s.sum[i] : (R)0 + s.sum[i];      // its master takes it from there
            }
            __syncthreads();
            if (tid == 0) grid_arrive(&a.control->barrier);
        }
        // rows that no other part holds go on while the blocks arrive
        for (int j = s.n_masters + s.n_mirrors + tid; j < s.n_rows; j += kSliceThreads) {
            const int i = several ? s.order[j] : j, od = s.od[i];
            const R d = (R)0 + s.sum[i];
            if (JOB) {
                commit(i);
                R by;
                R out = not_pushed<R>();
                if (delta_of(i, d, &by)) {
                    if (od == 0) dangling += by / p.global_v;
                    else if (od > 0) out = by / od;
                }
                publish[s.place[i]] = out;
            } else {
                const R now = base + a.damping * (d + share);
                if (last) {
                    p.pr[s.row[i]] = now;
                    p.diff[s.row[i]] = d;
                } else {
                    if (od == 0) dangling += now;
                    publish[s.place[i]] = od <= 0 ? not_pushed<R>() : now / od;
                }
            }
        }
        if (several && !grid_wait(&a.control->barrier, phase, a.barrier_polls)) return give_up(a, p.pr, p.n, first, stride);
        if (JOB && step == 0 && blockIdx.x == 0 && tid == 0) a.control->t_pull = now_ns();
        if (several) {
            // a master takes what its mirrors hold, in ascending rank order (Mirror2MasterSend, pr.cu:215-297), and hands the
            // total back (Master2MirrorSend, :299-373): here it takes the mirrors' next step with its own, since all replicas of
            // a vertex have the same state.  Only flagged entries travel in the job, and they are counted.
            unsigned moved[MAXP <= 8 ? MAXP : 1] = {0};
#pragma unroll 1
            for (int j = tid; j < s.n_masters; j += kSliceThreads) {
                const int i = s.order[j];
                const Mirrors m = j == tid ? kept : mirrors_of(p, s.row[i]);
                const int od = s.od[i];
                R d = (R)0 + s.sum[i];
                R v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = m.at[u].x >= 0 ? of.diff[m.at[u].x][m.at[u].y] : not_pushed<R>();
                if (JOB) {
                    commit(i);
                    int got = 0;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (!is_pushed(v[u])) continue;
                        d += v[u];
                        ++got;
                        note_moved<MAXP>(moved, counts, m.at[u].x, 0);
                    }
#pragma unroll 1
                    for (int k = m.k0 + 4; k < m.k1; ++k) {
                        const int2 at = __ldg(p.pairs + k);
                        const R more = of.diff[at.x][at.y];
                        if (!is_pushed(more)) continue;
                        d += more;
                        ++got;
                        note_moved<MAXP>(moved, counts, at.x, 0);
                    }
                    const bool tell = got > 0 || is_pushed(s.sum[i]);
                    s.place[i] = (s.place[i] & kPlaceMask) | (got > 0 ? kGotSome : 0) | (tell ? kToldMirrors : 0);
                    if (MAXP > 8) {
                        if (got) atomicAdd(&counts[4 * me + 1], got);
                        if (tell) atomicAdd(&counts[4 * me + 2], m.k1 - m.k0);
                    }
                    R by;
                    const bool push_it = delta_of(i, d, &by);
                    if (push_it && od == 0) dangling += by / p.global_v;
                    const R out = push_it && od > 0 ? by / od : not_pushed<R>();
                    publish[s.place[i] & kPlaceMask] = out;
                    for_each_mirror(p, m, [&](int q, int, int place, int degree) {
                        if (tell) note_moved<MAXP>(moved, counts, q, 3);
                        publish_of[q][place] = degree == od ? out : push_it && degree != 0 ? by / degree : not_pushed<R>();
                    });
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (m.at[u].x >= 0) d += v[u];
#pragma unroll 1
                    for (int k = m.k0 + 4; k < m.k1; ++k) {
                        const int2 at = __ldg(p.pairs + k);
                        d += of.diff[at.x][at.y];
                    }
                    const R now = base + a.damping * (d + share);
                    const R out = od <= 0 ? not_pushed<R>() : now / od;
                    if (last) {
                        const int row = __ldg(p.m_rows + s.row[i]);
                        p.pr[row] = now;
                        p.diff[row] = (R)0 + s.sum[i];
                    } else {
                        publish[s.place[i]] = out;
                        if (od == 0) dangling += now;
                    }
                    for_each_mirror(p, m, [&](int q, int row, int place, int degree) {
                        if (last) of.pr[q][row] = now;
                        else publish_of[q][place] = degree == od ? out : degree == 0 ? not_pushed<R>() : now / degree;
                    });
                }
            }
            if (JOB) {
                if (MAXP <= 8) {      // what came up to this part's masters went down to them as counted here
                    int up = 0, down = 0;
#pragma unroll
                    for (int q = 0; q < (MAXP <= 8 ? MAXP : 1); ++q) {
                        if (q >= a.n_parts) break;
                        const unsigned both = __reduce_add_sync(0xffffffffu, moved[q]);      // few rows a thread: 16 bits hold either
                        if (lane == q) {
                            up = (int)(both & 0xffffu);
                            down = (int)(both >> 16);
                        }
                    }
                    if (up) {
                        atomicAdd(&counts[4 * lane], up);
                        atomicAdd(&counts[4 * me + 1], up);
                    }
                    if (down) {
                        atomicAdd(&counts[4 * lane + 3], down);
                        atomicAdd(&counts[4 * me + 2], down);
                    }
                }
                __syncthreads();
                int *h = a.history + (long long)step * a.n_parts * 4;
                for (int q = tid; q < a.n_parts * 4; q += kSliceThreads)
                    if (counts[q]) atomicAdd(h + q, counts[q]);
            }
        }
        iso = ((R)1 - a.damping) / p.global_v + a.damping * (all / p.global_v);
    }
    if (JOB) {      // the state after the last superstep, for whoever continues or looks
        if (block == 0 && tid == 0) {
            p.scalars[0] = gdiff;
            p.scalars[1] = gacc;
        }
        if (blockIdx.x == 0 && tid == 0) {
            a.control->steps = step;
            a.control->done = done ? 1 : 0;
        }
        int seen = 0;
        for (int j = tid; j < s.n_rows; j += kSliceThreads) {
            const int i = several ? s.order[j] : j, row = j < s.n_masters ? __ldg(p.m_rows + s.row[i]) : s.row[i];
            const bool pushed = is_pushed(s.sum[i]);
            seen += pushed;
            p.active[row] = pushed ? 1 : 0;
            if (j >= s.n_masters && j < s.n_masters + s.n_mirrors) continue;      // the rest of a mirror's state is its master's
            const R acc = s.acc[i], pr = s.pr[i], total = s.total[i];
            p.acc[row] = acc;
            p.pr[row] = pr;
            p.diff[row] = total;
            const int flags = j < s.n_masters ? s.place[i] : 0;
            p.ubm[row] = (flags & kGotSome) ? 1 : 0;
            if (j >= s.n_masters) continue;
            for_each_mirror(p, mirrors_of(p, s.row[i]), [&](int q, int at, int, int) {
                of.acc[q][at] = acc;
                of.pr[q][at] = pr;
                of.diff[q][at] = total;
                of.ubm[q][at] = (flags & kToldMirrors) ? 1 : 0;
            });
        }
        if (a.count_visited) {
            seen = __reduce_add_sync(0xffffffffu, seen);
            if (lane == 0 && seen) atomicAdd(&a.control->visited[me], seen);
        }
    }
    if (blockIdx.x == 0 && tid == 0) a.control->t_end = now_ns();
}

}  // namespace drone
