// Power iterations of one part of many edges.
//
// The rows lie in the order of `place`, like the published values, and their edges as one stream of columns with the last edge
// of a row marked: a warp takes pieces of it, a lane 8 neighbouring edges of every 256, whatever rows they belong to, so
// that all of its gathers are in flight together (a chunk of a long row has 141 edges on average, and a short row's sum took
// a scan over 32 lanes for every 32 edges), and the vertex step reads and publishes in order.
//
// Bound: the LSU, one wavefront per gather that misses the table, and the lines of L1 that gathers in flight wait in: a table of 128 KB
// is the best on R-MAT-22 and within 3 % of the best elsewhere (64 / 96 / 128 / 160 KB, ms, float: R-MAT-22 3.31 / 3.36 / 2.94 / 2.98,
// R-MAT-18 0.324 / 0.312 / 0.316 / 0.316, a million vertices with 16 in-edges drawn uniformly 1.56 / 1.55 / 1.56 / 1.60, power law, 2.4
// M of 24 4.78 / 4.74 / 4.74 / 4.86; double 5.22 / 5.19 / 5.33 / 5.84, R-MAT-22 4.23 / 4.06 / 4.10 / 4.31).  ms for 20 iterations,
// chunks and scans / stream: R-MAT-18 float 0.54 / 0.32, double 0.60 / 0.39; R-MAT-20 1.20 / 0.72 and 1.55 / 1.02; R-MAT-22 float 5.03
// / 2.93.
#pragma once

namespace drone {

// 64 registers hold a tile of floats, not of doubles (R-MAT-22, float, 768 / 1024 threads: 3.28 / 3.02 ms; R-MAT-20, double:
// 1.09 / 1.45).
template <typename R> constexpr int stream_threads() { return sizeof(R) == 4 ? 1024 : 768; }
constexpr int kStreamTableBytes = 128 * 1024;

template <typename R>
struct StreamArgs {
    PartView<R> part;
    RowStream rows;
    const int *od;                // [n] out degree in stream order; -1: neither publishes nor counts as dangling
    R *sum, *tails;               // [n] sums of the rows with edges; [pieces] what a piece has of the row open at its end
    R *block_sums;
    RunControl *control;
    unsigned barrier_start, barrier_polls, run;
    R damping;
    int iterations;
    long long n_isolated;
};

// od[i] for the row at position i
__global__ void pr_stream_degrees_kernel(const int *__restrict__ row_of, const int *__restrict__ out_degree,
                                         const int *__restrict__ mirror2worker, int n, int *__restrict__ od) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int row = row_of[i], d = out_degree[row];
        od[i] = d == 0 && mirror2worker[row] != -1 ? -1 : d;
    }
}

template <typename R>
__device__ __forceinline__ R warp_sum(R v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sum[k] = what the in-edges of the k-th row with edges published, without what pieces before the one it ends in have of it:
// that is in their tails.
template <typename R>
__device__ __forceinline__ void stream_sums(const StreamArgs<R> &a, unsigned table, int warp, int n_warps) {
    const int lane = threadIdx.x & 31;
    const int n_pieces = a.rows.n_pieces, table_n = a.part.table_n;
    const R *push = a.part.push;
    R *sum = a.sum;
#pragma unroll 1
    for (int piece = warp; piece < n_pieces; piece += n_warps) {
        const int tile = a.rows.first_tile(piece);
        int tiles = a.rows.first_tile(piece + 1) - tile;
        const uint4 *at = reinterpret_cast<const uint4 *>(a.rows.col) + (long long)tile * (kTileEdges / 4) + lane * 2;
        uint4 c0 = __ldcs(at), c1 = __ldcs(at + 1);
        int base = __ldg(a.rows.first + piece);
        R carry = 0, open = 0;      // of the row open at the start of a tile: in every lane, and the lane's own share
#pragma unroll 1
        for (; tiles > 0; --tiles) {
            const unsigned c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
            at += kTileEdges / 4;
            if (tiles > 1) {
                c0 = __ldcs(at);
                c1 = __ldcs(at + 1);
            }
            R v[8];
            unsigned ends = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = published(table, table_n, push, (int)(c[j] & ~kRowEnd));
                ends |= (c[j] >> 31) << j;
            }
            if (!__any_sync(0xffffffffu, ends != 0)) {
#pragma unroll
                for (int j = 0; j < 8; ++j) open += v[j];
                continue;
            }
            carry += warp_sum(open);
            open = 0;
            // (sum since the last end, ends) of the lanes up to this one
            R tail = 0;
            int count = __popc(ends);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                tail += v[j];
                if (ends >> j & 1) tail = 0;
            }
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const R t = __shfl_up_sync(0xffffffffu, tail, d);
                const int k = __shfl_up_sync(0xffffffffu, count, d);
                if (lane >= d) {
                    if (count == 0) tail = t + tail;
                    count += k;
                }
            }
            R s = __shfl_up_sync(0xffffffffu, tail, 1);
            int before = __shfl_up_sync(0xffffffffu, count, 1);
            if (lane == 0) {
                s = 0;
                before = 0;
            }
            if (before == 0) s += carry;
            R *to = sum + base + before;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                s += v[j];
                if (ends >> j & 1) {
                    *to++ = s;
                    s = 0;
                }
            }
            base += __shfl_sync(0xffffffffu, count, 31);
            carry = __shfl_sync(0xffffffffu, tail, 31);
        }
        open = warp_sum(open);
        if (lane == 0) a.tails[piece] = carry + open;
    }
}

// d and what the pieces before its last one have of row i, for the lanes in `spanning`.  A row of few pieces is its lane's, the
// others are the warp's, one after the other.
template <typename R>
__device__ __forceinline__ R with_tails(const StreamArgs<R> &a, int i, unsigned spanning, R d) {
    const int lane = threadIdx.x & 31;
    int q0 = 0, q1 = 0;
    if (spanning >> lane & 1) {
        q0 = a.rows.piece_of(__ldg(a.rows.ptr + i));
        q1 = a.rows.piece_of(__ldg(a.rows.ptr + i + 1) - 1);
    }
    const bool many = q1 - q0 > 16;
    R before = 0;
    if (!many) {
#pragma unroll 4
        for (int q = q0; q < q1; ++q) before += a.tails[q];
    }
    for (unsigned left = __ballot_sync(0xffffffffu, many); left; left &= left - 1) {
        const int owner = __ffs(left) - 1, from = __shfl_sync(0xffffffffu, q0, owner), to = __shfl_sync(0xffffffffu, q1, owner);
        R sum = 0;
#pragma unroll 4
        for (int q = from + lane; q < to; q += 32) sum += a.tails[q];
        sum = warp_sum(sum);
        if (lane == owner) before = sum;
    }
    return spanning >> lane & 1 ? before + d : d;
}

// power_vertices in stream order.  LONG: some row reaches over more than kSerialPieces pieces, which one thread alone takes too long
// to add: us of 20 iterations, by a thread / by its warp, 65,536 vertices with one of 65,535 in-edges, 590,000 edges, float 339 / 212,
// double 399 / 256; 4.2 M vertices with two of as many in-edges 2055 / 1442 and 2723 / 1982.  Elsewhere the other form is the better one
// (R-MAT-18 to R-MAT-22, whose longest rows have 10 to 23 pieces, float 317 / 325, 732 / 743, 2930 / 2968).
constexpr int kSerialPieces = 32;
template <typename R, bool LONG>
__device__ __forceinline__ R stream_vertices(const StreamArgs<R> &a, R dang, bool last, int first, int stride) {
    const PartView<R> &p = a.part;
    const R base = ((R)1 - a.damping) / p.global_v, share = dang / p.global_v;
    R dangling = 0;
    const int lane = LONG ? (int)threadIdx.x & 31 : 0;      // whole warps, then
#pragma unroll 1
    for (int i0 = first; i0 - lane < p.n; i0 += kVertexBatch * stride) {
        int at[kVertexBatch], od[kVertexBatch];
        R d[kVertexBatch];
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) {
            const int i = i0 + b * stride;
            at[b] = i < p.n ? __ldg(a.rows.at + i) : -1;
            od[b] = i < p.n ? __ldg(a.od + i) : 1;
        }
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) d[b] = at[b] >= 0 ? a.sum[at[b] & ~kSpansPieces] : (R)0;
        if constexpr (LONG) {
            unsigned spans = 0;
#pragma unroll
            for (int b = 0; b < kVertexBatch; ++b) spans |= at[b] >= 0 && (at[b] & kSpansPieces) ? 1u << b : 0u;
            if (__any_sync(0xffffffffu, spans != 0)) {
#pragma unroll
                for (int b = 0; b < kVertexBatch; ++b) d[b] = with_tails(a, i0 + b * stride, __ballot_sync(0xffffffffu, spans >> b & 1), d[b]);
            }
        }
#pragma unroll
        for (int b = 0; b < kVertexBatch; ++b) {
            const int i = i0 + b * stride;
            if (i >= p.n) break;
            if (!LONG && at[b] >= 0 && (at[b] & kSpansPieces)) {
                const int q0 = a.rows.piece_of(__ldg(a.rows.ptr + i)), q1 = a.rows.piece_of(__ldg(a.rows.ptr + i + 1) - 1);
                R before = 0;
#pragma unroll 8
                for (int q = q0; q < q1; ++q) before += a.tails[q];
                d[b] = before + d[b];
            }
            const R now = base + a.damping * (d[b] + share);
            if (last) {
                const int row = __ldg(a.rows.row_of + i);
                p.pr[row] = now;
                p.diff[row] = d[b];
                continue;
            }
            if (od[b] == 0) dangling += now;
            p.push[i] = od[b] <= 0 ? not_pushed<R>() : now / od[b];
        }
    }
    return dangling;
}

template <typename R, bool LONG>
__global__ void __launch_bounds__(stream_threads<R>(), 1) pr_stream_kernel(const __grid_constant__ StreamArgs<R> a) {
    extern __shared__ __align__(16) char table_bytes[];
    R *table_ptr = reinterpret_cast<R *>(table_bytes);
    const unsigned table = (unsigned)__cvta_generic_to_shared(table_ptr);
    const PartView<R> &p = a.part;
    constexpr int THREADS = stream_threads<R>();
    const int first = blockIdx.x * THREADS + threadIdx.x, stride = gridDim.x * THREADS;
    // warps numbered across the blocks first: neighbours in the stream go to different SMs
    const int warp = (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x), n_warps = (int)(gridDim.x * (THREADS / 32));
    unsigned phase = a.barrier_start;
    R iso = (R)1 / (R)p.global_v, dangling = 0;
    for (int i = first; i < p.n; i += stride) {
        const int od = __ldg(a.od + i);
        p.pr[i] = iso;
        p.acc[i] = 0;
        p.diff[i] = 0;
        p.active[i] = 0;
        p.ubm[i] = 0;
        if (od == 0) dangling += iso;
        p.push[i] = od <= 0 ? not_pushed<R>() : iso / od;
    }
    for (int step = 0; step < a.iterations; ++step) {
        const R mine = block_sum<R>(dangling);
        if (threadIdx.x == 0) a.block_sums[blockIdx.x] = mine;
        if (!grid_barrier(&a.control->barrier, phase, a.barrier_polls)) break;
        load_table(p, table_ptr);
        const R dang = fold_blocks<R>(a.block_sums);      // its barrier also closes the table
        stream_sums(a, table, warp, n_warps);
        if (!grid_barrier(&a.control->barrier, phase, a.barrier_polls)) break;
        const R all = dang + (R)a.n_isolated * iso;
        const bool last = step + 1 == a.iterations;
        dangling = stream_vertices<R, LONG>(a, all, last, first, stride);
        iso = ((R)1 - a.damping) / p.global_v + a.damping * (all / p.global_v);
        if (last) return;
    }
    if (a.iterations == 0) return;
    // a wait ran out (give_up)
    if (threadIdx.x == 0) *p.unfinished = a.run;
    for (int i = first; i < p.n; i += stride) p.pr[i] = (R)NAN;
}

}  // namespace drone
