// Sparse aggregation kernels:  Y[r,:] = sum_k val[k] * X[col[k],:]  over CSR rows.
//
// The work of one call is split three ways, all decided when the plan was built:
//   1. short rows (at most short_row_limit nonzeros) are stored once more as one
//      contiguous stream with end-of-row flags; a lane group walks about 64
//      entries of it (whole rows), adding a row's nonzeros in CSR order into one
//      accumulator and writing the row at its last entry, so the per-row cost
//      is one store and no warp is spent on a row of two nonzeros;
//   2. long rows: cut into chunks of chunk_nnz nonzeros, one warp per chunk with
//      its 32/G lane groups taking interleaved nonzeros; a row that is a single
//      chunk is written directly, otherwise the chunk sum goes to a partial slot.
//      The warps of a resident grid take the chunks from a shared counter, four
//      at a time, so that no warp idles while another still has a queue;
//   3. split rows: the partial slots of a row are added in slot order.
// A lane group is G lanes that together hold one dense row: each lane owns VPL
// vectors of VEC floats (float4 when the operands allow 16-byte accesses).
// No atomics touch the data, so the summation order is fixed by the plan and two
// calls give the same bits whichever warp happens to take which chunk.
//
// Template switches shared by the kernels:
//   UNIT  every stored coefficient counts as 1 (the val stream is not read);
//   HOT   columns carry a tag: a tagged column is a position in the plan's table of
//         hot rows (a compact copy of the most often gathered rows of X, small
//         enough to stay in L2 when X itself is many times larger than L2).
//
// The CSR streams (col, val) and the output are touched once and use streaming
// cache hints so that L2 capacity is left to the gathered rows of X.
//
// This header is compiled into several translation units, one per combination of
// the switches, so that they build side by side.
#pragma once

#include "plan.cuh"

namespace drone {

// L2 cache policies.  Rows of X are gathered many times and should stay resident; the CSR
// streams, the chunk list and the output pass through once and should be the first to go.
__device__ __forceinline__ unsigned long long l2_policy_keep() {
    unsigned long long p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ unsigned long long l2_policy_stream() {
    unsigned long long p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ float4 ld_keep(const float4 *ptr, unsigned long long pol) {
    float4 v;
    asm("ld.global.nc.L2::cache_hint.v4.f32 {%0,%1,%2,%3}, [%4], %5;"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(ptr), "l"(pol));
    return v;
}
__device__ __forceinline__ float ld_keep(const float *ptr, unsigned long long pol) {
    float v;
    asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(ptr), "l"(pol));
    return v;
}
// The same through the coherent path, for kernels that start before the one that writes X has finished (EARLY below).
__device__ __forceinline__ float4 ld_coherent(const float4 *ptr, unsigned long long pol) {
    float4 v;
    asm volatile("ld.global.L2::cache_hint.v4.f32 {%0,%1,%2,%3}, [%4], %5;"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(ptr), "l"(pol));
    return v;
}
__device__ __forceinline__ float ld_coherent(const float *ptr, unsigned long long pol) {
    float v;
    asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(ptr), "l"(pol));
    return v;
}
// A gathered vector, or zeros where `live` is false.  The load is predicated inside one volatile statement: written as a
// conditional expression it became a branch, which the compiler moved down to the multiply-add that uses the value, so
// that the loads of a batch followed one another instead of being in flight together (R-MAT-16, F = 160: 597 us a call,
// against 333 at F = 256, where no lane's vectors run past the row and the loads need no condition).
template <bool EARLY>
__device__ __forceinline__ float4 ld_gathered_if(const float4 *ptr, unsigned long long pol, bool live) {
    float4 v;
    if (EARLY)
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %6, 0;\n\t"
                     "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                     "@q ld.global.L2::cache_hint.v4.f32 {%0,%1,%2,%3}, [%4], %5;\n\t}"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(ptr), "l"(pol), "r"((int)live));
    else
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %6, 0;\n\t"
                     "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                     "@q ld.global.nc.L2::cache_hint.v4.f32 {%0,%1,%2,%3}, [%4], %5;\n\t}"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(ptr), "l"(pol), "r"((int)live));
    return v;
}
template <bool EARLY>
__device__ __forceinline__ float ld_gathered_if(const float *ptr, unsigned long long pol, bool live) {
    float v;
    if (EARLY)
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.b32 %0, 0;\n\t"
                     "@q ld.global.L2::cache_hint.f32 %0, [%1], %2;\n\t}"
                     : "=f"(v) : "l"(ptr), "l"(pol), "r"((int)live));
    else
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.b32 %0, 0;\n\t"
                     "@q ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;\n\t}"
                     : "=f"(v) : "l"(ptr), "l"(pol), "r"((int)live));
    return v;
}
template <bool EARLY, typename T>
__device__ __forceinline__ T ld_gathered(const T *ptr, unsigned long long pol) {
    return EARLY ? ld_coherent(ptr, pol) : ld_keep(ptr, pol);
}
__device__ __forceinline__ int ld_stream(const int *ptr, unsigned long long pol) {
    int v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(ptr), "l"(pol));
    return v;
}
__device__ __forceinline__ float ld_stream(const float *ptr, unsigned long long pol) {
    float v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(ptr), "l"(pol));
    return v;
}
__device__ __forceinline__ void st_stream(float4 *ptr, const float4 &v, unsigned long long pol) {
    asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1,%2,%3,%4}, %5;"
                 :: "l"(ptr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "l"(pol) : "memory");
}
__device__ __forceinline__ void st_stream(float *ptr, const float &v, unsigned long long pol) {
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" :: "l"(ptr), "f"(v), "l"(pol) : "memory");
}

template <int VEC> struct Vec;
template <> struct Vec<4> {
    using type = float4;
    static __device__ __forceinline__ float4 zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
    static __device__ __forceinline__ void fma(float4 &a, float v, const float4 &x) {
        a.x = fmaf(v, x.x, a.x);
        a.y = fmaf(v, x.y, a.y);
        a.z = fmaf(v, x.z, a.z);
        a.w = fmaf(v, x.w, a.w);
    }
    static __device__ __forceinline__ void add(float4 &a, const float4 &x) {
        a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
    }
    static __device__ __forceinline__ float4 shfl_xor(const float4 &a, int o) {
        return make_float4(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o),
                           __shfl_xor_sync(0xffffffffu, a.z, o), __shfl_xor_sync(0xffffffffu, a.w, o));
    }
    static __device__ __forceinline__ float4 finish(const float4 &a, float scale, int relu) {
        float4 r = make_float4(a.x * scale, a.y * scale, a.z * scale, a.w * scale);
        if (relu) { r.x = fmaxf(r.x, 0.f); r.y = fmaxf(r.y, 0.f); r.z = fmaxf(r.z, 0.f); r.w = fmaxf(r.w, 0.f); }
        return r;
    }
};
template <> struct Vec<1> {
    using type = float;
    static __device__ __forceinline__ float zero() { return 0.f; }
    static __device__ __forceinline__ void fma(float &a, float v, const float &x) { a = fmaf(v, x, a); }
    static __device__ __forceinline__ void add(float &a, const float &x) { a += x; }
    static __device__ __forceinline__ float shfl_xor(const float &a, int o) {
        return __shfl_xor_sync(0xffffffffu, a, o);
    }
    static __device__ __forceinline__ float finish(const float &a, float scale, int relu) {
        const float r = a * scale;
        return relu ? fmaxf(r, 0.f) : r;
    }
};

// Of a lane's VPL vectors, how many lie inside the row at every width that the shape is used for (dispatch_floats: a shape
// of 32 x VPL single floats starts where the next smaller one ends).  Their loads need no test against the width (us with a
// test per vector / without, power law: 90,000 rows of 41, F = 131 268 / 248, F = 401 868 / 730; 250,000 rows of 7, F = 95
// 155 / 128).  Above 512 floats half of the tests stay, and without the other half F = 601 was slower: 60,000 rows of 13,
// 419 / 463.
constexpr int sure_vectors(int G, int VPL, int VEC) {
    if (VEC != 1 || G != 32) return 0;
    return VPL == 4 ? 2 : VPL == 8 ? 4 : VPL == 12 ? 8 : VPL == 16 ? 12 : 0;
}

// The condition of a lane's vector p of a row.  BRANCH: lanes with many single floats of a row (odd widths above 128) in the
// short-row kernel, and above 512 everywhere, are bound by instructions, and nearly all of their loads are live: a branch
// costs them less than the zeroing of the predicated form.
template <bool BRANCH, int VEC, bool EARLY>
__device__ __forceinline__ typename Vec<VEC>::type ld_row_if(const typename Vec<VEC>::type *ptr, unsigned long long pol, bool live) {
    if (BRANCH) return live ? ld_gathered<EARLY>(ptr, pol) : Vec<VEC>::zero();
    return ld_gathered_if<EARLY>(ptr, pol, live);
}

template <int A, int B> struct MinOf { static constexpr int value = A < B ? A : B; };

// What happens to a finished row before it is stored: Y[r,:] = act(row_scale[r] * sum).  Without a scale array the
// multiplication is skipped, so the plain call stores exactly the sum.
struct Epilogue {
    const float *row_scale = nullptr;   // [n_rows] or NULL
    int relu = 0;                       // 1: negative results are stored as 0
    // Routed rows (the aggregation that also performs the upward half of the mirror/master exchange): route[r] =
    // {peer, row in that peer's receive area} for a row whose total another GPU forms, {-1, ..} otherwise.  A routed
    // row is stored into the peer's memory (rows of route_nvec vectors there; this call writes vectors route_col0 ..)
    // and not into Y.
    const int2 *route = nullptr;        // [n_rows] or NULL
    float *const *peer_rows = nullptr;  // [peers] base of every peer's receive area
    int route_nvec = 0, route_col0 = 0;
};

template <int VEC>
__device__ __forceinline__ typename Vec<VEC>::type finish_row(const typename Vec<VEC>::type &acc, const Epilogue &e,
                                                              float scale) {
    if (e.row_scale == nullptr && !e.relu) return acc;
    return Vec<VEC>::finish(acc, scale, e.relu);
}

// Where a finished row goes: its row of Y, or its place in the owner's receive area (remote: the caller uses a plain
// store, no cache policy of this GPU's L2 on a peer's address).
template <int VEC>
struct RowDestination {
    typename Vec<VEC>::type *ptr;
    bool remote;
};

template <int VEC>
__device__ __forceinline__ RowDestination<VEC> row_destination(const Epilogue &e, float *Y, long long ldy, int row) {
    using V = typename Vec<VEC>::type;
    if (e.route != nullptr) {
        const int2 r = __ldg(e.route + row);
        if (r.x >= 0)
            return {reinterpret_cast<V *>(e.peer_rows[r.x]) + (long long)r.y * e.route_nvec + e.route_col0, true};
    }
    return {reinterpret_cast<V *>(Y + (long long)row * ldy), false};
}

// Where the gathered rows come from.  Without HOT only X is used.
struct Gather {
    const float *X = nullptr;
    long long ldv = 0;                  // leading dimension of X in vectors
    const float *hot = nullptr;         // table of hot rows, [hot_rows, nvec] vectors, dense
    const int *hot_ids = nullptr;       // column of every hot position (all tagged positions, also those beyond hot_rows)
    int hot_rows = 0;                   // tagged positions below this are served from the table
};

// Tagged columns whose position lies beyond the rows the table holds at this call's width are turned back into
// plain columns (one look-up in hot_ids).  Done on the freshly loaded (col) registers of a lane, before they are
// handed around, so that the gathers themselves need no branch and no dependent load.
template <bool HOT>
__device__ __forceinline__ unsigned resolve_column(const Gather &g, unsigned c) {
    if (HOT && (c & kHotTag) && (int)(c & kHotMask) >= g.hot_rows) c = (unsigned)__ldg(g.hot_ids + (c & kHotMask));
    return c;
}

// Address of the row a resolved column stands for: a row of the table for a tagged column, a row of X otherwise.
// Branch-free, so that the gathers of a batch stay independent loads in flight together.  The table is written by
// the fill kernel that precedes the gathering kernels of the same call in stream order, so the read-only load path
// is safe for it as well.
template <int VEC, bool HOT>
__device__ __forceinline__ const typename Vec<VEC>::type *row_address(const Gather &g, unsigned c, int gl, int nvec) {
    using V = typename Vec<VEC>::type;
    if (!HOT) return reinterpret_cast<const V *>(g.X) + (long long)c * g.ldv + gl;
    const bool tagged = (c & kHotTag) != 0;
    const V *base = reinterpret_cast<const V *>(tagged ? g.hot : g.X);
    const long long stride = tagged ? (long long)nvec : g.ldv;
    return base + (long long)(c & kHotMask) * stride + gl;
}

// Programmatic dependent launch: the next kernel of the stream may start once every block of this one has, and waits
// (wait_for_operands) until this one has finished and its results are visible.
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_operands() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <bool EARLY>
__device__ __forceinline__ float row_scale_of(const Epilogue &e, int row) {
    if (e.row_scale == nullptr) return 1.f;
    if (!EARLY) return __ldg(e.row_scale + row);
    return ld_coherent(e.row_scale + row, l2_policy_keep());
}

// ---------------------------------------------------------------------------
// 0. table of hot rows: hot[pos, :] = X[hot_ids[pos], :] for pos < hot_rows (dense, nvec vectors per row).
// ---------------------------------------------------------------------------
template <int VEC>
__global__ void __launch_bounds__(256)
spmm_fill_hot_kernel(const int *__restrict__ hot_ids, int hot_rows, const float *__restrict__ X, long long ldv, int nvec,
                     float *__restrict__ hot) {
    using V = typename Vec<VEC>::type;
    const long long total = (long long)hot_rows * nvec;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int pos = (int)(i / nvec), j = (int)(i - (long long)pos * nvec);
        reinterpret_cast<V *>(hot)[i] = __ldg(reinterpret_cast<const V *>(X) + (long long)__ldg(hot_ids + pos) * ldv + j);
    }
}

// Blocks per SM the two kernels of large plans are compiled for.  Left to itself (0) the compiler aims at 40 registers in
// the chunk kernel, which hold five of a batch's eight row vectors and fewer where the loads are predicated; 64 registers
// hold all eight, and 32 warps with eight loads each are worth more than 48 with four or five (R-MAT-24, F = 32: 4.69 ->
// 4.37 ms; R-MAT-20 symmetrised: F = 64 599 -> 574 us, F = 100 1427 -> 984; products-shaped, F = 47: 6.7 -> 4.6 ms).  Wider
// rows need more registers for the same (F = 400 on R-MAT-20: 7.8 -> 4.4 ms, F = 1000: 23.6 -> 13.0); where all of a lane's
// vectors lie inside the row the compiler's own choice was the better one above one vector a lane.
constexpr int chunk_blocks_per_sm(int G, int VPL, int VEC, bool EXACT) {
    if (VEC != 4 || G < 8) return 0;
    if (VPL == 1) return 4;
    if (EXACT) return 0;
    return VPL == 2 ? 4 : VPL <= 4 ? 3 : 2;
}
// Short rows: five blocks leave 48 registers, enough for the four row vectors of a step (56 / 48 / 40 registers, us: power law,
// 1.2 M rows of 17, F = 32 417 / 388 / 461, F = 64 765 / 713 / 799; R-MAT-22 F = 32 865 / 838 / 897).  Groups of one or two
// lanes take 44 or fewer anyway, and with the bound at five came out slower (1.2 M rows of 9, F = 8: 129 / 156).
constexpr int short_blocks_per_sm(int G, int VPL, int VEC, bool EXACT) {
    return VEC != 4 || VPL > 1 ? 0 : EXACT && G < 4 ? 4 : 5;
}

// ---------------------------------------------------------------------------
// 1. short rows: one lane group walks a range of the short-row stream
//    (about kShortRangeNnz entries, whole rows only) and writes each row when
//    its last entry has been added.  Entries of a row are added in CSR order
//    into one accumulator.
// ---------------------------------------------------------------------------
// `range`: the lane group's range; groups beyond the last one only take part in the shuffles.  EARLY: the kernel may have
// started before its operands were complete; the plan's lists are read before it waits for them.
template <int G, int VPL, int VEC, int U, bool EXACT, bool UNIT, bool HOT, bool EARLY>
__device__ __forceinline__ void walk_short_range(long long range, const int *__restrict__ s_range_row, int n_ranges,
                                                 const int *__restrict__ s_rowptr, const int *__restrict__ s_rows,
                                                 const int *__restrict__ s_col, const float *__restrict__ s_val,
                                                 const Gather &g, float *__restrict__ Y, long long ldy, int nvec,
                                                 const Epilogue &epi) {
    using V = typename Vec<VEC>::type;
    constexpr int UU = MinOf<U, G>::value;
    constexpr bool BRANCH = VEC == 1 && VPL >= 8 && !EARLY;
    constexpr int SURE = VPL == 8 || VPL == 12 ? 0 : sure_vectors(G, VPL, VEC);      // those two lost by it here
    const int gl = threadIdx.x & (G - 1);
    int ri = 0, k = 0, kend = 0;
    if (range < n_ranges) {
        ri = s_range_row[range];
        const int ri_end = s_range_row[range + 1];
        k = s_rowptr[ri];
        kend = s_rowptr[ri_end];
    }
    int maxlen = kend - k;
#pragma unroll
    for (int o = G; o < 32; o <<= 1) maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, o));

    const unsigned long long pol_keep = l2_policy_keep(), pol_stream = l2_policy_stream();
    V acc[VPL];
#pragma unroll
    for (int p = 0; p < VPL; ++p) acc[p] = Vec<VEC>::zero();

    unsigned c_next = 0;
    float v_next = UNIT ? 1.f : 0.f;
    if (k + gl < kend) {
        c_next = (unsigned)ld_stream(s_col + k + gl, pol_stream);
        if (!UNIT) v_next = ld_stream(s_val + k + gl, pol_stream);
    }
    if (EARLY) wait_for_operands();
    for (int base = 0; base < maxlen; base += G) {
        const unsigned c = (c_next & ~kColMask) | resolve_column<HOT>(g, c_next & kColMask);
        const float v = v_next;
        c_next = 0;
        if (!UNIT) v_next = 0.f;
        if (k + base + G + gl < kend) {   // next batch, requested before this batch's gathers
            c_next = (unsigned)ld_stream(s_col + k + base + G + gl, pol_stream);
            if (!UNIT) v_next = ld_stream(s_val + k + base + G + gl, pol_stream);
        }
        const int lim = min(G, maxlen - base);
        for (int j = 0; j < lim; j += UU) {
            unsigned cc[UU];
            float vv[UU];
            V x[UU][VPL];
#pragma unroll
            for (int u = 0; u < UU; ++u) {
                cc[u] = __shfl_sync(0xffffffffu, c, j + u, G);
                vv[u] = UNIT ? 1.f : __shfl_sync(0xffffffffu, v, j + u, G);
            }
#pragma unroll
            for (int u = 0; u < UU; ++u) {
                const bool live = (k + base + j + u < kend) && !(cc[u] & kPlaceholder);
                const V *xr = row_address<VEC, HOT>(g, live ? (cc[u] & kColMask) : 0u, gl, nvec);
#pragma unroll
                for (int p = 0; p < VPL; ++p)
                    x[u][p] = ld_row_if<BRANCH, VEC, EARLY>(xr + p * G, pol_keep, live && (EXACT || p < SURE || gl + p * G < nvec));
            }
#pragma unroll
            for (int u = 0; u < UU; ++u) {
#pragma unroll
                for (int p = 0; p < VPL; ++p) Vec<VEC>::fma(acc[p], vv[u], x[u][p]);
                if ((cc[u] & kLastInRow) && (k + base + j + u < kend)) {
                    const int row = s_rows[ri];
                    const float scale = row_scale_of<EARLY>(epi, row);
                    const RowDestination<VEC> dest = row_destination<VEC>(epi, Y, ldy, row);
                    const bool remote = dest.remote;
                    V *yr = dest.ptr + gl;
#pragma unroll
                    for (int p = 0; p < VPL; ++p) {
                        if (EXACT || gl + p * G < nvec) {
                            const V out = finish_row<VEC>(acc[p], epi, scale);
                            if (remote) yr[p * G] = out;
                            else st_stream(yr + p * G, out, pol_stream);
                        }
                        acc[p] = Vec<VEC>::zero();
                    }
                    ++ri;
                }
            }
        }
    }
}

// The same for rows that one or two lanes hold: with an entry a lane their group would have one or two gathers in flight, so a
// lane takes EPL entries of the stream at a time (the neighbours of the first come from L1).  us a call before / with it, and with
// the chunks' batches below: F = 1 R-MAT-12 15 / 9, power law 60,000 rows of 21 30 / 16, 1 M rows of 21 358 / 149; F = 2 R-MAT-18
// 69 / 46; F = 4 R-MAT-12 16 / 11, 300,000 rows of 8 34 / 24, R-MAT-21 472 / 334; F = 8 R-MAT-12 10.2 / 9.4, R-MAT-21 400 / 370.
// Two lanes with four entries each were no better (R-MAT-20, F = 8: 123 / 141), nor were groups of four lanes with two.
constexpr int short_entries_per_lane(int G, int VPL, int VEC) {
    return VPL > 1 || G > 2 ? 1 : VEC == 1 ? 8 / G : 4 / G;
}
template <int G, int VEC, bool EXACT, bool UNIT, bool HOT, bool EARLY>
__device__ __forceinline__ void walk_short_range_narrow(long long range, const int *__restrict__ s_range_row, int n_ranges,
                                                        const int *__restrict__ s_rowptr, const int *__restrict__ s_rows,
                                                        const int *__restrict__ s_col, const float *__restrict__ s_val,
                                                        const Gather &g, float *__restrict__ Y, long long ldy, int nvec,
                                                        const Epilogue &epi) {
    using V = typename Vec<VEC>::type;
    constexpr int EPL = short_entries_per_lane(G, 1, VEC), BATCH = G * EPL;
    const int gl = threadIdx.x & (G - 1);
    int ri = 0, k = 0, kend = 0;
    if (range < n_ranges) {
        ri = s_range_row[range];
        const int ri_end = s_range_row[range + 1];
        k = s_rowptr[ri];
        kend = s_rowptr[ri_end];
    }
    int maxlen = kend - k;
#pragma unroll
    for (int o = G; o < 32; o <<= 1) maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, o));
    const unsigned long long pol_keep = l2_policy_keep(), pol_stream = l2_policy_stream();
    V acc = Vec<VEC>::zero();
    unsigned c_next[EPL];
    float v_next[EPL];
    auto request = [&](int at) {      // entry e * G + gl of the batch at `at`
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            const int i = at + e * G + gl;
            c_next[e] = i < kend ? (unsigned)__ldg(s_col + i) : kPlaceholder;
            v_next[e] = UNIT ? 1.f : i < kend ? __ldg(s_val + i) : 0.f;
        }
    };
    request(k);
    if (EARLY) wait_for_operands();
    for (int base = 0; base < maxlen; base += BATCH) {
        unsigned c[EPL];
        float v[EPL];
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            c[e] = (c_next[e] & ~kColMask) | resolve_column<HOT>(g, c_next[e] & kColMask);
            v[e] = v_next[e];
        }
        request(k + base + BATCH);      // next batch, before this batch's gathers
        unsigned cc[BATCH];
        float vv[BATCH];
        V x[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            cc[u] = __shfl_sync(0xffffffffu, c[u / G], u, G);      // lane numbers count modulo G
            vv[u] = UNIT ? 1.f : __shfl_sync(0xffffffffu, v[u / G], u, G);
            const bool live = !(cc[u] & kPlaceholder);
            x[u] = ld_gathered_if<EARLY>(row_address<VEC, HOT>(g, live ? (cc[u] & kColMask) : 0u, gl, nvec), pol_keep,
                                         live && (EXACT || gl < nvec));
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            Vec<VEC>::fma(acc, vv[u], x[u]);
            if (cc[u] & kLastInRow) {
                const int row = s_rows[ri];
                const float scale = row_scale_of<EARLY>(epi, row);
                const RowDestination<VEC> dest = row_destination<VEC>(epi, Y, ldy, row);
                if (EXACT || gl < nvec) {
                    const V out = finish_row<VEC>(acc, epi, scale);
                    if (dest.remote) dest.ptr[gl] = out;
                    else st_stream(dest.ptr + gl, out, pol_stream);
                }
                acc = Vec<VEC>::zero();
                ++ri;
            }
        }
    }
}

template <int G, int VPL, int VEC, int U, bool EXACT, bool UNIT, bool HOT>
__global__ void __launch_bounds__(256, short_blocks_per_sm(G, VPL, VEC, EXACT))
spmm_short_stream_kernel(const int *__restrict__ s_range_row, int n_ranges, const int *__restrict__ s_rowptr,
                         const int *__restrict__ s_rows, const int *__restrict__ s_col,
                         const float *__restrict__ s_val, Gather g, float *__restrict__ Y, long long ldy, int nvec,
                         Epilogue epi) {
    const long long range = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * (32 / G) + (threadIdx.x & 31) / G;
    if constexpr (short_entries_per_lane(G, VPL, VEC) > 1)
        walk_short_range_narrow<G, VEC, EXACT, UNIT, HOT, false>(range, s_range_row, n_ranges, s_rowptr, s_rows, s_col, s_val, g, Y, ldy,
                                                                 nvec, epi);
    else
        walk_short_range<G, VPL, VEC, U, EXACT, UNIT, HOT, false>(range, s_range_row, n_ranges, s_rowptr, s_rows, s_col, s_val, g, Y,
                                                                  ldy, nvec, epi);
}

// ---------------------------------------------------------------------------
// 2. chunks of long rows: one warp per chunk.  The warp loads 32 (col, val)
//    pairs at a time; its 32/G lane groups take interleaved entries.  Warps take
//    chunks from `counter` kChunkGroup at a time (the counter starts at 0; the group size is a compile-time
//    constant on purpose: with a run-time size the compiler produced a tighter loop over the group that ran a
//    quarter slower on the largest graphs); the
//    next group's index is requested while the current group is being worked on,
//    and the first (col, val) batch of the next chunk while the current chunk is.
// ---------------------------------------------------------------------------
constexpr int kChunkGroup = 4;

// SURE: how many of a lane's vectors need no test against the width.
// Sum of one chunk: nonzeros [k0, k0 + len), taken in interleaved order by the warp's lane groups; (c, v) hold the
// lane's entry of the first 32.  Every lane group ends with the same totals in acc.
template <int G, int VPL, int VEC, int U, bool EXACT, bool UNIT, bool HOT, bool EARLY, int SURE>
__device__ __forceinline__ void sum_chunk(typename Vec<VEC>::type *acc, const int *__restrict__ col,
                                          const float *__restrict__ val, const Gather &g, int k0, int len, int c, float v,
                                          int nvec, unsigned long long pol_keep, unsigned long long pol_stream) {
    using V = typename Vec<VEC>::type;
    constexpr int RPW = 32 / G;
    constexpr int UU = MinOf<U, G>::value;
    constexpr bool BRANCH = VEC == 1 && VPL == 32 && !EARLY;
    const int lane = threadIdx.x & 31;
    const int gl = lane & (G - 1);
    const int gi = lane / G;
#pragma unroll
    for (int p = 0; p < VPL; ++p) acc[p] = Vec<VEC>::zero();

    int base = 0;
    // full batches of 32 entries: no bounds checks.  (col, val) of the next batch are requested before the
    // gathers of the current one, so the dependent chain col -> X row costs one memory latency per batch
    for (; base + 32 <= len; base += 32) {
        int c_next = 0;
        float v_next = UNIT ? 1.f : 0.f;
        if (base + 32 + lane < len) {
            c_next = ld_stream(col + k0 + base + 32 + lane, pol_stream);
            if (!UNIT) v_next = ld_stream(val + k0 + base + 32 + lane, pol_stream);
        }
#pragma unroll
        for (int t = 0; t < G; t += UU) {
            int cc[UU];
            float vv[UU];
            V x[UU][VPL];
#pragma unroll
            for (int u = 0; u < UU; ++u) {
                cc[u] = __shfl_sync(0xffffffffu, c, (t + u) * RPW + gi);
                vv[u] = UNIT ? 1.f : __shfl_sync(0xffffffffu, v, (t + u) * RPW + gi);
            }
#pragma unroll
            for (int u = 0; u < UU; ++u) {
                const V *xr = row_address<VEC, HOT>(g, (unsigned)cc[u], gl, nvec);
#pragma unroll
                for (int p = 0; p < VPL; ++p)
                    x[u][p] = EXACT || p < SURE ? ld_gathered<EARLY>(xr + p * G, pol_keep)
                                                : ld_row_if<BRANCH, VEC, EARLY>(xr + p * G, pol_keep, gl + p * G < nvec);
            }
#pragma unroll
            for (int u = 0; u < UU; ++u)
#pragma unroll
                for (int p = 0; p < VPL; ++p) Vec<VEC>::fma(acc[p], vv[u], x[u][p]);
        }
        c = (int)resolve_column<HOT>(g, (unsigned)c_next);
        v = v_next;
    }
    // last, partial batch (entries beyond the chunk were loaded as zeros)
    if (base < len) {
        const int cnt = len - base;
        const int steps = (cnt + RPW - 1) / RPW;  // <= G
        for (int t = 0; t < steps; t += UU) {
            int cc[UU];
            float vv[UU];
            V x[UU][VPL];
#pragma unroll
            for (int u = 0; u < UU; ++u) {
                const int e = (t + u) * RPW + gi;
                cc[u] = __shfl_sync(0xffffffffu, c, e & 31);
                vv[u] = UNIT ? 1.f : __shfl_sync(0xffffffffu, v, e & 31);
                if (e >= cnt) { vv[u] = 0.f; cc[u] = 0; }
            }
#pragma unroll
            for (int u = 0; u < UU; ++u) {
                const bool live = (t + u) * RPW + gi < cnt;
                const V *xr = row_address<VEC, HOT>(g, (unsigned)cc[u], gl, nvec);
#pragma unroll
                for (int p = 0; p < VPL; ++p)
                    x[u][p] = ld_row_if<BRANCH, VEC, EARLY>(xr + p * G, pol_keep, live && (EXACT || p < SURE || gl + p * G < nvec));
            }
#pragma unroll
            for (int u = 0; u < UU; ++u)
#pragma unroll
                for (int p = 0; p < VPL; ++p) Vec<VEC>::fma(acc[p], vv[u], x[u][p]);
        }
    }
    // combine the lane groups (butterfly: every lane ends with the same total)
#pragma unroll
    for (int o = G; o < 32; o <<= 1)
#pragma unroll
        for (int p = 0; p < VPL; ++p) Vec<VEC>::add(acc[p], Vec<VEC>::shfl_xor(acc[p], o));
}

// Batches of 32 entries that a warp takes together: a batch of rows that one or two lanes hold is one or two gathers a lane.
// Four, but two in the one launch of a small plan for pairs of lanes, where four cost registers that its short rows want (us, F = 8,
// two / four: power law, 100,000 rows of 51 51 / 75; the separate kernels: R-MAT-18 70 / 60, R-MAT-20 129 / 123).  Fewer where the
// work does without (large_plan_batches, small_plan_batches); the sums and their order are the same.
constexpr int chunk_batches(int G, int VPL, int VEC, bool one_launch) {
    return VPL > 1 || G > 2 ? 1 : G == 2 && VEC == 4 && one_launch ? 2 : 4;
}

// The lane's entries of the first NB batches of [k0, k0 + len).
template <int NB, bool UNIT>
__device__ __forceinline__ void first_batches(int (&c)[NB], float (&v)[NB], const int *__restrict__ col, const float *__restrict__ val,
                                              int k0, int len, unsigned long long pol_stream) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const bool live = b * 32 + lane < len;
        c[b] = live ? ld_stream(col + k0 + b * 32 + lane, pol_stream) : 0;
        v[b] = UNIT ? 1.f : live ? ld_stream(val + k0 + b * 32 + lane, pol_stream) : 0.f;
    }
}

// sum_chunk for such rows, the same sums in the same order.
template <int G, int VEC, bool EXACT, bool UNIT, bool HOT, bool EARLY, int NB>
__device__ __forceinline__ void sum_chunk_narrow(typename Vec<VEC>::type &acc, const int *__restrict__ col, const float *__restrict__ val,
                                                 const Gather &g, int k0, int len, int (&c)[NB], float (&v)[NB], int nvec,
                                                 unsigned long long pol_keep, unsigned long long pol_stream) {
    using V = typename Vec<VEC>::type;
    constexpr int RPW = 32 / G;
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), gi = lane / G;
    acc = Vec<VEC>::zero();
    for (int base = 0; base < len; base += 32 * NB) {
        int c_next[NB];
        float v_next[NB], vv[NB * G];
        V x[NB * G];
        first_batches<NB, UNIT>(c_next, v_next, col, val, k0 + base + 32 * NB, len - base - 32 * NB, pol_stream);
#pragma unroll
        for (int i = 0; i < NB * G; ++i) {
            const int e = (i % G) * RPW + gi, cc = __shfl_sync(0xffffffffu, c[i / G], e);
            vv[i] = UNIT ? 1.f : __shfl_sync(0xffffffffu, v[i / G], e);
            x[i] = ld_gathered_if<EARLY>(row_address<VEC, HOT>(g, (unsigned)cc, gl, nvec), pol_keep,
                                         base + i / G * 32 + e < len && (EXACT || gl < nvec));
        }
#pragma unroll
        for (int i = 0; i < NB * G; ++i) Vec<VEC>::fma(acc, vv[i], x[i]);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            c[b] = (int)resolve_column<HOT>(g, (unsigned)c_next[b]);
            v[b] = v_next[b];
        }
    }
#pragma unroll
    for (int o = G; o < 32; o <<= 1) Vec<VEC>::add(acc, Vec<VEC>::shfl_xor(acc, o));
}

template <int G, int VPL, int VEC, int U, bool EXACT, bool UNIT, bool HOT, int NB>
__global__ void __launch_bounds__(256, chunk_blocks_per_sm(G, VPL, VEC, EXACT))
spmm_chunks_kernel(const Chunk *__restrict__ chunks, int n_chunks, const int *__restrict__ col,
                   const float *__restrict__ val, Gather g, float *__restrict__ Y, long long ldy,
                   float *__restrict__ partials, int nvec, Epilogue epi, unsigned *counter) {
    using V = typename Vec<VEC>::type;
    const int lane = threadIdx.x & 31;
    const int gl = lane & (G - 1);
    const int gi = lane / G;
    const unsigned long long pol_keep = l2_policy_keep(), pol_stream = l2_policy_stream();

    unsigned group = 0;
    if (lane == 0) group = atomicAdd(counter, (unsigned)kChunkGroup);
    group = __shfl_sync(0xffffffffu, group, 0);
    while (group < (unsigned)n_chunks) {
        int4 desc = make_int4(0, 0, 0, 0);
        if (lane < kChunkGroup && group + lane < (unsigned)n_chunks)
            desc = __ldg(reinterpret_cast<const int4 *>(chunks) + group + lane);
        const int in_group = min(kChunkGroup, n_chunks - (int)group);
        unsigned next_group = 0;
        if (lane == 0) next_group = atomicAdd(counter, (unsigned)kChunkGroup);   // needed only after this group

        // first batch of the group's first chunk
        int cs[NB];      // the same of several batches (NB > 1)
        float vs[NB];
        int c = 0;
        float v = UNIT ? 1.f : 0.f;
        if constexpr (NB > 1) {
            first_batches<NB, UNIT>(cs, vs, col, val, __shfl_sync(0xffffffffu, desc.y, 0), __shfl_sync(0xffffffffu, desc.z, 0), pol_stream);
#pragma unroll
            for (int b = 0; b < NB; ++b) cs[b] = (int)resolve_column<HOT>(g, (unsigned)cs[b]);
        } else {
            const int k0 = __shfl_sync(0xffffffffu, desc.y, 0), len = __shfl_sync(0xffffffffu, desc.z, 0);
            if (lane < len) {
                c = ld_stream(col + k0 + lane, pol_stream);
                if (!UNIT) v = ld_stream(val + k0 + lane, pol_stream);
            }
            c = (int)resolve_column<HOT>(g, (unsigned)c);
        }
        for (int j = 0; j < in_group; ++j) {
            const int row = __shfl_sync(0xffffffffu, desc.x, j), k0 = __shfl_sync(0xffffffffu, desc.y, j);
            const int len = __shfl_sync(0xffffffffu, desc.z, j), slot = __shfl_sync(0xffffffffu, desc.w, j);
            // first batch of the chunk after this one, requested now and used when this chunk is done
            int cs_ahead[NB];
            float vs_ahead[NB];
            int c_ahead = 0;
            float v_ahead = UNIT ? 1.f : 0.f;
            if constexpr (NB > 1) {
                const int nk0 = __shfl_sync(0xffffffffu, desc.y, j + 1), nlen = __shfl_sync(0xffffffffu, desc.z, j + 1);
                first_batches<NB, UNIT>(cs_ahead, vs_ahead, col, val, nk0, j + 1 < in_group ? nlen : 0, pol_stream);
            } else if (j + 1 < in_group) {
                const int nk0 = __shfl_sync(0xffffffffu, desc.y, j + 1), nlen = __shfl_sync(0xffffffffu, desc.z, j + 1);
                if (lane < nlen) {
                    c_ahead = ld_stream(col + nk0 + lane, pol_stream);
                    if (!UNIT) v_ahead = ld_stream(val + nk0 + lane, pol_stream);
                }
            }

            V acc[VPL];
            if constexpr (NB > 1)
                sum_chunk_narrow<G, VEC, EXACT, UNIT, HOT, false, NB>(acc[0], col, val, g, k0, len, cs, vs, nvec, pol_keep, pol_stream);
            else
                sum_chunk<G, VPL, VEC, U, EXACT, UNIT, HOT, false, sure_vectors(G, VPL, VEC)>(acc, col, val, g, k0, len, c, v, nvec, pol_keep, pol_stream);

            if (gi == 0) {
                if (slot < 0) {
                    const float scale = epi.row_scale ? __ldg(epi.row_scale + row) : 1.f;
                    const RowDestination<VEC> dest = row_destination<VEC>(epi, Y, ldy, row);
                    const bool remote = dest.remote;
                    V *out = dest.ptr + gl;
#pragma unroll
                    for (int p = 0; p < VPL; ++p)
                        if (EXACT || gl + p * G < nvec) {
                            const V tot = finish_row<VEC>(acc[p], epi, scale);
                            if (remote) out[p * G] = tot;
                            else st_stream(out + p * G, tot, pol_stream);
                        }
                } else {
                    V *out = reinterpret_cast<V *>(partials + (long long)slot * nvec * VEC) + gl;
#pragma unroll
                    for (int p = 0; p < VPL; ++p)
                        if (EXACT || gl + p * G < nvec) out[p * G] = acc[p];
                }
            }
            if constexpr (NB > 1) {
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    cs[b] = (int)resolve_column<HOT>(g, (unsigned)cs_ahead[b]);
                    vs[b] = vs_ahead[b];
                }
            } else {
                c = (int)resolve_column<HOT>(g, (unsigned)c_ahead);
                v = v_ahead;
            }
        }  // chunks of the group
        group = __shfl_sync(0xffffffffu, next_group, 0);
    }
}

// ---------------------------------------------------------------------------
// 3. split rows: add the partial slots of a row in slot order.
//    The first n_wide blocks take one entry each of the plan's list of wide rows, all eight warps share the row and
//    their sums are added in warp order through shared memory; the other blocks take eight rows each, one per warp,
//    leaving rows with more than kWideSlots slots to the first ones.  A warp's lane groups take interleaved slots.
//    Bound: latency, since a row is a handful of loads; four of them are in flight per lane, and both kinds of rows share
//    one launch (R-MAT-20 symmetrised, F = 64: 18 + 13 us in two launches, the whole call 619 -> 599 us in one).
// ---------------------------------------------------------------------------
template <int G, int VPL, int VEC>
__global__ void __launch_bounds__(256)
spmm_reduce_partials_kernel(const SplitRow *__restrict__ split, int n_split, const SplitRow *__restrict__ wide, int n_wide,
                            const float *__restrict__ partials, float *__restrict__ Y, long long ldy, int nvec, Epilogue epi) {
    using V = typename Vec<VEC>::type;
    constexpr int RPW = 32 / G;
    extern __shared__ float smem[];  // [8][nvec*VEC] for the wide rows
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const int gl = lane & (G - 1);
    const int gi = lane / G;
    const bool is_wide = (int)blockIdx.x < n_wide;
    const long long entry = is_wide ? (long long)blockIdx.x : ((long long)blockIdx.x - n_wide) * 8 + w;
    if (!is_wide && entry >= n_split) return;
    const int4 raw = __ldg(reinterpret_cast<const int4 *>(is_wide ? wide : split) + entry);
    const int row = raw.x, slot0 = raw.y, nslots = raw.z;
    if (!is_wide && nslots > kWideSlots) return;

    V acc[VPL];
#pragma unroll
    for (int p = 0; p < VPL; ++p) acc[p] = Vec<VEC>::zero();
    const int first = is_wide ? w * RPW + gi : gi;
    const int stride = is_wide ? 8 * RPW : RPW;
    constexpr int UR = VPL <= 2 ? 4 : 1;
    for (int sidx = first; sidx < nslots; sidx += UR * stride) {
        V x[UR][VPL];
#pragma unroll
        for (int u = 0; u < UR; ++u) {
            const V *pr = reinterpret_cast<const V *>(partials + (long long)(slot0 + sidx + u * stride) * nvec * VEC);
#pragma unroll
            for (int p = 0; p < VPL; ++p)
                x[u][p] = sidx + u * stride < nslots && gl + p * G < nvec ? pr[gl + p * G] : Vec<VEC>::zero();
        }
#pragma unroll
        for (int u = 0; u < UR; ++u)
#pragma unroll
            for (int p = 0; p < VPL; ++p)
                if (sidx + u * stride < nslots) Vec<VEC>::add(acc[p], x[u][p]);
    }
#pragma unroll
    for (int o = G; o < 32; o <<= 1)
#pragma unroll
        for (int p = 0; p < VPL; ++p) Vec<VEC>::add(acc[p], Vec<VEC>::shfl_xor(acc[p], o));

    const float scale = epi.row_scale ? __ldg(epi.row_scale + row) : 1.f;
    const RowDestination<VEC> dest = row_destination<VEC>(epi, Y, ldy, row);
    const bool remote = dest.remote;
    V *yr = dest.ptr;
    if (!is_wide) {
        if (gi == 0) {
#pragma unroll
            for (int p = 0; p < VPL; ++p) {
                const int vi = gl + p * G;
                if (vi < nvec) {
                    if (remote) yr[vi] = finish_row<VEC>(acc[p], epi, scale);
                    else __stcs(yr + vi, finish_row<VEC>(acc[p], epi, scale));
                }
            }
        }
        return;
    }
    V *sm = reinterpret_cast<V *>(smem);
    if (gi == 0) {
#pragma unroll
        for (int p = 0; p < VPL; ++p) {
            const int vi = gl + p * G;
            if (vi < nvec) sm[w * nvec + vi] = acc[p];
        }
    }
    __syncthreads();
    if (w == 0 && gi == 0) {
#pragma unroll
        for (int p = 0; p < VPL; ++p) {
            const int vi = gl + p * G;
            if (vi < nvec) {
                V tot = sm[vi];
                for (int ww = 1; ww < 8; ++ww) Vec<VEC>::add(tot, sm[ww * nvec + vi]);
                if (remote) yr[vi] = finish_row<VEC>(tot, epi, scale);
                else __stcs(yr + vi, finish_row<VEC>(tot, epi, scale));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// 4. small plans: the three steps in one launch.  Blocks below `chunk_blocks` take one chunk per warp, the others walk
//    the short-row stream; the warp that writes the last partial sum of a split row (counted in `arrived`, which it
//    sets back to 0) adds the row's slots, lane groups taking interleaved slots.  A call on such a plan is a few
//    microseconds of work, so the memset, the four launches and the fork and join of the big plans' path used to be
//    most of it (R-MAT-12 symmetrised, F = 16: 24 us of GPU and host time per call, 8 with this kernel; F = 64: 44, 12).
//    The kernel starts while the one before it in the stream still runs, reads the plan's lists, and only then waits for
//    the operands (9.2 -> 8.0 us a call in a row of calls).
// ---------------------------------------------------------------------------
template <int VEC>
__device__ __forceinline__ void store_vector(const RowDestination<VEC> &dest, int vi, const typename Vec<VEC>::type &v,
                                             unsigned long long pol) {
    if (dest.remote) dest.ptr[vi] = v;
    else st_stream(dest.ptr + vi, v, pol);
}

// NB = 1 for rows that one or two lanes hold: the short rows too have one entry a lane at a time, in fewer registers.
template <int G, int VPL, int VEC, int U, bool EXACT, bool UNIT, int BLOCKS_PER_SM, int SURE = sure_vectors(G, VPL, VEC),
          int NB = chunk_batches(G, VPL, VEC, true)>
__global__ void __launch_bounds__(256, BLOCKS_PER_SM)
spmm_small_kernel(const Chunk *__restrict__ chunks, int n_chunks, int chunk_blocks, const int *__restrict__ col,
                  const float *__restrict__ val, const SplitRow *__restrict__ split, const int *__restrict__ slot_split,
                  int *arrived, float *partials, const int *__restrict__ s_range_row, int n_ranges,
                  const int *__restrict__ s_rowptr, const int *__restrict__ s_rows, const int *__restrict__ s_col,
                  const float *__restrict__ s_val, Gather g, float *__restrict__ Y, long long ldy, int nvec, Epilogue epi) {
    using V = typename Vec<VEC>::type;
    constexpr int RPW = 32 / G;
    const int lane = threadIdx.x & 31;
    const int gl = lane & (G - 1);
    const int gi = lane / G;
    let_next_kernel_start();
    if ((int)blockIdx.x >= chunk_blocks) {
        const long long warp = (((int)blockIdx.x - chunk_blocks) * (long long)blockDim.x + threadIdx.x) >> 5;
        if constexpr (short_entries_per_lane(G, VPL, VEC) > 1 && NB > 1)
            walk_short_range_narrow<G, VEC, EXACT, UNIT, false, true>(warp * RPW + gi, s_range_row, n_ranges, s_rowptr, s_rows, s_col,
                                                                      s_val, g, Y, ldy, nvec, epi);
        else
            walk_short_range<G, VPL, VEC, U, EXACT, UNIT, false, true>(warp * RPW + gi, s_range_row, n_ranges, s_rowptr, s_rows, s_col,
                                                                       s_val, g, Y, ldy, nvec, epi);
        return;
    }
    const int at = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (at >= n_chunks) return;
    const unsigned long long pol_keep = l2_policy_keep(), pol_stream = l2_policy_stream();
    const int4 ch = __ldg(reinterpret_cast<const int4 *>(chunks) + at);      // row, first nonzero, length, slot
    int cs[NB];
    float vs[NB];
    int c = 0;
    float v = UNIT ? 1.f : 0.f;
    if constexpr (NB > 1) {
        first_batches<NB, UNIT>(cs, vs, col, val, ch.y, ch.z, pol_stream);
    } else if (lane < ch.z) {
        c = ld_stream(col + ch.y + lane, pol_stream);
        if (!UNIT) v = ld_stream(val + ch.y + lane, pol_stream);
    }
    const int which = ch.w >= 0 ? __ldg(slot_split + ch.w) : 0;
    const int4 sr = ch.w >= 0 ? __ldg(reinterpret_cast<const int4 *>(split) + which) : ch;      // row, first slot, slots
    V acc[VPL];
    wait_for_operands();
    if constexpr (NB > 1)
        sum_chunk_narrow<G, VEC, EXACT, UNIT, false, true, NB>(acc[0], col, val, g, ch.y, ch.z, cs, vs, nvec, pol_keep, pol_stream);
    else
        sum_chunk<G, VPL, VEC, 2 * U, EXACT, UNIT, false, true, SURE>(acc, col, val, g, ch.y, ch.z, c, v, nvec, pol_keep, pol_stream);
    int row = ch.x;
    if (ch.w >= 0) {
        if (gi == 0) {
            V *out = reinterpret_cast<V *>(partials + (long long)ch.w * nvec * VEC) + gl;
#pragma unroll
            for (int p = 0; p < VPL; ++p)
                if (EXACT || gl + p * G < nvec) out[p * G] = acc[p];
        }
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) last = atomicAdd(arrived + which, 1) == sr.z - 1;
        if (!__shfl_sync(0xffffffffu, last, 0)) return;
        __threadfence();
        if (lane == 0) arrived[which] = 0;
        // the order of spmm_reduce_partials_kernel: one pass over interleaved slots, or for many slots its eight warps'
        // shares one after the other
        const int shares = sr.z > kWideSlots ? 8 : 1;
        V tot[VPL];
        for (int w = 0; w < shares; ++w) {
#pragma unroll
            for (int p = 0; p < VPL; ++p) acc[p] = Vec<VEC>::zero();
#pragma unroll 4
            for (int sidx = w * RPW + gi; sidx < sr.z; sidx += shares * RPW) {
                const V *pr = reinterpret_cast<const V *>(partials + (long long)(sr.y + sidx) * nvec * VEC);
#pragma unroll
                for (int p = 0; p < VPL; ++p)
                    if (EXACT || gl + p * G < nvec) Vec<VEC>::add(acc[p], __ldcg(pr + gl + p * G));
            }
#pragma unroll
            for (int o = G; o < 32; o <<= 1)
#pragma unroll
                for (int p = 0; p < VPL; ++p) Vec<VEC>::add(acc[p], Vec<VEC>::shfl_xor(acc[p], o));
#pragma unroll
            for (int p = 0; p < VPL; ++p) {
                if (w == 0) tot[p] = acc[p];
                else Vec<VEC>::add(tot[p], acc[p]);
            }
        }
#pragma unroll
        for (int p = 0; p < VPL; ++p) acc[p] = tot[p];
        row = sr.x;
    }
    if (gi == 0) {
        const float scale = row_scale_of<true>(epi, row);
        const RowDestination<VEC> dest = row_destination<VEC>(epi, Y, ldy, row);
#pragma unroll
        for (int p = 0; p < VPL; ++p)
            if (EXACT || gl + p * G < nvec)
                store_vector<VEC>(dest, gl + p * G, finish_row<VEC>(acc[p], epi, scale), pol_stream);
    }
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
struct SpmmArgs {
    const Side *side;
    int n_rows;
    int nnz;
    int sms;         // multiprocessors of the device
    int nvec;
    Gather gather;
    float *Y;
    long long ldy;   // leading dimension of Y in floats
    float *partials;
    unsigned *counter;   // chunk counter of the plan (one word, set to 0 in front of every chunk launch)
    Epilogue epi;
    cudaStream_t st;
    // when set, the short-row kernel is launched on `side_stream` between the two events (fork after what precedes the
    // call on `st`, join before what follows), so that it overlaps the chunk kernels
    cudaStream_t side_stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    int row_class = -1;   // >= 0: only the rows of that class of a plan with row classes
    int resident_per_sm = 0;   // 0: as many blocks of the chunk kernel as fit; > 0: at most this many per SM
};

// The part of a class-major list with class starts `start` that the call computes.
static inline void class_range(int row_class, int n_classes, const int *start, int *lo, int *count) {
    *lo = row_class < 0 ? 0 : start[row_class];
    *count = (row_class < 0 ? start[n_classes] : start[row_class + 1]) - *lo;
}

// Blocks of a kernel that one SM holds at a time (asked once per instantiation) times the SM count of the device.
template <typename Kernel>
static int resident_grid(Kernel kernel, int cap_per_sm) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0) != cudaSuccess) return 0;
    if (cap_per_sm > 0 && per_sm > cap_per_sm) per_sm = cap_per_sm;
    return per_sm * sms;
}

// Batches of a large plan's chunks.  With enough chunks every SM has gathers in flight whatever a warp has, and out of L2 more of them
// a warp only cost registers; out of HBM they pay.  us with four / two / one: F = 8 power law 700,000 rows of 71 354 / 319 / 314, 1.4 M
// of 88 760 / 698 / 679, 2 M of 50 836 / 784 / 716, 700,000 of 21 138 / 137 / 136, 50,000 of 500 143 / 145 / 148, of 1000 237 / 234 /
// 234, R-MAT-19 16 M nonzeros 106 / 109 / 111, R-MAT-18 64 / 75 / 75, R-MAT-23 (X is 268 MB) 923 / 982 / 1008; value-free 2 M of 50 686
// / 645 / 651, 700,000 of 36 177 / 173 / 185, 50,000 of 500 131 / 134 / 142.  F = 4 700,000 of 71 326 / 307 / 306, 1.4 M of 88 688 /
// 669 / 660, 50,000 of 1000 192 / 197 / 194, 200,000 of 250 248 / 253 / 254, of 500 466 / 457 / 458, R-MAT-24 1758 / 1663 / 1697,
// R-MAT-18 66 / 76 / 75; value-free 50,000 of 2000 242 / 252 / 236, 2 M of 50 620 / 601 / 595. Widths of 1 and 2 keep four.
template <int G, int VEC, bool UNIT>
static int large_plan_batches(int nnz, int n_rows) {
    const int most = chunk_batches(G, 1, VEC, false);
    const bool in_l2 = 4LL * G * VEC * n_rows <= 160000000;
    if (VEC == 4 && G == 2) return nnz > (n_rows >= 100000 ? 20000000 : 40000000) && in_l2 ? (UNIT ? 2 : 1) : most;
    if (VEC == 4 && G == 1) return nnz > 64000000 && in_l2 ? 1 : !UNIT && nnz > 20000000 && n_rows >= 400000 ? 2 : most;
    return most;
}

// The same for the one launch of a small plan, where one batch also halves the registers of the whole kernel: for graphs whose rows are
// nearly all long.  us with four (F = 8: two) / one and the short rows as wide shapes have them: F = 1 20,000 rows of 300 29.2 / 26.7,
// 8,000 of 200 9.4 / 10.1, value-free 23.7 / 19.5 and 8.7 / 7.5, 20,000 of 120 13.4 / 13.7; F = 4 12,000 of 480 34.5 / 32.8, 40,000 of
// 150 36.3 / 37.3, 3,000 of 300 7.2 / 8.0, value-free 31.2 / 27.7 and 33.1 / 32.1; F = 8 value-free 12,000 of 480 35.0 / 33.5.  F = 4
// value-free with four / two: 100,000 rows of 60 50.5 / 44.0, 200,000 of 28 47.7 / 42.9, 20,000 of 40 13.2 / 14.6.
template <int G, int VEC, bool UNIT>
static int small_plan_batches(int nnz, int n_rows) {
    if (nnz >= 3 << 19 && (UNIT || G == 1) && nnz / (UNIT ? 140 : 256) >= n_rows) return 1;
    if (VEC == 4 && G == 1 && UNIT && nnz >= 3000000) return 2;
    return chunk_batches(G, 1, VEC, true);
}

template <int G, int VPL, int VEC, int U, bool EXACT, bool UNIT, bool HOT, int NB>
static int launch_chunks(const SpmmArgs &a, int chunk_lo, int n_chunks) {
    const Side &s = *a.side;
    auto kernel = spmm_chunks_kernel<G, VPL, VEC, 2 * U, EXACT, UNIT, HOT, NB>;
    static int resident_all = 0;
    if (resident_all == 0) resident_all = resident_grid(kernel, 0);
    int resident = resident_all;
    if (a.resident_per_sm > 0) resident = std::min(resident, a.resident_per_sm * a.sms);
    int grid = ceil_div(ceil_div(n_chunks, kChunkGroup), 8);
    if (resident > 0 && grid > resident) grid = resident;
    DRONE_CUDA(cudaMemsetAsync(a.counter, 0, sizeof(unsigned), a.st));
    kernel<<<grid, 256, 0, a.st>>>(s.chunks + chunk_lo, n_chunks, s.col, s.val, a.gather, a.Y, a.ldy, a.partials, a.nvec, a.epi, a.counter);
    DRONE_LAUNCH_CHECK("spmm_chunks_kernel");
    return DRONE_OK;
}

template <int G, int VPL, int VEC, int U, bool EXACT, bool UNIT, bool HOT>
static int launch_all(const SpmmArgs &a) {
    constexpr int RPW = 32 / G;
    const Side &s = *a.side;
    int range_lo, n_ranges, chunk_lo, n_chunks, split_lo, n_split, wide_lo, n_wide;
    // Odd widths above 128, one launch / separate kernels, us, power law: F = 131 30,000 rows of 41 89 / 136, 130,000 of 25 261 / 305,
    // of 41 394 / 374, 60,000 of 61 252 / 253; F = 301 60,000 of 41 308 / 336, 130,000 of 25 624 / 606; F = 401 10,000 of 13 39 / 42,
    // 30,000 of 13 87 / 80; F = 601 3,000 of 13 32 / 47, 30,000 of 13 224 / 210.
    const bool one_launch = s.small && (VEC == 4 || a.nnz <= small_nnz_floats(VPL));
    // (Above 512 single floats the line of the separate kernels lies lower; ranges of 16 / 64, us, F = 601: 28,000 rows of 4 62 / 65,
    // 20,000 rows of 7 81 / 74.)
    const long long fine_lanes = one_launch || VPL < 32 ? kFineRangeLanes : 4LL << 20;
    const bool fine = s.fine.row != nullptr && (G <= 2 || (long long)s.n_short_entries * G < fine_lanes);
    const Ranges &ranges = fine ? s.fine : s.ranges;
    class_range(a.row_class, s.n_classes, ranges.start, &range_lo, &n_ranges);
    class_range(a.row_class, s.n_classes, s.chunk_start, &chunk_lo, &n_chunks);
    class_range(a.row_class, s.n_classes, s.split_start, &split_lo, &n_split);
    class_range(a.row_class, s.n_classes, s.wide_start, &wide_lo, &n_wide);
    if (!HOT && one_launch) {
        const int chunk_blocks = ceil_div(n_chunks, 8), short_blocks = ceil_div(n_ranges, 8 * RPW);
        if (chunk_blocks + short_blocks == 0) return DRONE_OK;
        cudaLaunchAttribute early;
        early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        early.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(chunk_blocks + short_blocks);
        cfg.blockDim = dim3(256);
        cfg.stream = a.st;
        cfg.attrs = &early;
        cfg.numAttrs = 1;
        // Chunks want 64 registers, short rows want warps: 48 registers where most nonzeros lie in short rows and these are
        // more than four blocks per SM work on at a time (64 / 48 registers, us: power law, 270,000 rows of 5, F = 32
        // 39 / 30, F = 64 65 / 50; of 17, F = 128 275 / 246; but R-MAT-16 + I, F = 64, three quarters in chunks: 29 / 38, and
        // 120,000 rows of 5, F = 64, one wave: 22 / 25).
        auto kernel = spmm_small_kernel<G, VPL, VEC, U, EXACT, UNIT, 0>;
        if constexpr (VEC == 4 && VPL == 1 && G >= 4 && EXACT) {
            if (short_blocks > a.sms * 4 && s.n_short_entries >= a.nnz / 2) kernel = spmm_small_kernel<G, VPL, VEC, U, EXACT, UNIT, 5>;
        }
        // On the smallest plans the chunks of F = 65 to 128 are quicker with a test per vector (without / with, us, F = 95: 10,000
        // rows of 81 39 / 37, 30,000 rows of 41 53 / 60, 250,000 of 7 130 / 153).
        if constexpr (VEC == 1 && VPL == 4 && sure_vectors(G, VPL, VEC) > 0) {
            if (a.nnz < 1 << 20) kernel = spmm_small_kernel<G, VPL, VEC, U, EXACT, UNIT, 0, 0>;
        }
        if constexpr (chunk_batches(G, VPL, VEC, true) > 1 && (UNIT || G == 1)) {
            const int batches = small_plan_batches<G, VEC, UNIT>(a.nnz, a.n_rows);
            if (batches == 1) kernel = spmm_small_kernel<G, VPL, VEC, U, EXACT, UNIT, 0, sure_vectors(G, VPL, VEC), 1>;
            if constexpr (VEC == 4 && G == 1 && UNIT) {
                if (batches == 2) kernel = spmm_small_kernel<G, VPL, VEC, U, EXACT, UNIT, 0, sure_vectors(G, VPL, VEC), 2>;
            }
        }
        DRONE_CUDA(cudaLaunchKernelEx(&cfg, kernel, (const Chunk *)s.chunks + chunk_lo, n_chunks,
                                      chunk_blocks, (const int *)s.col, (const float *)s.val, (const SplitRow *)s.split,
                                      (const int *)s.slot_split, s.arrived, a.partials, (const int *)ranges.row + range_lo,
                                      n_ranges, (const int *)s.s_rowptr, (const int *)s.s_rows, (const int *)s.s_col,
                                      (const float *)s.s_val, a.gather, a.Y, a.ldy, a.nvec, a.epi));
        count_launch();
        return DRONE_OK;
    }
    if (HOT && a.gather.hot_rows > 0) {
        const long long total = (long long)a.gather.hot_rows * a.nvec;
        const int grid = (int)std::min<long long>((total + 255) / 256, 148 * 16);
        spmm_fill_hot_kernel<VEC><<<grid, 256, 0, a.st>>>(a.gather.hot_ids, a.gather.hot_rows, a.gather.X, a.gather.ldv,
                                                         a.nvec, const_cast<float *>(a.gather.hot));
        DRONE_LAUNCH_CHECK("spmm_fill_hot_kernel");
    }
    const bool overlap = a.side_stream != nullptr && n_ranges > 0 && n_chunks > 0;
    if (n_ranges > 0) {
        cudaStream_t short_stream = a.st;
        if (overlap) {
            DRONE_CUDA(cudaEventRecord(a.fork, a.st));
            DRONE_CUDA(cudaStreamWaitEvent(a.side_stream, a.fork, 0));
            short_stream = a.side_stream;
        }
        const int grid = ceil_div(n_ranges, 8 * RPW);
        spmm_short_stream_kernel<G, VPL, VEC, U, EXACT, UNIT, HOT><<<grid, 256, 0, short_stream>>>(
            ranges.row + range_lo, n_ranges, s.s_rowptr, s.s_rows, s.s_col, s.s_val, a.gather, a.Y, a.ldy, a.nvec, a.epi);
        DRONE_LAUNCH_CHECK("spmm_short_stream_kernel");
        if (overlap) DRONE_CUDA(cudaEventRecord(a.join, a.side_stream));
    }
    if (n_chunks > 0) {
        constexpr int MOST = chunk_batches(G, VPL, VEC, false);
        auto launch = launch_chunks<G, VPL, VEC, U, EXACT, UNIT, HOT, MOST>;
        if constexpr (MOST > 1 && VEC == 4) {
            const int batches = large_plan_batches<G, VEC, UNIT>(a.nnz, a.n_rows);
            if constexpr (G == 1 || !UNIT) {
                if (batches == 1) launch = launch_chunks<G, VPL, VEC, U, EXACT, UNIT, HOT, 1>;
            }
            if constexpr ((G == 2) == UNIT) {
                if (batches == 2) launch = launch_chunks<G, VPL, VEC, U, EXACT, UNIT, HOT, 2>;
            }
        }
        const int rc = launch(a, chunk_lo, n_chunks);
        if (rc) return rc;
    }
    if (n_split > 0) {
        const size_t smem = n_wide > 0 ? sizeof(float) * 8 * (size_t)a.nvec * VEC : 0;
        spmm_reduce_partials_kernel<G, VPL, VEC><<<n_wide + ceil_div(n_split, 8), 256, smem, a.st>>>(
            s.split + split_lo, n_split, s.wide + wide_lo, n_wide, a.partials, a.Y, a.ldy, a.nvec, a.epi);
        DRONE_LAUNCH_CHECK("spmm_reduce_partials_kernel");
    }
    if (overlap) DRONE_CUDA(cudaStreamWaitEvent(a.st, a.join, 0));
    return DRONE_OK;
}

template <int G, int VPL, int VEC, int U, bool UNIT, bool HOT>
static int launch_exact(const SpmmArgs &a) {
    return a.nvec == G * VPL ? launch_all<G, VPL, VEC, U, true, UNIT, HOT>(a) : launch_all<G, VPL, VEC, U, false, UNIT, HOT>(a);
}

// Entries of a translation unit: pick the lane-group shape for the width (nvec vectors of four floats, or floats, per row).
template <bool UNIT, bool HOT>
static int dispatch_vectors(const SpmmArgs &a) {
    const int nv = a.nvec;
    if (nv <= 1) return launch_exact<1, 1, 4, 4, UNIT, HOT>(a);
    if (nv <= 2) return launch_exact<2, 1, 4, 4, UNIT, HOT>(a);
    if (nv <= 4) return launch_exact<4, 1, 4, 4, UNIT, HOT>(a);
    if (nv <= 8) return launch_exact<8, 1, 4, 4, UNIT, HOT>(a);
    if (nv <= 16) return launch_exact<16, 1, 4, 4, UNIT, HOT>(a);
    if (nv <= 32) return launch_exact<32, 1, 4, 4, UNIT, HOT>(a);
    if (nv <= 64) return launch_exact<32, 2, 4, 2, UNIT, HOT>(a);
    if (nv <= 96) return launch_exact<32, 3, 4, 2, UNIT, HOT>(a);
    if (nv <= 128) return launch_exact<32, 4, 4, 1, UNIT, HOT>(a);
    if (nv <= 256) return launch_exact<32, 8, 4, 1, UNIT, HOT>(a);
    return set_error(DRONE_E_INVALID, "drone_spmm: feature width %d is above 1024", nv * 4);
}

// Rows that are read float by float: widths below 4, and wider ones for which there is no padded copy.  The latter take
// the lane groups the padded copy would (four floats for every vector of a lane), so that a row's nonzeros are added
// in the same order and the result has the same bits by either route.
template <bool UNIT, bool HOT>
static int dispatch_floats(const SpmmArgs &a) {
    const int f = a.nvec, nv = (f + 3) / 4;
    if (f <= 1) return launch_all<1, 1, 1, 4, true, UNIT, HOT>(a);
    if (f <= 2) return launch_all<2, 1, 1, 4, true, UNIT, HOT>(a);
    if (f <= 4) return launch_all<4, 1, 1, 4, false, UNIT, HOT>(a);
    if (f <= 8 && !a.side->small) return launch_all<8, 1, 1, 4, false, UNIT, HOT>(a);
    if (nv <= 2) return launch_all<2, 4, 1, 2, false, UNIT, HOT>(a);
    if (nv <= 4) return launch_all<4, 4, 1, 2, false, UNIT, HOT>(a);
    if (nv <= 8) return launch_all<8, 4, 1, 2, false, UNIT, HOT>(a);
    if (nv <= 16) return launch_all<16, 4, 1, 2, false, UNIT, HOT>(a);
    if (nv <= 32) return launch_all<32, 4, 1, 2, false, UNIT, HOT>(a);
    if (nv <= 64) return launch_all<32, 8, 1, 1, false, UNIT, HOT>(a);
    if (nv <= 96) return launch_all<32, 12, 1, 1, false, UNIT, HOT>(a);
    if (nv <= 128) return launch_all<32, 16, 1, 1, false, UNIT, HOT>(a);
    if (nv <= 256) return launch_all<32, 32, 1, 1, false, UNIT, HOT>(a);
    return set_error(DRONE_E_INVALID, "drone_spmm: feature width %d is above 1024", f);
}

// The four combinations, each defined in a translation unit of its own (spmm_variants_*.cu).
int spmm_dispatch_plain(const SpmmArgs &a, bool vec4);
int spmm_dispatch_unit(const SpmmArgs &a, bool vec4);
int spmm_dispatch_hot(const SpmmArgs &a, bool vec4);
int spmm_dispatch_unit_hot(const SpmmArgs &a, bool vec4);

}  // namespace drone
