// Host side of the aggregation: argument checks, column slicing, the choice of kernel variant and the entry points
// of the C ABI.  The kernels are in spmm_kernels.cuh, compiled once per variant in spmm_variants_*.cu.
#include "spmm_kernels.cuh"
#include "exchange.cuh"

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <new>

namespace drone {

// in_scale[i] = 1/sqrt(inDegree[i]), out_scale[i] = 1/sqrt(outDegree[i]) (0 for a degree of 0): the two factors of the
// reference's edge coefficient 1/sqrt(outDegree[u] * inDegree[v]).
__global__ void degree_scales_kernel(const int *__restrict__ in_deg, const int *__restrict__ out_deg, int n,
                                     float *__restrict__ in_scale, float *__restrict__ out_scale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    in_scale[i] = in_deg[i] > 0 ? (float)(1.0 / sqrt((double)in_deg[i])) : 0.f;
    out_scale[i] = out_deg[i] > 0 ? (float)(1.0 / sqrt((double)out_deg[i])) : 0.f;
}

// padded[r, 0:F] = X[r, 0:F], padded[r, F:Fp] = 0          (Fp = F rounded up to a multiple of 4; rows `stride` floats apart)
__global__ void pad_rows_kernel(const float *__restrict__ X, long long ldx, int n_rows, int F, int nvec, int stride,
                                float *__restrict__ padded) {
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (RowColumn at(first, step, nvec); at.row < n_rows; at.advance()) {
        const float *x = X + (long long)at.row * ldx + 4 * at.col;
        const int left = F - 4 * at.col;
        float4 v;
        v.x = left > 0 ? __ldg(x) : 0.f;
        v.y = left > 1 ? __ldg(x + 1) : 0.f;
        v.z = left > 2 ? __ldg(x + 2) : 0.f;
        v.w = left > 3 ? __ldg(x + 3) : 0.f;
        *reinterpret_cast<float4 *>(padded + (long long)at.row * stride + 4 * at.col) = v;
    }
}

// Y[row, 0:F] = padded[row, 0:F] for the rows of `rows` (rows == NULL: rows 0..n_rows-1)
__global__ void unpad_rows_kernel(const float *__restrict__ padded, int Fp, const int *__restrict__ rows, int n_rows, int F,
                                  float *__restrict__ Y, long long ldy) {
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (RowColumn at(first, step, F); at.row < n_rows; at.advance()) {
        const int r = rows ? __ldg(rows + at.row) : at.row;
        Y[(long long)r * ldy + at.col] = __ldcs(padded + (long long)r * Fp + at.col);
    }
}

// Whether work put on this stream runs now; otherwise (or where the stream does not say) it becomes part of a graph, and nothing
// may be allocated.
static bool runs_now(cudaStream_t st) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &status) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return status == cudaStreamCaptureStatusNone;
}

// A buffer that has been replaced is freed, unless a captured graph uses it.
static void give_back_replaced(drone_plan *p, float *buffer, bool *captured) {
    if (!*captured) {
        cudaFree(buffer);
        return;
    }
    *captured = false;
    drone_plan::Kept *k = new (std::nothrow) drone_plan::Kept{buffer, p->kept};
    if (k) p->kept = k;      // else it outlives the plan
}

static int ensure_scratch(drone_plan *p, size_t bytes) {
    if (bytes <= p->scratch_bytes) return DRONE_OK;
    // grow: frees and reallocates, so earlier calls that use the scratch must have finished
    DRONE_CUDA(cudaDeviceSynchronize());
    give_back_replaced(p, p->scratch, &p->scratch_captured);
    p->scratch = nullptr;
    p->scratch_bytes = 0;
    DRONE_CUDA(cudaMalloc(&p->scratch, bytes));
    p->scratch_bytes = bytes;
    return DRONE_OK;
}

// Floats between the rows of a padded copy.  A row that starts on a 128-byte line is read with one line less than one
// that starts anywhere, and the gathers pay per line (Reddit-shaped, F = 41: 2.42 ms float by float, 1.70 copied to rows 44 apart, 1.52 to rows 64 apart), so rows wider than half a
// line start on a line and shorter ones do not straddle one, as long as the copy then still fits the part of L2 the
// gathers can count on; larger copies, whose rows come from HBM, start on the 64 bytes HBM delivers.
static long long padded_stride(int n_rows, int F) {
    const long long fp = (F + 3) & ~3;
    long long lines = 4;
    while (lines < fp && lines < 32) lines *= 2;
    if (lines < fp) lines = (fp + 31) / 32 * 32;
    if ((double)n_rows * lines * 4 <= 64e6) return lines;
    return (fp + 15) / 16 * 16;
}

// The same for a call that runs in column slices, each of which then starts on a line (slices_by_counts).
static long long line_stride(int F) { return (F + 31) / 32 * 32; }
// Nobody asked for that copy: it stays below half a gigabyte.
static bool lines_fit(int n_rows, int F) { return line_stride(F) * n_rows <= 1 << 27; }

// The copies' buffers.  drone_plan_reserve makes them ahead of time; otherwise the first call that wants them does, unless
// that call must not allocate (its width was reserved without them, the stream is being captured), they would take more
// than kPadBytes nobody asked for, or so much did not fit before: the next drone_plan_reserve tries again.
constexpr size_t kPadBytes = (size_t)4 << 30;

// Floats of new memory that buffers of these sizes (0: not needed) take.
static size_t padding_to_make(const drone_plan *p, size_t x_floats, size_t y_floats) {
    return (x_floats > p->pad_x_floats ? x_floats : 0) + (y_floats > p->pad_y_floats ? y_floats : 0);
}

// What is there stays until its replacement exists, so that a failure costs nothing that was reserved before.
static int ensure_padding(drone_plan *p, size_t x_floats, size_t y_floats) {
    const bool new_x = x_floats > p->pad_x_floats, new_y = y_floats > p->pad_y_floats;
    if (!new_x && !new_y) return DRONE_OK;
    float *x = nullptr, *y = nullptr;
    cudaError_t e = new_x ? cudaMalloc(&x, sizeof(float) * x_floats) : cudaSuccess;
    if (e == cudaSuccess && new_y) e = cudaMalloc(&y, sizeof(float) * y_floats);
    if (e != cudaSuccess) {
        cudaFree(x);
        return set_error(DRONE_E_CUDA, "no memory for copies with padded rows (%zu bytes): %s",
                         sizeof(float) * padding_to_make(p, x_floats, y_floats), cudaGetErrorString(e));
    }
    if ((new_x && p->pad_x) || (new_y && p->pad_y)) cudaDeviceSynchronize();      // calls in flight use what is replaced
    if (new_x) {
        give_back_replaced(p, p->pad_x, &p->pad_x_captured);
        p->pad_x = x;
        p->pad_x_floats = x_floats;
    }
    if (new_y) {
        give_back_replaced(p, p->pad_y, &p->pad_y_captured);
        p->pad_y = y;
        p->pad_y_floats = y_floats;
    }
    return DRONE_OK;
}

// drone_plan_reserve's form: where old and new buffers do not fit together the old ones go first (unless a graph uses them), and
// come back if the new ones do not fit alone either.
static int replace_padding(drone_plan *p, size_t x_floats, size_t y_floats) {
    p->pad_refused_bytes = ~(size_t)0;
    if (ensure_padding(p, x_floats, y_floats) == DRONE_OK) return DRONE_OK;
    const size_t old_x = p->pad_x_floats, old_y = p->pad_y_floats;
    if (old_x + old_y == 0 || p->pad_x_captured || p->pad_y_captured) return DRONE_E_CUDA;
    DRONE_CUDA(cudaDeviceSynchronize());
    cudaFree(p->pad_x);
    cudaFree(p->pad_y);
    p->pad_x = p->pad_y = nullptr;
    p->pad_x_floats = p->pad_y_floats = 0;
    if (ensure_padding(p, std::max(x_floats, old_x), std::max(y_floats, old_y)) == DRONE_OK) return DRONE_OK;
    char message[512];
    snprintf(message, sizeof(message), "%s", last_error_buffer());
    ensure_padding(p, old_x, old_y);
    return set_error(DRONE_E_CUDA, "%s", message);
}

// The copies are passes over [n, F]; what they save is in the gathers, so the line lies at a number of nonzeros per row, and
// further out where the uncopied call is the one launch of a small plan.  us float by float / copied, power-law graphs:
//   F = 13, 270,000 rows of 9, 17, 33: 57 / 52, 94 / 76, 139 / 113; F = 63, rows of 33: 40,000 52 / 52, 250,000 266 / 239;
//   Reddit-shaped (491 a row), F = 41: 2410 / 1512; R-MAT-22 (17 a row), F = 41: 1710 / 2175.
//   F = 95 and 127, rows of 33: 90,000 122 / 149 and 130 / 159, 250,000 (above kSmallNnz) 440 / 408 and 543 / 493.
//   F = 131 and 255: in one launch 40,000 rows of 13 52 / 66 and 58 / 82, 30,000 rows of 41 89 / 111 and 99 / 115,
//   60,000 rows of 61 252 / 304 and 308 / 310; above kSmallNnz (130,000 rows of 61) 514 / 482 and 952 / 824.
//   F = 301, rows of 81: 10,000 (one launch) 82 / 101, 60,000 561 / 534.  F = 401, 10,000 rows of 13 (one launch) and 19: 39 / 47
//   and 79 / 54.  F = 511, 60,000 rows of 41 and 81: 531 / 486 and 1050 / 755.  F = 601, rows of 81: 60,000 3301 / 4111, 90,000
//   4961 / 2536.
// Copies whose rows are a whole number of 128-float steps run on kernels without a test per vector and pay off sooner.
static bool worth_copying(const drone_plan *p, int F) {
    const double per_row = (double)p->nnz / p->n_rows, bytes = (double)p->n_rows * F * 4;
    const bool many = p->nnz > kSmallNnz;
    if (F <= 64) return p->nnz >= 1 << 20 && per_row >= (F <= 32 ? 16 : 32);
    if (F <= 128) return many && per_row >= 32;
    const bool whole_steps = ((F + 3) & ~3) % 128 == 0;
    if (F <= 256 && !many) return whole_steps && per_row >= 60;
    if (F <= 384 && p->nnz <= small_nnz_floats(12)) return false;
    if (F <= 512 && p->nnz <= small_nnz_floats(16)) return false;
    if (whole_steps && per_row >= 60) return true;
    if (per_row >= 64) return many || F <= 512 || bytes <= 100e6;
    return F > 384 && per_row >= 12 && bytes <= 40e6;
}

constexpr int kSliceFloats = 64;
constexpr double kL2Floats = 25e6;      // of gathered rows that L2 keeps

// How the columns of a call are cut.
struct Slices {
    int width = 0;             // 0: in one piece
    bool long_last = false;    // what is left of less than a slice goes with the slice before it
    bool by_counts = false;    // by the operand as well: another call of this width may run in one piece
    // Widths that were forced or fit L2 divide the columns; of the others a short rest goes with the slice before it.
    int next(int left) const {
        const int rest = !by_counts ? 1 : long_last ? width : kSliceFloats / 4;
        return width == 0 || left < width + rest ? left : width;
    }
    // Columns that partial sums are kept for: calls of a width leave room for each other, so that one of them can be captured.
    int partial_columns(int F) const { return width == 0 || by_counts ? F : width; }
};

// Slices of 64 columns where not even a slice fits L2: by the share of the gathers that go to the rows L2 can keep (GatherCounts), at
// the rates of gathers out of HBM and out of L2.  Graphs without popular rows gain most: of 300,000 rows of 1 KB L2 keeps a third, of
// their slices all.  R-MAT graphs, whose popular rows are in L2 at any width, keep calls in one piece (from a third of the gathers
// missing on; R-MAT-20 F = 256 in one piece / slices 2085 / 2297 us, R-MAT-22 F = 128 2688 / 2861).  Power law, us in one piece /
// slices: 300,000 rows of 201 F = 256 5908 / 3997, F = 512 14202 / 8627; 400,000 of 61 F = 256 2976 / 1989; 600,000 of 101 F = 128
// 3186 / 2532, F = 512 16370 / 11643; 150,000 of 37 F = 512 1370 / 1097; 1.2 M of 101 F = 256 16403 / 13709; 2.4 M of 51 F = 256 18120 /
// 17350.  Rows below 24 nonzeros lose: 2.4 M of 17 F = 128 3072 / 3194.  So do slices that do not start on 128-byte lines (2.4 M of 51
// F = 180 15246 / 18470), and rows read float by float (600,000 of 31 F = 177 2178 / 2605).
// A rest of 32 columns is read out of HBM at 5 TB/s instead of 7: where more than half of a slice's gathers miss, it stays with the
// slice before it (2.4 M of 51, F = 224: in one piece 16389, 3 x 64 + 32 17001).
// copied: X has to be copied for it, at 3 TB/s; the slices then have to save a tenth (600,000 rows of 31, F = 232 2556 / 2294, F = 300
// 3240 / 3172).
static Slices slices_by_counts(const drone_plan *p, const Side &s, int F, bool copied) {
    Slices cut;
    if (!s.counted || !slices_possible(p->n_rows, p->nnz) || F < 2 * kSliceFloats) return cut;
    const double hbm = 7, l2 = 17, stream = 6.5, copying = 3;      // TB/s
    const auto picoseconds = [&](int width, double missed) { return 4.0 * width * (missed / hbm + (1 - missed) / l2) + 8 / stream; };
    const double missed = 1 - s.counts.share(kL2Floats / F), in_slice = 1 - s.counts.share(kL2Floats / kSliceFloats);
    const double sliced = picoseconds(kSliceFloats, in_slice) * F / kSliceFloats + (copied ? 8.0 * F / copying * p->n_rows / p->nnz : 0);
    if (missed < 0.35 || sliced > (copied ? 0.9 : 0.95) * picoseconds(F, missed)) return cut;
    cut.width = kSliceFloats;
    cut.by_counts = true;
    cut.long_last = in_slice > 0.5;
    return cut;
}

constexpr double kL2Budget = 64e6;                      // about half of the 126 MB L2 for the gathered operand

// Columns of a slice that fits L2 (0: none does).
static int slices_that_fit(const drone_plan *p, int F) {
    for (int w : {128, 64})
        if (w < F && F % w == 0 && (double)p->n_rows * w * 4 <= kL2Budget) return w;
    return 0;
}

static bool rows_on_lines(const float *X, long long ldx) { return ldx % 32 == 0 && (reinterpret_cast<uintptr_t>(X) & 127) == 0; }

// Column slices of a call.  Gathering a slice of w columns touches only
// n*w*4 bytes of X; when the whole operand does not fit in L2 but a slice does, running the slices one after the
// other turns HBM gathers into L2 gathers at the price of re-reading the CSR stream once per slice.
// on_lines: the rows of X start on 128-byte lines.
static Slices column_slices(const drone_plan *p, const Side &s, int F, bool vec4, bool on_lines) {
    Slices cut;
    const int forced = p->slice_forced;
    if (forced == 0 || !vec4) return cut;
    if (forced > 0) {
        if (forced % 4 == 0 && forced < F && F % forced == 0) cut.width = forced;
        return cut;
    }
    if (p->hot_table) return cut;                       // tagged plan: the hot rows are kept in L2 by their table
    if ((double)p->n_rows * F * 4 <= kL2Budget) return cut;
    cut.width = slices_that_fit(p, F);
    if (cut.width > 0) return cut;
    return on_lines ? slices_by_counts(p, s, F, false) : cut;
}

// Whether rows of F floats, ld apart from base, can be accessed 16 bytes at a time.
static bool rows_of_vectors(int F, long long ld, const float *base) {
    return F % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(base) & 15) == 0;
}

// Whether X is to be copied to rows on lines for the slices of a call (where there is room, spmm_impl).  Power law, us in one
// piece / in slices of X where it lies / of the copy: 300,000 rows of 201 F = 180 4075 / 3455 / 2698, F = 300 7928 / 6025 / 4552; 300,000
// of 41 F = 180 1151 / 1041 / 937, F = 392 3171 / 2188 / 2167; 600,000 of 101 F = 152 4693 / 4872 / 3713, F = 180 5739 / 5878 / 4027;
// 690,000 of 121 F = 180 8133 / 8651 / 5742; 180,000 of 101 F = 500 4152 / 2624 / 2517.  A plan that was reserved for the width without
// the copies keeps its calls in one piece.
static bool copy_x_for_slices(const drone_plan *p, const Side &s, int F, const float *X, long long ldx) {
    if (p->slice_forced >= 0 || p->hot_table || rows_on_lines(X, ldx) || slices_that_fit(p, F) > 0) return false;
    if (F <= p->reserved_features && F > p->reserved_copies) return false;
    return lines_fit(p->n_rows, F) && slices_by_counts(p, s, F, true).width > 0;
}

// What a call may ask for beyond the plain product (drone_spmm_opts of the C ABI, already checked).
struct CallOptions {
    int row_class = -1;
    bool unit_values = false;
    Epilogue epi;
    drone_xplan *push_up_to = nullptr;   // the call also sends the mirror rows of Y to their owners
    bool no_allocation = false;
};

// One launch sequence over columns [0, width) of the operands a.gather.X / a.Y point at.
static int run_variant(const drone_plan *p, const Side &s, SpmmArgs &a, bool vec4, int width, bool unit_values) {
    if (vec4) {
        a.nvec = width / 4;
    } else {
        a.nvec = width;
    }
    const bool tagged = s.hot_ids != nullptr;
    if (tagged) {
        // rows of the table at this width; positions beyond it fall back to X through hot_ids
        const long long fit = (long long)(p->hot_table_bytes / (sizeof(float) * (size_t)width));
        a.gather.hot = p->hot_table;
        a.gather.hot_ids = s.hot_ids;
        a.gather.hot_rows = (int)std::min<long long>(fit, s.n_hot);
        return unit_values ? spmm_dispatch_unit_hot(a, vec4) : spmm_dispatch_hot(a, vec4);
    }
    return unit_values ? spmm_dispatch_unit(a, vec4) : spmm_dispatch_plain(a, vec4);
}

static int spmm_impl(drone_plan *p, int orientation, int F, const float *X, long long ldx, float *Y,
                     long long ldy, cudaStream_t st, const CallOptions &opt = CallOptions()) {
    const Side &s = p->side[orientation];
    if (p->n_rows == 0) return DRONE_OK;
    // Operands whose rows cannot be accessed as float4 where they lie are copied to where they can (X before the kernels,
    // Y after them), where that is worth it; also an X whose rows could, but do not start on lines, for a call that then runs in
    // slices.
    float *const caller_Y = Y;
    const long long caller_ldy = ldy;
    const int caller_F = F, Fp = (F + 3) & ~3;
    const bool x_vectors = rows_of_vectors(F, ldx, X), y_vectors = rows_of_vectors(F, ldy, Y);
    bool vec4 = x_vectors && y_vectors;
    const bool to_vectors = !vec4 && F > 8 && worth_copying(p, F), to_lines = vec4 && copy_x_for_slices(p, s, F, X, ldx);
    bool copy_x = to_lines || (to_vectors && !x_vectors), copy_y = to_vectors && !y_vectors;
    const long long stride = to_lines ? line_stride(F) : padded_stride(p->n_rows, F);
    // The columns are cut as for the copies also where these have no room, or are left out: a row class, a call under capture and
    // one that found no memory add in the order of the whole, eager call.  Read float by float the slices mostly lose what they cost
    // (us in one piece / in slices: 600,000 rows of 81 F = 177 5160 / 5740, a million of 64 F = 255 10650 / 12450, 300,000 of 201 F = 255 7600 /
    // 6750), on plans that were reserved for an odd width without the copies.
    const Slices cut = column_slices(p, s, Fp, vec4 || to_vectors, copy_x ? stride % 32 == 0 : rows_on_lines(X, ldx));
    // Every class of rows copies X anew, which a small class does not make up for (us for all classes, 2 / 4 / 16 equal ones, X where
    // it lies against copied: 300,000 rows of 201 F = 180 4035 / 4161 / 6665 and 3312 / 3547 / 6878, of 41 F = 392 2462 / 3005 / 6443 and
    // 2549 / 3432 / 8751, 690,000 of 121 F = 180 9156 / 9550 / 11661 and 6974 / 7257 / 11632).
    if (to_lines && opt.row_class >= 0 && p->n_classes > 1 &&
        (p->class_start[opt.row_class + 1] - p->class_start[opt.row_class]) < p->n_rows / 8)
        copy_x = false;
    // Room for the copies: there, or made by this call.
    const auto room_for = [&](size_t x_floats, size_t y_floats) {
        const size_t missing = sizeof(float) * padding_to_make(p, x_floats, y_floats);
        if (missing == 0) return true;
        if (opt.no_allocation || caller_F <= p->reserved_features || missing >= p->pad_refused_bytes ||
            sizeof(float) * (std::max(x_floats, p->pad_x_floats) + std::max(y_floats, p->pad_y_floats)) > kPadBytes || !runs_now(st))
            return false;
        if (ensure_padding(p, x_floats, y_floats) == DRONE_OK) return true;
        p->pad_refused_bytes = missing;      // the call does without, from now on without asking again
        return false;
    };
    const size_t rows = (size_t)p->n_rows;
    if ((copy_x || copy_y) && room_for(copy_x ? (size_t)stride * rows : 0, copy_y ? (size_t)Fp * rows : 0)) {
        if (!runs_now(st)) {
            p->pad_x_captured |= copy_x;
            p->pad_y_captured |= copy_y;
        }
        if (copy_x) {
            const long long total = (long long)p->n_rows * (Fp / 4);
            pad_rows_kernel<<<(int)std::min<long long>((total + 255) / 256, 148 * 16), 256, 0, st>>>(X, ldx, p->n_rows, F, Fp / 4,
                                                                                                    (int)stride, p->pad_x);
            DRONE_LAUNCH_CHECK("pad_rows_kernel");
            X = p->pad_x;
            ldx = stride;
        }
        if (copy_y) {
            Y = p->pad_y;
            ldy = Fp;
        }
        vec4 = true;
        F = Fp;
    } else {
        copy_x = copy_y = false;
    }
    // The upward half of the exchange inside this call: the kernels store mirror rows into their owners' memory
    // (rows read as float4 where they lie), or the copy kernel sends them afterwards (any other layout).
    bool routed = false, send_after = false;
    const int2 *route = nullptr;
    float *const *peer_rows = nullptr;
    if (opt.push_up_to) {
        const int rc = p2p_route_begin(opt.push_up_to, p->n_rows, caller_F, &route, &peer_rows);
        if (rc) return rc;
        routed = route != nullptr && vec4 && !copy_y;
        send_after = route != nullptr && !routed;
    }
    p->last_slice_width = cut.width;
    if (s.n_partials > 0) {
        const int rc = ensure_scratch(p, sizeof(float) * (size_t)s.n_partials * (size_t)cut.partial_columns(F));
        if (rc) return rc;
        if (!opt.no_allocation && !p->scratch_captured) p->scratch_captured = !runs_now(st);      // else it is not the plan's
    }
    SpmmArgs a;
    a.side = &s;
    a.n_rows = p->n_rows;
    a.nnz = p->nnz;
    a.sms = p->sms;
    a.ldy = ldy;
    a.partials = p->scratch;
    a.counter = p->counter;
    a.epi = opt.epi;
    a.st = st;
    a.side_stream = p->side_stream;
    a.fork = p->fork_event;
    a.join = p->join_event;
    a.row_class = opt.row_class;
    a.resident_per_sm = p->chunk_blocks_per_sm;
    a.gather.ldv = vec4 ? ldx / 4 : ldx;
    if (routed) {
        a.epi.route = route;
        a.epi.peer_rows = peer_rows;
        a.epi.route_nvec = F / 4;
    }
    for (int c0 = 0, now; c0 < F; c0 += now) {
        now = cut.next(Fp - c0);
        a.gather.X = X + c0;
        a.Y = Y + c0;
        a.epi.route_col0 = c0 / 4;
        const int rc = run_variant(p, s, a, vec4, std::min(now, F - c0), opt.unit_values);
        if (rc) return rc;
    }
    if (routed) {
        const int rc = p2p_route_publish(opt.push_up_to, st);
        if (rc) return rc;
    }
    if (copy_y) {
        const int *rows = nullptr;
        int n_out = p->n_rows;
        if (opt.row_class >= 0 && p->row_order) {      // only the rows this call computed
            rows = p->row_order + p->class_start[opt.row_class];
            n_out = p->class_start[opt.row_class + 1] - p->class_start[opt.row_class];
        }
        if (n_out > 0) {
            const long long total = (long long)n_out * caller_F;
            unpad_rows_kernel<<<(int)std::min<long long>((total + 255) / 256, 148 * 16), 256, 0, st>>>(
                p->pad_y, F, rows, n_out, caller_F, caller_Y, caller_ldy);
            DRONE_LAUNCH_CHECK("unpad_rows_kernel");
        }
    }
    if (send_after) return p2p_push_up(opt.push_up_to, caller_Y, caller_F, (int)caller_ldy, st);
    return DRONE_OK;
}

}  // namespace drone

using namespace drone;

extern "C" {

int drone_spmm(drone_plan *p, int orientation, int F, const float *d_X, int ldx, float *d_Y, int ldy,
               void *stream) {
    DRONE_REQUIRE(p != nullptr, "drone_spmm: plan is NULL");
    DRONE_REQUIRE(orientation == DRONE_OP_A || orientation == DRONE_OP_AT, "drone_spmm: orientation=%d", orientation);
    DRONE_REQUIRE(p->side[orientation].ready, "drone_spmm: orientation %d was not prepared by drone_plan_create",
                  orientation);
    DRONE_REQUIRE(F >= 1 && F <= 1024, "drone_spmm: feature width F=%d outside 1..1024", F);
    DRONE_REQUIRE(ldx >= F && ldy >= F, "drone_spmm: leading dimensions (ldx=%d, ldy=%d) below F=%d", ldx, ldy, F);
    if (p->n_rows == 0) return DRONE_OK;
    DRONE_REQUIRE(d_X && d_Y, "drone_spmm: NULL operand");
    DRONE_REQUIRE(d_X != d_Y, "drone_spmm: X and Y must not alias");
    OnDevice guard;
    const int rc = guard.enter(p->device);
    if (rc) return rc;
    return spmm_impl(p, orientation, F, d_X, ldx, d_Y, ldy, (cudaStream_t)stream);
}

int drone_spmm_ex(drone_plan *p, int orientation, int F, const float *d_X, int ldx, float *d_Y, int ldy,
                  const drone_spmm_opts *opts, void *stream) {
    DRONE_REQUIRE(p != nullptr, "drone_spmm_ex: plan is NULL");
    DRONE_REQUIRE(orientation == DRONE_OP_A || orientation == DRONE_OP_AT, "drone_spmm_ex: orientation=%d", orientation);
    DRONE_REQUIRE(p->side[orientation].ready, "drone_spmm_ex: orientation %d was not prepared by drone_plan_create",
                  orientation);
    DRONE_REQUIRE(F >= 1 && F <= 1024, "drone_spmm_ex: feature width F=%d outside 1..1024", F);
    DRONE_REQUIRE(ldx >= F && ldy >= F, "drone_spmm_ex: leading dimensions (ldx=%d, ldy=%d) below F=%d", ldx, ldy, F);
    CallOptions opt;
    if (opts) {
        DRONE_REQUIRE(opts->epilogue == DRONE_EPILOGUE_NONE || opts->epilogue == DRONE_EPILOGUE_RELU,
                      "drone_spmm_ex: epilogue=%d is not a DRONE_EPILOGUE_* value", opts->epilogue);
        DRONE_REQUIRE(opts->row_class >= -1 && opts->row_class < p->n_classes,
                      "drone_spmm_ex: row_class=%d, the plan has %d classes", opts->row_class, p->n_classes);
        DRONE_REQUIRE(opts->unit_values == 0 || opts->unit_values == 1, "drone_spmm_ex: unit_values=%d is not 0 or 1",
                      opts->unit_values);
        opt.row_class = opts->row_class;
        opt.unit_values = opts->unit_values == 1;
        opt.epi.relu = opts->epilogue == DRONE_EPILOGUE_RELU;
        opt.epi.row_scale = opts->d_row_scale;
        opt.push_up_to = opts->push_up_to;
        DRONE_REQUIRE(!(opt.push_up_to && opt.epi.relu),
                      "drone_spmm_ex: DRONE_EPILOGUE_RELU cannot be combined with push_up_to (the sum over the replicas comes first)");
    }
    if (p->n_rows == 0) {
        if (opt.push_up_to) {      // a rank without rows still takes part in the exchange that follows
            const int2 *route = nullptr;
            float *const *peer_rows = nullptr;
            return p2p_route_begin(opt.push_up_to, 0, F, &route, &peer_rows);
        }
        return DRONE_OK;
    }
    DRONE_REQUIRE(d_X && d_Y, "drone_spmm_ex: NULL operand");
    DRONE_REQUIRE(d_X != d_Y, "drone_spmm_ex: X and Y must not alias");
    OnDevice guard;
    int rc = guard.enter(p->device);
    if (rc) return rc;
    return spmm_impl(p, orientation, F, d_X, ldx, d_Y, ldy, (cudaStream_t)stream, opt);
}

int drone_degree_scales(const int *d_in_degree, const int *d_out_degree, int n_rows, float *d_in_scale, float *d_out_scale,
                        void *stream) {
    DRONE_REQUIRE(n_rows >= 0, "drone_degree_scales: n_rows=%d is negative", n_rows);
    if (n_rows == 0) return DRONE_OK;
    DRONE_REQUIRE(d_in_degree && d_out_degree && d_in_scale && d_out_scale, "drone_degree_scales: NULL argument");
    degree_scales_kernel<<<ceil_div(n_rows, 256), 256, 0, (cudaStream_t)stream>>>(d_in_degree, d_out_degree, n_rows,
                                                                                 d_in_scale, d_out_scale);
    DRONE_LAUNCH_CHECK("degree_scales_kernel");
    return DRONE_OK;
}

int drone_spmm_rows(drone_plan *p, int orientation, int row_class, int F, const float *d_X, int ldx, float *d_Y, int ldy,
                    void *stream) {
    DRONE_REQUIRE(p != nullptr, "drone_spmm_rows: plan is NULL");
    DRONE_REQUIRE(orientation == DRONE_OP_A || orientation == DRONE_OP_AT, "drone_spmm_rows: orientation=%d", orientation);
    DRONE_REQUIRE(p->side[orientation].ready, "drone_spmm_rows: orientation %d was not prepared by drone_plan_create",
                  orientation);
    DRONE_REQUIRE(row_class >= 0 && row_class < p->n_classes, "drone_spmm_rows: row_class=%d, the plan has %d classes",
                  row_class, p->n_classes);
    DRONE_REQUIRE(F >= 1 && F <= 1024, "drone_spmm_rows: feature width F=%d outside 1..1024", F);
    DRONE_REQUIRE(ldx >= F && ldy >= F, "drone_spmm_rows: leading dimensions (ldx=%d, ldy=%d) below F=%d", ldx, ldy, F);
    if (p->n_rows == 0) return DRONE_OK;
    DRONE_REQUIRE(d_X && d_Y, "drone_spmm_rows: NULL operand");
    DRONE_REQUIRE(d_X != d_Y, "drone_spmm_rows: X and Y must not alias");
    OnDevice guard;
    const int rc = guard.enter(p->device);
    if (rc) return rc;
    CallOptions opt;
    opt.row_class = row_class;
    return spmm_impl(p, orientation, F, d_X, ldx, d_Y, ldy, (cudaStream_t)stream, opt);
}

static int ensure_staging(drone_plan *p, size_t bytes) {
    if (bytes <= p->stage_bytes) return DRONE_OK;
    DRONE_CUDA(cudaDeviceSynchronize());
    cudaFree(p->stage_x);
    cudaFree(p->stage_y);
    p->stage_x = p->stage_y = nullptr;
    p->stage_bytes = 0;
    DRONE_CUDA(cudaMalloc(&p->stage_x, bytes));
    DRONE_CUDA(cudaMalloc(&p->stage_y, bytes));
    p->stage_bytes = bytes;
    return DRONE_OK;
}

// Pinned host operands of at least 64 columns (a multiple of 8): the call can run as two column halves, the
// second half's host-to-device copy and the first half's result going over PCIe at the same time, in opposite
// directions.  DRONE_HOST_PIPELINE=0 keeps the copy - compute - copy sequence.
static bool host_call_can_be_pipelined(const drone_plan *p, int F, const float *h_X, const float *h_Y) {
    static const bool enabled = [] {
        const char *v = getenv("DRONE_HOST_PIPELINE");
        return !(v && v[0] == '0');
    }();
    (void)p;
    if (!enabled || F < 64 || F % 8 != 0) return false;
    for (const void *ptr : {(const void *)h_X, (const void *)h_Y}) {
        cudaPointerAttributes attr;
        if (cudaPointerGetAttributes(&attr, ptr) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (attr.type != cudaMemoryTypeHost) return false;
    }
    void *mapped = nullptr;      // the kernels store into Y through its device alias: it must be mapped memory
    if (cudaHostGetDevicePointer(&mapped, const_cast<float *>(h_Y), 0) != cudaSuccess || mapped == nullptr) {
        cudaGetLastError();
        return false;
    }
    return (reinterpret_cast<uintptr_t>(h_X) & 15) == 0 && (reinterpret_cast<uintptr_t>(mapped) & 15) == 0;
}

// The two halves: half h of X is copied (strided, the DMA engine reads 4·F/2 bytes of every host row) into the
// plan's staging on the copy stream; the aggregation of that half starts when it has landed and stores its result
// rows straight into the caller's pinned Y (the kernels' stores go out over PCIe as they are issued), while the copy
// engine is already bringing the other half of X in.
static int spmm_host_pipelined(drone_plan *p, int orientation, int F, const float *h_X, float *h_Y) {
    if (!p->copy_stream) DRONE_CUDA(cudaStreamCreateWithFlags(&p->copy_stream, cudaStreamNonBlocking));
    for (cudaEvent_t &e : p->half_loaded)
        if (!e) DRONE_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    float *d_Y = nullptr;
    DRONE_CUDA(cudaHostGetDevicePointer((void **)&d_Y, h_Y, 0));
    const int w = F / 2;
    const size_t pitch = sizeof(float) * (size_t)F;
    for (int h = 0; h < 2; ++h) {
        DRONE_CUDA(cudaMemcpy2DAsync(p->stage_x + h * w, pitch, h_X + h * w, pitch, sizeof(float) * (size_t)w, (size_t)p->n_rows,
                                     cudaMemcpyHostToDevice, p->copy_stream));
        DRONE_CUDA(cudaEventRecord(p->half_loaded[h], p->copy_stream));
    }
    for (int h = 0; h < 2; ++h) {
        DRONE_CUDA(cudaStreamWaitEvent(p->own_stream, p->half_loaded[h], 0));
        const int rc = spmm_impl(p, orientation, w, p->stage_x + h * w, F, d_Y + h * w, F, p->own_stream);
        if (rc) return rc;
    }
    DRONE_CUDA(cudaStreamSynchronize(p->own_stream));
    return DRONE_OK;
}

int drone_plan_reserve(drone_plan *p, int max_features, int what) {
    DRONE_REQUIRE(p != nullptr, "drone_plan_reserve: plan is NULL");
    DRONE_REQUIRE(max_features >= 1 && max_features <= 1024, "drone_plan_reserve: max_features=%d outside 1..1024",
                  max_features);
    OnDevice guard;
    int rc = guard.enter(p->device);
    if (rc) return rc;
    DRONE_REQUIRE((what & ~(DRONE_RESERVE_HOST_OPERANDS | DRONE_RESERVE_PADDED_ROWS)) == 0,
                  "drone_plan_reserve: what=%d is not a combination of DRONE_RESERVE_* flags", what);
    const size_t slots = (size_t)std::max(p->side[0].n_partials, p->side[1].n_partials);
    const int copied_features = (max_features + 3) & ~3;      // the width of a call on padded copies
    if (slots > 0 && (rc = ensure_scratch(p, sizeof(float) * slots * (size_t)copied_features))) return rc;
    if (what & DRONE_RESERVE_HOST_OPERANDS) {
        if ((rc = ensure_staging(p, sizeof(float) * (size_t)p->n_rows * (size_t)max_features))) return rc;
        if (!p->own_stream) DRONE_CUDA(cudaStreamCreateWithFlags(&p->own_stream, cudaStreamNonBlocking));
    }
    if ((what & DRONE_RESERVE_PADDED_ROWS) && p->n_rows > 0) {
        long long stride = 0;      // of the widths up to max_features, the one whose copy is largest
        for (int f = 9; f <= max_features; ++f) stride = std::max(stride, std::max(padded_stride(p->n_rows, f), slices_possible(p->n_rows, p->nnz) && lines_fit(p->n_rows, f) ? line_stride(f) : 0));
        rc = replace_padding(p, (size_t)stride * (size_t)p->n_rows, (size_t)copied_features * (size_t)p->n_rows);
        if (rc) return rc;
    }
    p->reserved_features = std::max(p->reserved_features, max_features);
    if (what & DRONE_RESERVE_PADDED_ROWS) p->reserved_copies = std::max(p->reserved_copies, max_features);
    return DRONE_OK;
}

int drone_spmm_host(drone_plan *p, int orientation, int F, const float *h_X, float *h_Y) {
    DRONE_REQUIRE(p != nullptr, "drone_spmm_host: plan is NULL");
    DRONE_REQUIRE(orientation == DRONE_OP_A || orientation == DRONE_OP_AT, "drone_spmm_host: orientation=%d",
                  orientation);
    DRONE_REQUIRE(p->side[orientation].ready, "drone_spmm_host: orientation %d was not prepared", orientation);
    DRONE_REQUIRE(F >= 1 && F <= 1024, "drone_spmm_host: feature width F=%d outside 1..1024", F);
    if (p->n_rows == 0) return DRONE_OK;
    DRONE_REQUIRE(h_X && h_Y, "drone_spmm_host: NULL operand");
    OnDevice guard;
    int rc = guard.enter(p->device);
    if (rc) return rc;
    const size_t bytes = sizeof(float) * (size_t)p->n_rows * (size_t)F;
    if ((rc = ensure_staging(p, bytes))) return rc;      // no-op after drone_plan_reserve(.., host_operands = 1)
    if (!p->own_stream) DRONE_CUDA(cudaStreamCreateWithFlags(&p->own_stream, cudaStreamNonBlocking));
    if (host_call_can_be_pipelined(p, F, h_X, h_Y)) return spmm_host_pipelined(p, orientation, F, h_X, h_Y);
    DRONE_CUDA(cudaMemcpyAsync(p->stage_x, h_X, bytes, cudaMemcpyHostToDevice, p->own_stream));
    if ((rc = spmm_impl(p, orientation, F, p->stage_x, F, p->stage_y, F, p->own_stream))) return rc;
    DRONE_CUDA(cudaMemcpyAsync(h_Y, p->stage_y, bytes, cudaMemcpyDeviceToHost, p->own_stream));
    DRONE_CUDA(cudaStreamSynchronize(p->own_stream));
    return DRONE_OK;
}

// Queue of host-operand calls.  Slot s = call number mod 2 owns one pair of staging buffers; three streams carry
// the three stages of a call (copy in, aggregation, copy out), chained by events, so that call k's operands come in
// while call k-1 is aggregated and call k-2's result goes out: PCIe is busy in both directions at once.
static int ensure_queue(drone_plan *p, size_t bytes) {
    if (!p->own_stream) DRONE_CUDA(cudaStreamCreateWithFlags(&p->own_stream, cudaStreamNonBlocking));
    if (!p->copy_stream) DRONE_CUDA(cudaStreamCreateWithFlags(&p->copy_stream, cudaStreamNonBlocking));
    if (!p->out_stream) DRONE_CUDA(cudaStreamCreateWithFlags(&p->out_stream, cudaStreamNonBlocking));
    for (int s = 0; s < 2; ++s)
        for (cudaEvent_t *e : {&p->queue_in[s], &p->queue_done[s], &p->queue_out[s]})
            if (!*e) DRONE_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    if (bytes <= p->queue_bytes) return DRONE_OK;
    DRONE_CUDA(cudaDeviceSynchronize());      // calls in flight use the buffers about to be replaced
    for (int s = 0; s < 2; ++s) {
        cudaFree(p->queue_x[s]);
        cudaFree(p->queue_y[s]);
        p->queue_x[s] = p->queue_y[s] = nullptr;
    }
    p->queue_bytes = 0;
    for (int s = 0; s < 2; ++s) {
        DRONE_CUDA(cudaMalloc(&p->queue_x[s], bytes));
        DRONE_CUDA(cudaMalloc(&p->queue_y[s], bytes));
    }
    p->queue_bytes = bytes;
    return DRONE_OK;
}

int drone_spmm_host_submit(drone_plan *p, int orientation, int F, const float *h_X, float *h_Y, long long *ticket) {
    DRONE_REQUIRE(p != nullptr, "drone_spmm_host_submit: plan is NULL");
    DRONE_REQUIRE(orientation == DRONE_OP_A || orientation == DRONE_OP_AT, "drone_spmm_host_submit: orientation=%d",
                  orientation);
    DRONE_REQUIRE(p->side[orientation].ready, "drone_spmm_host_submit: orientation %d was not prepared", orientation);
    DRONE_REQUIRE(F >= 1 && F <= 1024, "drone_spmm_host_submit: feature width F=%d outside 1..1024", F);
    DRONE_REQUIRE(ticket != nullptr, "drone_spmm_host_submit: ticket is NULL");
    DRONE_REQUIRE(p->n_rows == 0 || (h_X && h_Y), "drone_spmm_host_submit: NULL operand");
    OnDevice guard;
    int rc = guard.enter(p->device);
    if (rc) return rc;
    const long long k = p->submitted;
    const int s = (int)(k & 1);
    if (p->n_rows > 0) {
        const size_t bytes = sizeof(float) * (size_t)p->n_rows * (size_t)F;
        if ((rc = ensure_queue(p, bytes))) return rc;
        // the slot's previous call (k - 2) must have left it: its result copied out, hence its operands consumed
        if (k >= 2) DRONE_CUDA(cudaEventSynchronize(p->queue_out[s]));
        DRONE_CUDA(cudaMemcpyAsync(p->queue_x[s], h_X, bytes, cudaMemcpyHostToDevice, p->copy_stream));
        DRONE_CUDA(cudaEventRecord(p->queue_in[s], p->copy_stream));
        DRONE_CUDA(cudaStreamWaitEvent(p->own_stream, p->queue_in[s], 0));
        if ((rc = spmm_impl(p, orientation, F, p->queue_x[s], F, p->queue_y[s], F, p->own_stream))) return rc;
        DRONE_CUDA(cudaEventRecord(p->queue_done[s], p->own_stream));
        DRONE_CUDA(cudaStreamWaitEvent(p->out_stream, p->queue_done[s], 0));
        DRONE_CUDA(cudaMemcpyAsync(h_Y, p->queue_y[s], bytes, cudaMemcpyDeviceToHost, p->out_stream));
        DRONE_CUDA(cudaEventRecord(p->queue_out[s], p->out_stream));
    }
    *ticket = k;
    p->submitted = k + 1;
    return DRONE_OK;
}

int drone_spmm_host_wait(drone_plan *p, long long ticket) {
    DRONE_REQUIRE(p != nullptr, "drone_spmm_host_wait: plan is NULL");
    DRONE_REQUIRE(ticket >= 0 && ticket < p->submitted, "drone_spmm_host_wait: ticket %lld was not issued (%lld calls so far)",
                  ticket, p->submitted);
    if (p->n_rows == 0 || ticket + 2 < p->submitted) return DRONE_OK;     // a later submit on the slot waited for it
    OnDevice guard;
    const int rc = guard.enter(p->device);
    if (rc) return rc;
    DRONE_CUDA(cudaEventSynchronize(p->queue_out[ticket & 1]));
    return DRONE_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Aggregation without any allocation.
//
// Some callers hand every byte of device memory to their own pool when they start, or run on a
// thread that must never wait on the driver's allocator; for them a library call that may reach
// cudaMalloc is unusable.  drone_spmm can reach it (the partial sums of split rows live in a buffer
// that grows on demand).  The entry point below does the same work with the partial sums in a
// fixed array that is part of the library image: DRONE_STATIC_SCRATCH_BYTES on every GPU that loads
// the library, until the process exits.
// ---------------------------------------------------------------------------
namespace drone {

constexpr size_t kStaticScratchFloats = DRONE_STATIC_SCRATCH_BYTES / sizeof(float);

// Partial sums of split rows, [n_partials, F] floats.  In host code this name is only a handle for
// cudaGetSymbolAddress; kernels receive the device address obtained from it.
static __device__ __align__(256) float g_static_partials[kStaticScratchFloats];

static const int kMaxDevices = 64;
static float *g_static_partials_addr[kMaxDevices];   // device address of the array on each device, once known
static std::mutex g_static_partials_mutex;

// Device address of g_static_partials on the CURRENT device (looked up once per device).
static int static_partials_address(int device, float **out) {
    if (device < 0 || device >= kMaxDevices)
        return set_error(DRONE_E_INVALID, "drone_spmm_static_scratch: device ordinal %d is outside 0..%d", device,
                         kMaxDevices - 1);
    std::lock_guard<std::mutex> lock(g_static_partials_mutex);
    if (!g_static_partials_addr[device]) {
        float *addr = nullptr;
        const cudaError_t err = cudaGetSymbolAddress((void **)&addr, g_static_partials);
        if (err != cudaSuccess || !addr)
            return set_error(DRONE_E_CUDA, "drone_spmm_static_scratch: cudaGetSymbolAddress failed on device %d: %s", device,
                             cudaGetErrorString(err));
        g_static_partials_addr[device] = addr;
    }
    *out = g_static_partials_addr[device];
    return DRONE_OK;
}

}  // namespace drone

extern "C" int drone_spmm_static_scratch(drone_plan *p, int orientation, int F, const float *d_X, int ldx, float *d_Y,
                                         int ldy, void *stream) {
    DRONE_REQUIRE(p != nullptr, "drone_spmm_static_scratch: plan is NULL");
    DRONE_REQUIRE(orientation == DRONE_OP_A || orientation == DRONE_OP_AT, "drone_spmm_static_scratch: orientation=%d",
                  orientation);
    const drone::Side &s = p->side[orientation];
    DRONE_REQUIRE(s.ready, "drone_spmm_static_scratch: orientation %d was not prepared by drone_plan_create", orientation);
    DRONE_REQUIRE(F >= 1 && F <= 1024, "drone_spmm_static_scratch: feature width F=%d outside 1..1024", F);
    DRONE_REQUIRE(ldx >= F && ldy >= F, "drone_spmm_static_scratch: leading dimensions (ldx=%d, ldy=%d) below F=%d", ldx,
                  ldy, F);
    if (p->n_rows == 0) return DRONE_OK;
    DRONE_REQUIRE(d_X && d_Y, "drone_spmm_static_scratch: NULL operand");
    DRONE_REQUIRE(d_X != d_Y, "drone_spmm_static_scratch: X and Y must not alias");
    const size_t need = (size_t)s.n_partials * (size_t)((F + 3) & ~3);   // the width the kernels may run at (padded copy)
    if (need > drone::kStaticScratchFloats)
        return drone::set_error(DRONE_E_TOO_LARGE,
                                "drone_spmm_static_scratch: this plan needs %zu bytes of partial sums at F=%d, the built-in "
                                "scratch holds %zu; use drone_spmm",
                                need * sizeof(float), F, (size_t)DRONE_STATIC_SCRATCH_BYTES);
    drone::OnDevice guard;
    int rc = guard.enter(p->device);
    if (rc) return rc;
    float *partials = nullptr;
    rc = drone::static_partials_address(p->device, &partials);
    if (rc == DRONE_OK) {
        // the route of drone_spmm (copies where the plan already has room for them), with the partial sums in the built-in array: the
        // plan's own scratch pointer is swapped for the duration of the call
        float *const plan_scratch = p->scratch;
        const size_t plan_scratch_bytes = p->scratch_bytes;
        p->scratch = partials;
        p->scratch_bytes = DRONE_STATIC_SCRATCH_BYTES;
        drone::CallOptions opt;
        opt.no_allocation = true;
        rc = drone::spmm_impl(p, orientation, F, d_X, ldx, d_Y, ldy, (cudaStream_t)stream, opt);
        p->scratch = plan_scratch;
        p->scratch_bytes = plan_scratch_bytes;
    }
    return rc;
}
