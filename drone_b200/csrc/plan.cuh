// Internal layout of an aggregation plan (opaque drone_plan of the C ABI).
#pragma once

#include "common.cuh"

namespace drone {

// Plans with at most this many nonzeros run a call as one launch: up to here the launches of the separate kernels take
// longer than what handing chunks out dynamically, and overlapping the two kinds of rows, gains.  The two cross between 6 and
// 8.5 M nonzeros at every width of 8 and more (time of one launch over time of the separate kernels, R-MAT and power law, at 4.2 |
// 6.4 | 7.9 | 8.5 | 12.6 M nonzeros: F = 16 0.74 | 0.96 | 0.95 | 1.07 | 1.16, F = 64 0.81 | 0.97 | 1.00 | 1.08 | 1.05, F = 256
// 0.71 | 1.01 | 0.93 | 0.88 | 1.02; F = 4 still 0.91 at 12.6 M).
constexpr int kSmallNnz = 6 << 20;
// Of those, lanes with 8, 12, 16, and 32 single floats of a row keep few warps resident, so that one launch covers less.
constexpr int small_nnz_floats(int VPL) {
    return VPL < 8 ? 0x7fffffff : VPL == 8 ? 5 << 20 : VPL < 16 ? 3 << 20 : VPL < 32 ? 1 << 17 : 1 << 15;
}
constexpr int kWideSlots = 64;              // split rows above this many partial slots are reduced by a whole block
constexpr int kShortRangeNnz = 64;          // stream entries per lane group (plus at most one more row) ...
// ... and in small plans, where one group's walk is the length of the call, as long as the stream's entries times the lanes of
// a group stay below kFineRangeLanes: above it the longer ranges fill the GPU too and their rows stay closer together
// (us a call, ranges of 16 / 64; power law, 1.2 M rows of 5: F = 8 69 / 100, F = 16 110 / 104, F = 64 354 / 291; power law,
// 270,000 rows of 9: F = 8 27 / 44, F = 16 33 / 28, F = 64 114 / 87; R-MAT-18 + I: F = 16 52 / 59, F = 128 198 / 179).
constexpr int kFineRangeNnz = 16;
constexpr long long kFineRangeLanes = 6LL << 20;
// Calls on such plans may run in column slices (slices_by_counts): the widest operand is larger than L2, and the rows are long enough
// for the lists to be read once a slice.
inline bool slices_possible(int n_rows, int nnz) { return (long long)n_rows * 4096 > 100000000 && nnz / 24 >= n_rows; }
constexpr unsigned kLastInRow = 0x80000000u; // flag on s_col: last entry of its row
constexpr unsigned kPlaceholder = 0x40000000u; // flag on s_col: row has no nonzeros, entry carries no data
constexpr unsigned kColMask = 0x3fffffffu;
// Plans of very large graphs tag their most often gathered columns (bit 29 on the entries of col and s_col): the
// remaining bits of a tagged entry are the column's position in the plan's table of hot rows instead of the column.
constexpr unsigned kHotTag = 0x20000000u;
constexpr unsigned kHotMask = 0x1fffffffu;
constexpr int kMaxRowClasses = 16;         // row classes a plan can be given (drone_plan_set_row_classes)

// One chunk of a long row: nonzeros [k0, k0+len) of `row`.  slot >= 0 means the
// chunk's sum goes to partial-sum slot `slot` (the row has several chunks);
// slot < 0 means the chunk is the whole row and its sum goes straight to Y.
struct Chunk {
    int row;
    int k0;
    int len;
    int slot;
};

// A row whose chunks were summed separately: partial sums slot0 .. slot0+nslots-1,
// added in that order into Y[row].
struct SplitRow {
    int row;
    int slot0;
    int nslots;
    int pad;
};

// A cut of the short-row stream at row boundaries: range i starts at row row[i].
struct Ranges {
    int *row = nullptr;         // [n + 1]
    int n = 0;
    int start[kMaxRowClasses + 1] = {0};   // with row classes, class c's ranges are [start[c], start[c + 1])
};

// How the gathers of an orientation are spread over the rows of X: how many rows are gathered about how often, classes of the
// number of times being quarters of a power of two.
constexpr int kGatherClasses = 128;
struct GatherCounts {
    unsigned long long rows[kGatherClasses], gathers[kGatherClasses];
    static __host__ __device__ int class_of(int times) {      // times >= 1
        int e = 0;
        while (times >> e > 1) ++e;
        return e * 4 + (e >= 2 ? times >> (e - 2) : times << (2 - e)) % 4;
    }
    // Share of the gathers that go to the `n` most often gathered rows.
    double share(double n) const {
        double reached = 0, all = 0;
        for (int c = kGatherClasses - 1; c >= 0; --c) {
            all += (double)gathers[c];
            if (rows[c] == 0 || n <= 0) continue;
            reached += (double)gathers[c] * (n < (double)rows[c] ? n / (double)rows[c] : 1.0);
            n -= (double)rows[c];
        }
        return all > 0 ? reached / all : 1.0;
    }
};

// CSR of one orientation plus the work lists of its long rows.
struct Side {
    bool ready = false;
    int *rowptr = nullptr;     // [n_rows + 1]
    int *col = nullptr;        // [nnz]; in a tagged plan the hot columns carry kHotTag | position
    float *val = nullptr;      // [nnz]
    // tagged plans only: hot_ids[pos] = column that position pos of the table of hot rows stands for, most often
    // gathered first; col_plain = untagged copy of col, made when a caller asks for the CSR arrays
    int *hot_ids = nullptr;    // [n_hot]
    int n_hot = 0;
    int *col_plain = nullptr;  // [nnz] or NULL
    Chunk *chunks = nullptr;   // [n_chunks]
    SplitRow *split = nullptr; // [n_split_rows]
    SplitRow *wide = nullptr;  // [n_wide_rows] the split rows with more than kWideSlots slots (any order)
    int n_wide_rows = 0;
    bool counted = false;      // `counts` is known (count_gathers)
    GatherCounts counts;
    // Short rows (at most short_row_limit nonzeros) as one contiguous stream: their nonzeros copied
    // in row order, bit 31 of the column marking the last nonzero of a row.  A row without nonzeros
    // contributes one placeholder entry (bit 30) so that it is still written.  The stream is cut into
    // ranges of about kShortRangeNnz entries, in small plans also into ranges of about kFineRangeNnz.
    int *s_rows = nullptr;      // [n_short_rows] row id of each short row
    int *s_rowptr = nullptr;    // [n_short_rows + 1] start of each short row in the stream
    int *s_col = nullptr;       // [n_short_entries] column | flags
    float *s_val = nullptr;     // [n_short_entries]
    Ranges ranges, fine;
    DeviceBlock stream, lists;  // what the arrays of the short rows, and those of the chunks, are pieces of
    int n_short_rows = 0;
    int n_short_entries = 0;
    // Small plans (kSmallNnz): a call is one launch (spmm_small_kernel), in which split rows are closed by whoever
    // arrives last; slot_split[slot] = the slot's entry of `split`, arrived[entry] = slots written so far (0 between calls)
    bool small = false;
    int *slot_split = nullptr; // [n_partials]
    int *arrived = nullptr;    // [n_split_rows]
    int n_long_rows = 0;
    int n_chunks = 0;
    int n_split_rows = 0;
    int n_partials = 0;
    int max_nslots = 0;        // largest nslots over split rows
    // With row classes the four lists are class-major (all work of class 0 first, then class 1, ...; rows ascending
    // inside a class) and list x of class c is [x_start[c], x_start[c+1]).  Without classes everything is class 0.
    int n_classes = 1;
    int chunk_start[kMaxRowClasses + 1] = {0};
    int split_start[kMaxRowClasses + 1] = {0}, wide_start[kMaxRowClasses + 1] = {0};
};

}  // namespace drone

struct drone_plan;
namespace drone {
// slot_split[slot] = the slot's entry of s.split, for all partial slots of the side.
int fill_slot_split(const Side &s, int *slot_split, cudaStream_t st);
// drone_plan_create for users inside the library that read the plan's lists with kernels of their own (the
// PageRank pull): never tags columns.
int plan_create_untagged(drone_plan **out, int n_rows, int nnz, const int *d_index, const int *d_dst, const float *d_values,
                         const int *d_in_degree, const int *d_out_degree, int orientations, void *stream);
// Renumbers the columns of one orientation of an untagged plan by how often they occur, most frequent first (the
// frequencies are the row lengths of d_other_rowptr, the row pointer of the opposite orientation): afterwards column c of
// the plan's lists means position (*d_place_out)[c], a device array of n_rows ints the caller owns.  For users inside
// the library whose gathered operand is their own array and can be laid out in that order (the PageRank pull).
int plan_order_columns_by_frequency(drone_plan *p, int orientation, const int *d_other_rowptr, int **d_place_out, void *stream);

// The rows of one orientation of such a plan in the order of `place` as well, their edges as one stream.  Pieces of it are what
// warps work on (power iterations on R-MAT-22: see pagerank_stream.cuh).
constexpr int kTileEdges = 256;                  // what a warp takes at a time
constexpr unsigned kRowEnd = 0x80000000u;        // flag on a column: last edge of its row
constexpr int kSpansPieces = 0x40000000;         // flag on `at`: the row begins in an earlier piece than it ends in
struct RowStream {
    int *ptr = nullptr;        // [n + 1] first edge of the row at position i
    int *at = nullptr;         // [n] which of the rows with edges it is, | kSpansPieces; -1: it has none
    int *row_of = nullptr;     // [n] the row at position i
    int *first = nullptr;      // [n_pieces] which of the rows with edges a piece's first edge belongs to
    unsigned *col = nullptr;   // [n_tiles * kTileEdges] columns | kRowEnd; 0 beyond the last edge
    int n_pieces = 0, n_tiles = 0;
    int most_spanned = 0;      // pieces that a row reaches over before its last one, at most
#ifdef __CUDACC__
    // Piece q is tiles [first_tile(q), first_tile(q + 1)), one more or less than any other piece; none is empty.
    __host__ __device__ int first_tile(int q) const { return (int)((long long)n_tiles * q / n_pieces); }
    __host__ __device__ int piece_of(int edge) const {
        return (int)(((long long)(edge / kTileEdges + 1) * n_pieces - 1) / n_tiles);
    }
#endif
};
// Fills in what `out` points to: `block` is made with its arrays.  `warps`: how many will share the pieces.  kNoRoom: the device has
// no memory for it; anything else that fails is an error.
constexpr int kNoRoom = 1;
int plan_rows_in_order(const drone_plan *p, int orientation, const int *d_place, int warps, RowStream *out, DeviceBlock *block, cudaStream_t st);
}  // namespace drone

struct drone_plan {
    int device = 0;
    int sms = 0;               // multiprocessors of the device
    int n_rows = 0;
    int nnz = 0;
    bool for_spmm = true;      // false: a plan whose lists other kernels of the library read (plan_create_untagged)
    int short_row_limit = 0;   // rows with deg <= this are summed by one lane group
    int chunk_nnz = 0;         // nonzeros per chunk of longer rows
    int last_slice_width = 0;  // what the most recent call used (reported by drone_plan_get_stats)
    int slice_forced = -1;     // column-slice width of a call: -1 chosen per call, 0 never slice, w > 0 slices of w columns
    drone::Side side[2];       // [DRONE_OP_A], [DRONE_OP_AT]
    // partial sums of split rows, [n_partials, F] floats, grown on demand
    float *scratch = nullptr;
    size_t scratch_bytes = 0;
    // device staging for drone_spmm_host
    float *stage_x = nullptr, *stage_y = nullptr;
    size_t stage_bytes = 0;
    // row classes: rows in class-major order and where each class starts in that order (NULL / 1 class: none set)
    int *row_order = nullptr;  // [n_rows]
    int n_classes = 1;
    int class_start[drone::kMaxRowClasses + 1] = {0};
    // one word: the chunk kernel's work counter (set to 0 in front of every launch)
    unsigned *counter = nullptr;
    // tagged plans: the table of hot rows, refilled from X by every call
    float *hot_table = nullptr;
    size_t hot_table_bytes = 0;
    // Copies of X and Y with rows that can be accessed as float4, for operands whose rows cannot where they lie (a width
    // that is not a multiple of 4, odd leading dimensions or addresses): made by drone_plan_reserve or by the first such
    // call.  X is copied into pad_x before the kernels, the result out of pad_y after them.
    float *pad_x = nullptr, *pad_y = nullptr;
    size_t pad_x_floats = 0, pad_y_floats = 0;
    size_t pad_refused_bytes = ~(size_t)0;   // a call that needs this much new room for copies does without: so much did not fit
    // A graph captured from a call goes on using the buffers that the call used: replaced by larger ones they are kept until the
    // plan goes (give_back_replaced).
    struct Kept { void *buffer; Kept *before; };
    Kept *kept = nullptr;
    bool scratch_captured = false, pad_x_captured = false, pad_y_captured = false;
    int reserved_features = 0;     // drone_plan_reserve: calls up to this width allocate nothing
    int reserved_copies = 0;       // ... and up to this one have room for their copies
    int chunk_blocks_per_sm = 0;   // cap on resident blocks of the chunk kernel per SM (0: as many as fit)
    cudaStream_t own_stream = nullptr;
    // drone_spmm_host with pinned operands: second stream and one event per column half for the copy that runs ahead
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t half_loaded[2] = {nullptr, nullptr};
    // drone_spmm_host_submit / _wait: a second pair of staging buffers, a stream for the copies out, and per slot the
    // events "operand landed", "aggregation done", "result copied out"; `submitted` counts the calls queued so far
    float *queue_x[2] = {nullptr, nullptr}, *queue_y[2] = {nullptr, nullptr};
    size_t queue_bytes = 0;
    cudaStream_t out_stream = nullptr;
    cudaEvent_t queue_in[2] = {nullptr, nullptr}, queue_done[2] = {nullptr, nullptr}, queue_out[2] = {nullptr, nullptr};
    long long submitted = 0;
    // second stream and fork/join events: the short-row kernel runs beside the chunk kernels of the same call
    cudaStream_t side_stream = nullptr;
    cudaEvent_t fork_event = nullptr, join_event = nullptr;
};
