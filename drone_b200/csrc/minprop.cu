// Minimum propagation over an EBV-partitioned graph: the "cc_cuda" and "sssp_cuda" jobs.
//
// Both jobs push a value along the local out-edges until nothing changes (labels: the value itself; distances: value +
// edge length), then exchange the boundary: mirror -> master minimum, master -> mirror minimum.  Restated from
// DRONE/src/cuda/algorithm/cc.cu and sssp.cu (PEval / IncEval and their helper kernels) with these changes:
//   * one state, one set of kernels for both jobs: distances are non-negative floats, whose bit patterns order like
//     unsigned integers, so both kinds are "atomicMin on a 32-bit word";
//   * a local run is one launch: its rounds follow one another with a grid barrier between them instead of one or two
//     launches each and a look from the host, and vertices wait with large values until the small ones have spread;
//   * short rows of a frontier are walked as one flat list of edges, long ones in pieces handed to the whole grid (the
//     reference walks every row with one thread, which a hub row turns into one long serial loop);
//   * the exchange uses the static plan (rows in a fixed order, no ids on the wire, no allocation per superstep);
//     every boundary vertex travels as {value, flag} and only flagged entries count and are applied, which gives the
//     same values and the same Response sizes as the reference's lists of changed vertices.
// Labels start as GLOBAL vertex ids (the CPU job's choice, DRONE/src/algorithm/CC.go:73-79; cc_init writes the local
// index, cc.cu:14, which cannot be compared between workers).  A shorter distance always re-activates its vertex
// (sssp_exec asks for an improvement above 1e-6, sssp.cu:67; with the unit lengths build_graph stores both agree).
#include "exchange.cuh"
#include "grid_sync.cuh"

#include <algorithm>
#include <chrono>
#include <new>
#include <vector>

#include "../../include/drone_b200.h"

namespace drone {
int xplan_ensure_device(drone_xplan *x);
}

struct drone_mp {
    int device = 0, kind = 0, n_local = 0, nnz = 0, sms = 0;
    const int *index = nullptr, *dst = nullptr, *l2g = nullptr;   // borrowed device arrays
    const float *len = nullptr;                                   // borrowed, NULL = 1.0
    drone_xplan *xplan = nullptr;                                 // borrowed
    drone_comm *comm = nullptr;                                   // borrowed, may be NULL for one part
    unsigned *value = nullptr;     // [n] label, or the bits of a non-negative float distance
    int *state = nullptr;          // [n] during a run: r >= 0 waits to offer its value since round r (0: from the start),
                                   // kOffered after it did, kOfferedFirst the same but only from the start, kIdle neither
    int *active = nullptr;         // [n] after a run: 1 lowered in it, 0 in its first frontier and not lowered, -1 neither
    int *ubm = nullptr;            // [n] lowered by a received message since the last sweep
    uint2 *send = nullptr, *recv = nullptr;   // [max(up, down)] {value, flag}
    int *counters = nullptr;       // [0..3] exchange sizes, [4] VisitedSize; the run's control block follows them
    int4 *items = nullptr;         // [item_cap] {first edge, edges, value, 0}: pieces of the long rows of a round's frontier
    int item_cap = 0;
    drone::DeviceBlock block;             // what the arrays above are pieces of
    unsigned barrier_start = 0, barrier_polls = 0;   // what the grid barrier's count starts at, and when its waits run out
    bool started = false;
};

namespace drone {

constexpr int kWarpRow = 64;         // rows up to this many edges are walked by the warp that finds them in the frontier
constexpr int kIdle = -1, kOffered = -2, kOfferedFirst = -3;
constexpr int kItemEdges = 256;      // longer ones are cut into pieces of this many edges for the whole grid
constexpr int kRunThreads = 1024;
constexpr int kRoundsPerLaunch = 4096;
constexpr unsigned kFarBits = 0x4CBEBC20u;   // 1e8f, the reference's "not reached" (sssp.cu:33)

static inline int grid_mp(long long n, int cap = 148 * 16) {
    long long g = (n + 255) / 256;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

struct MpRound {
    int items;             // pieces of long rows in the queue
    int waiting;           // vertices left waiting above the limit, not counting those lowered in this round
    unsigned nearest;      // complement of the least value that waits after the round (0: nobody waits)
    int pad;
};

struct MpControl {
    GridBarrier barrier;
    int unfinished;        // 1: the launch stopped after kRoundsPerLaunch rounds
    int round;             // where the next launch goes on
    unsigned limit;
    int pad[3];
    MpRound rounds[4];     // round r uses rounds[r & 3]
};

enum MpStart { kMpPeval = 0, kMpIncEval = 1, kMpContinue = 2 };

struct MpArgs {
    int n, start, source_global, item_cap;
    unsigned barrier_start, barrier_polls;
    const int *index, *dst, *l2g;
    const float *len;
    unsigned *value;
    int *state, *active, *ubm, *counters;
    int4 *items;
    MpControl *control;
};

// The value an edge offers: a label as it is, a distance plus the edge's length.
template <int KIND>
__device__ __forceinline__ unsigned mp_offer(unsigned now, const float *len, int k) {
    if (KIND == DRONE_MP_CC) return now;
    return __float_as_uint(__uint_as_float(now) + (len ? __ldg(len + k) : 1.0f));
}

// `held`: value[w] as some moment of this run had it; values only fall, so it can only be too high.  Nobody waits for the
// atomic's result: whoever finds held > offer marks the vertex, and rightly so, since its value then was, or had been in
// this run, lowered to the offer or below.  (A vertex lowered further by somebody else may offer once more for nothing.)
// `least` keeps the least value offered this way.
__device__ __forceinline__ void mp_lower(const MpArgs &a, int w, unsigned offer, unsigned held, int round, unsigned &least) {
    if (offer < held) {
        atomicMin(a.value + w, offer);
        a.state[w] = round + 1;
        least = min(least, offer);
    }
}

// Values up to which waiting vertices offer theirs, given the least of them.  Labels: powers of 32, so that the vertices
// with the smallest labels, one of which will be nearly everybody's in the end, spread theirs before the others have
// offered labels that nobody keeps.  Distances: twice the least, so that few vertices offer a distance that a shorter
// path still replaces.  All labels, once few are left (distances have no such end: few wait at the start as well).
template <int KIND>
__device__ __forceinline__ unsigned mp_limit(unsigned least, bool few) {
    if (KIND == DRONE_MP_SSSP) return __float_as_uint(2.0f * __uint_as_float(least));
    if (few) return 0xfffffffeu;
    unsigned limit = 0;
    while (limit < least) {
        if (limit >= 1u << 26) return 0xfffffffeu;
        limit = limit * 32 + 31;
    }
    return limit;
}

constexpr int kGroup = 128;          // vertices a warp looks at together
constexpr int kEdgesInFlight = 8;    // edges a lane reads together: their ends, then the values there (through L1: a value that
                                     // is out of date there costs an offer for nothing, reading past it 40 % on R-MAT-20)
struct MpGroupRows {                 // the rows of a group: row i's edges are entries upto[i-1] .. upto[i] of one flat list
    int upto[kGroup];
    int row0[kGroup];                // entry e of the list is edge row0[i] + e of the graph
    unsigned value[kGroup];          // what the row's vertex offers
};

// Reduces the least waiting value and the number of waiting vertices of a block into the round's word.
__device__ __forceinline__ void mp_note_round(MpRound *r, unsigned least, int waiting, unsigned *block_nearest, int *block_waiting) {
    const unsigned nearest = __reduce_max_sync(0xffffffffu, ~least);
    waiting = __reduce_add_sync(0xffffffffu, waiting);
    if (threadIdx.x == 0) {
        *block_nearest = 0;
        *block_waiting = 0;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        if (nearest) atomicMax(block_nearest, nearest);
        if (waiting) atomicAdd(block_waiting, waiting);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (*block_nearest) atomicMax(&r->nearest, *block_nearest);
        if (*block_waiting) atomicAdd(&r->waiting, *block_waiting);
    }
}

// One local run, all rounds in one launch (cc_exec, cc.cu:21-46; sssp_exec, sssp.cu:41-74, until nothing changes).
//
// A round: every warp looks at 128 vertices at a time; those that wait and lie within the limit offer their value to
// their out-neighbours, short rows at once (the rows of the group as one flat list of edges, so that lanes stay busy
// whatever the degrees), long rows as pieces in a queue that the whole grid works off after a barrier.  The limit follows
// the least value that waits after the round.
//
// Bound: one scattered 4-byte read of the neighbour's value per edge offered, up to 32 LSU wavefronts a load instruction
// (about 2.8e11 a second on the whole part); the order above lets nearly every vertex offer once.  A step used to be two
// launches over all vertices, every label went out before the small ones had spread, and the host looked in every fourth
// step.  R-MAT-20 symmetrised, labels: 5.13 -> 0.26 ms; R-MAT-22, unit distances: 4.02 -> 0.58, weighted: 7.90 -> 1.34.
template <int KIND>
__global__ void __launch_bounds__(kRunThreads, 1) mp_run_kernel(const MpArgs a) {
    extern __shared__ __align__(16) char group_bytes[];
    const int lane = threadIdx.x & 31;
    MpGroupRows &rows = reinterpret_cast<MpGroupRows *>(group_bytes)[threadIdx.x >> 5];
    const int warp = (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x), n_warps = (int)((blockDim.x >> 5) * gridDim.x);
    const int first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    __shared__ unsigned block_nearest;
    __shared__ int block_waiting;
    unsigned phase = a.barrier_start;
    int round = 1;
    unsigned limit = 0;
    if (a.start == kMpContinue) {
        round = a.control->round;
        limit = a.control->limit;
    } else {
        // PEval: every label waits, or only the source.  IncEval: vertices lowered by a message (cc_process_messages,
        // cc.cu:385-398).  A vertex without out-edges has nobody to offer to.
        for (int i = first; i < a.n; i += stride) {
            bool front;
            if (a.start == kMpPeval) {
                const int gid = __ldg(a.l2g + i);
                front = KIND == DRONE_MP_CC || gid == a.source_global;
                a.value[i] = KIND == DRONE_MP_CC ? (unsigned)gid : front ? 0u : kFarBits;
            } else {
                front = a.ubm[i] != 0;
            }
            a.ubm[i] = 0;
            a.state[i] = !front ? kIdle : __ldg(a.index + i + 1) > __ldg(a.index + i) ? 0 : kOfferedFirst;
        }
        if (!grid_barrier(&a.control->barrier, phase, a.barrier_polls)) return;
    }
    const int last_round = round + kRoundsPerLaunch;
    const int few = max(1024, a.n / 64);
    bool finished = false;
    while (!finished && round < last_round) {
        MpRound *this_round = a.control->rounds + (round & 3);
        unsigned least = 0xffffffffu;
        int waiting = 0;
#pragma unroll 1
        for (long long base = (long long)warp * kGroup; base < a.n; base += (long long)n_warps * kGroup) {
            int mark[4];
            const int v0 = (int)base + lane * 4;
            if (base + kGroup <= a.n) {
                const int4 s4 = *reinterpret_cast<const int4 *>(a.state + v0);
                mark[0] = s4.x; mark[1] = s4.y; mark[2] = s4.z; mark[3] = s4.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) mark[j] = v0 + j < a.n ? a.state[v0 + j] : kIdle;
            }
            // a mark of this round's making (round + 1) waits for the next one
            bool any = false;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (mark[j] > round) mark[j] = kIdle;
                any = any || mark[j] >= 0;
            }
            if (!__any_sync(0xffffffffu, any)) continue;
            unsigned now[4];
            int begin[5];
#pragma unroll
            for (int j = 0; j < 4; ++j) now[j] = mark[j] >= 0 ? __ldcg(a.value + v0 + j) : 0u;
#pragma unroll
            for (int j = 0; j < 5; ++j) begin[j] = any ? __ldg(a.index + min(v0 + j, a.n)) : 0;
            int deg[4], pieces = 0, sum = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                deg[j] = 0;
                if (mark[j] < 0) continue;
                if (now[j] > limit) {
                    least = min(least, now[j]);
                    ++waiting;
                    continue;
                }
                // Off the list, unless somebody lowers the vertex just now: that leaves round + 1 there, before or after.
                // Whether the value read above was the one from before or after does not matter then.
                atomicCAS(a.state + v0 + j, mark[j], mark[j] > 0 ? kOffered : kOfferedFirst);
                deg[j] = begin[j + 1] - begin[j];
                if (deg[j] > kWarpRow) pieces += (deg[j] + kItemEdges - 1) / kItemEdges;
                else sum += deg[j];
            }
            // long rows: pieces into the queue
            if (__any_sync(0xffffffffu, pieces > 0)) {
                int before = pieces;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, before, d);
                    if (lane >= d) before += t;
                }
                int at = 0;
                if (lane == 31) at = atomicAdd(&this_round->items, before);
                at = __shfl_sync(0xffffffffu, at, 31) + before - pieces;
                if (pieces > 0 && at + pieces <= a.item_cap) {      // always: the capacity covers every long row at once
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (deg[j] > kWarpRow) {
                            for (int i = 0; i < deg[j]; i += kItemEdges)
                                a.items[at++] = make_int4(begin[j] + i, min(kItemEdges, deg[j] - i), (int)now[j], 0);
                            deg[j] = 0;
                        }
                }
            }
            // short rows
            int upto = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= d) upto += t;
            }
            const int total = __shfl_sync(0xffffffffu, upto, 31);
            if (total == 0) continue;
            __syncwarp();      // the previous group's list has been read
            int end = upto - sum;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                rows.row0[lane * 4 + j] = begin[j] - end;
                end += deg[j];
                rows.upto[lane * 4 + j] = end;
                rows.value[lane * 4 + j] = now[j];
            }
            __syncwarp();
            constexpr int UE = kEdgesInFlight;
#pragma unroll 1
            for (int e0 = 0; e0 < total; e0 += 32 * UE) {
                int k[UE], w[UE];
                unsigned offer[UE], held[UE];
#pragma unroll
                for (int u = 0; u < UE; ++u) {
                    const int e = e0 + u * 32 + lane;
                    int i = 0;      // the first row whose end lies beyond e
#pragma unroll
                    for (int d = kGroup / 2; d > 0; d >>= 1)
                        if (rows.upto[i + d - 1] <= e) i += d;
                    k[u] = rows.row0[i] + e;
                    offer[u] = rows.value[i];
                    w[u] = e < total ? __ldcs(a.dst + k[u]) : -1;
                }
#pragma unroll
                for (int u = 0; u < UE; ++u)
                    if (w[u] >= 0) {
                        offer[u] = mp_offer<KIND>(offer[u], a.len, k[u]);
                        held[u] = a.value[w[u]];
                    }
#pragma unroll
                for (int u = 0; u < UE; ++u)
                    if (w[u] >= 0) mp_lower(a, w[u], offer[u], held[u], round, least);
            }
        }
        mp_note_round(this_round, least, waiting, &block_nearest, &block_waiting);
        if (!grid_barrier(&a.control->barrier, phase, a.barrier_polls)) return;
        const int n_items = min(__ldcg(&this_round->items), a.item_cap);
        if (n_items > 0) {
            // pieces of long rows: a warp each
            constexpr int UE = kEdgesInFlight;
            least = 0xffffffffu;
#pragma unroll 1
            for (int i = warp; i < n_items; i += n_warps) {
                const int4 it = __ldcg(a.items + i);
#pragma unroll 1
                for (int e0 = 0; e0 < it.y; e0 += 32 * UE) {
                    int w[UE];
                    unsigned offer[UE], held[UE];
#pragma unroll
                    for (int u = 0; u < UE; ++u) {
                        const int e = e0 + u * 32 + lane;
                        w[u] = e < it.y ? __ldcs(a.dst + it.x + e) : -1;
                    }
#pragma unroll
                    for (int u = 0; u < UE; ++u)
                        if (w[u] >= 0) {
                            offer[u] = mp_offer<KIND>((unsigned)it.z, a.len, it.x + e0 + u * 32 + lane);
                            held[u] = a.value[w[u]];
                        }
#pragma unroll
                    for (int u = 0; u < UE; ++u)
                        if (w[u] >= 0) mp_lower(a, w[u], offer[u], held[u], round, least);
                }
            }
            mp_note_round(this_round, least, 0, &block_nearest, &block_waiting);
            if (!grid_barrier(&a.control->barrier, phase, a.barrier_polls)) return;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {      // used next two rounds from now; its last readers are behind the barrier
            MpRound *later = a.control->rounds + ((round + 2) & 3);
            later->items = 0;
            later->waiting = 0;
            later->nearest = 0;
        }
        const unsigned nearest = __ldcg(&this_round->nearest);
        if (nearest == 0) finished = true;
        else if (~nearest > limit) limit = mp_limit<KIND>(~nearest, __ldcg(&this_round->waiting) <= few);
        ++round;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.control->unfinished = finished ? 0 : 1;
        a.control->round = round;
        a.control->limit = limit;
    }
    if (finished) {      // VisitedSize as the reference counts it: entries of `active` that are not 0 (countActive, common.cu:6-16)
        int seen = 0;
        for (int i = first; i < a.n; i += stride) {
            const int st = a.state[i];
            const int active = st == kIdle ? -1 : st == kOfferedFirst ? 0 : 1;
            a.active[i] = active;
            seen += active != 0;
        }
        seen = __reduce_add_sync(0xffffffffu, seen);
        if (lane == 0 && seen) atomicAdd(a.counters + 4, seen);
    }
}

// Mirrors lowered in this run go up (cc_generate_sendBuff_mirror, cc.cu:82-106: active > 0).
__global__ void mp_pack_up_kernel(const int *__restrict__ up_rows, int n_up, const unsigned *value, const int *active,
                                  uint2 *send, int *counters) {
    int mine = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_up; i += (long long)gridDim.x * blockDim.x) {
        const int r = up_rows[i];
        const unsigned flag = active[r] > 0 ? 1u : 0u;
        send[i] = make_uint2(value[r], flag);
        mine += (int)flag;
    }
    if (mine) atomicAdd(counters + 0, mine);
}

// A master takes the minimum of what its mirrors sent (cc_process_recvBuff, cc.cu:135-157).
__global__ void mp_apply_up_kernel(const int *__restrict__ m_rows, const int *__restrict__ m_off,
                                   const int *__restrict__ m_pos, int n_m, const uint2 *recv, unsigned *value, int *ubm,
                                   int *counters) {
    int got = 0;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n_m; m += (long long)gridDim.x * blockDim.x) {
        const int r = m_rows[m];
        unsigned best = value[r];
        bool lowered = false;
        for (int k = m_off[m]; k < m_off[m + 1]; ++k) {
            const uint2 e = recv[m_pos[k]];
            if (!e.y) continue;
            ++got;
            if (e.x < best) { best = e.x; lowered = true; }
        }
        if (lowered) { value[r] = best; ubm[r] = 1; }
    }
    if (got) atomicAdd(counters + 1, got);
}

// Masters lowered in this run or by a message go down, once per mirror (cc_generate_sendBuff_master, cc.cu:108-133).
__global__ void mp_pack_down_kernel(const int *__restrict__ down_rows, int n_down, const unsigned *value, const int *active,
                                    const int *ubm, uint2 *send, int *counters) {
    int mine = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_down; i += (long long)gridDim.x * blockDim.x) {
        const int r = down_rows[i];
        const unsigned flag = (active[r] > 0 || ubm[r] != 0) ? 1u : 0u;
        send[i] = make_uint2(value[r], flag);
        mine += (int)flag;
    }
    if (mine) atomicAdd(counters + 2, mine);
}

__global__ void mp_apply_down_kernel(const int *__restrict__ up_rows, int n_up, const uint2 *recv, unsigned *value, int *ubm,
                                     int *counters) {
    int got = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_up; i += (long long)gridDim.x * blockDim.x) {
        const uint2 e = recv[i];
        if (!e.y) continue;
        ++got;
        const int r = up_rows[i];
        if (e.x < value[r]) { value[r] = e.x; ubm[r] = 1; }
    }
    if (got) atomicAdd(counters + 3, got);
}

// Moves the packed boundary entries of all parts: over NCCL (one part per process) or as device-to-device copies
// (all parts in this process).
static int mp_move(std::vector<drone_mp *> &parts, bool up, bool local, cudaStream_t st) {
    if (!local) {
        drone_mp *p = parts[0];
        const drone_xplan *x = p->xplan;
        if (x->nranks == 1) return DRONE_OK;
        const std::vector<int> &s_off = up ? x->up_off : x->down_off;
        const std::vector<int> &r_off = up ? x->down_off : x->up_off;
        DRONE_NCCL(ncclGroupStart());
        for (int q = 0; q < x->nranks; ++q) {
            if (q == x->rank) continue;
            const size_t ns = (size_t)(s_off[q + 1] - s_off[q]) * 2, nr = (size_t)(r_off[q + 1] - r_off[q]) * 2;
            if (ns) DRONE_NCCL(ncclSend(p->send + s_off[q], ns, ncclUint32, q, p->comm->comm, st));
            if (nr) DRONE_NCCL(ncclRecv(p->recv + r_off[q], nr, ncclUint32, q, p->comm->comm, st));
        }
        DRONE_NCCL(ncclGroupEnd());
        return DRONE_OK;
    }
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
                DRONE_CUDA(cudaMemcpyAsync(parts[q]->recv + r_off[p], parts[p]->send + s_off[q], ns * sizeof(uint2),
                                           cudaMemcpyDeviceToDevice, st));
        }
    return DRONE_OK;
}

// Counters and control block of a handle lie in one piece, so that one memset and one copy serve both.
struct MpReport {
    int counters[8];
    MpControl control;
};

// Launches (or continues) the local run of one part.
static int mp_launch(drone_mp *p, int start, int source_global, cudaStream_t st) {
    MpArgs a;
    a.n = p->n_local;
    a.start = start;
    a.source_global = source_global;
    a.item_cap = p->item_cap;
    a.index = p->index;
    a.dst = p->dst;
    a.l2g = p->l2g;
    a.len = p->len;
    a.value = p->value;
    a.state = p->state;
    a.active = p->active;
    a.ubm = p->ubm;
    a.counters = p->counters;
    a.items = p->items;
    a.control = &reinterpret_cast<MpReport *>(p->counters)->control;
    a.barrier_start = p->barrier_start;
    a.barrier_polls = p->barrier_polls;
    if (start == kMpContinue) DRONE_CUDA(cudaMemsetAsync(&a.control->barrier.arrived, 0, sizeof(unsigned), st));
    else DRONE_CUDA(cudaMemsetAsync(p->counters, 0, sizeof(MpReport), st));
    if (p->barrier_start != 0)
        DRONE_CUDA(cudaMemcpyAsync(&a.control->barrier.arrived, &p->barrier_start, sizeof(unsigned), cudaMemcpyHostToDevice, st));
    // a block has at least about 4096 edges and vertices to look at; more blocks only make the barriers longer
    const int grid = std::max(1, (int)std::min<long long>(p->sms, ((long long)p->n_local + p->nnz + 4095) / 4096));
    void *args[] = {&a};
    const size_t smem = sizeof(MpGroupRows) * (kRunThreads / 32);
    const void *kernel = p->kind == DRONE_MP_CC ? (const void *)mp_run_kernel<DRONE_MP_CC> : (const void *)mp_run_kernel<DRONE_MP_SSSP>;
    DRONE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    DRONE_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kRunThreads), args, smem, st));
    count_launch();
    return DRONE_OK;
}

// Local runs of all parts; on return they have finished and reports[i] is what part i's left.
static int mp_local_runs(std::vector<drone_mp *> &parts, bool peval, int source_global, std::vector<MpReport> &reports,
                         cudaStream_t st) {
    int rc;
    for (drone_mp *p : parts)
        if ((rc = mp_launch(p, peval ? kMpPeval : kMpIncEval, source_global, st))) return rc;
    for (bool again = true; again;) {
        for (size_t i = 0; i < parts.size(); ++i)
            DRONE_CUDA(cudaMemcpyAsync(&reports[i], parts[i]->counters, sizeof(MpReport), cudaMemcpyDeviceToHost, st));
        DRONE_CUDA(cudaStreamSynchronize(st));
        again = false;
        for (size_t i = 0; i < parts.size(); ++i) {
            if (reports[i].control.barrier.failed) {
                for (drone_mp *p : parts) p->started = false;
                return set_error(DRONE_E_STATE, "a wait between the blocks of a local run ran out");
            }
            if (!reports[i].control.unfinished) continue;
            again = true;
            if ((rc = mp_launch(parts[i], kMpContinue, source_global, st))) return rc;
        }
    }
    return DRONE_OK;
}

static int mp_exchange(std::vector<drone_mp *> &parts, bool local, cudaStream_t st) {
    int rc;
    for (drone_mp *p : parts) {
        const drone_xplan *x = p->xplan;
        const int n_up = (int)x->up_rows.size();
        if (n_up) {
            mp_pack_up_kernel<<<grid_mp(n_up), 256, 0, st>>>(x->d_up_rows, n_up, p->value, p->active, p->send, p->counters);
            DRONE_LAUNCH_CHECK("mp_pack_up_kernel");
        }
    }
    if ((rc = mp_move(parts, true, local, st))) return rc;
    for (drone_mp *p : parts) {
        const drone_xplan *x = p->xplan;
        const int n_m = (int)x->m_rows.size(), n_down = (int)x->down_rows.size();
        if (n_m) {
            mp_apply_up_kernel<<<grid_mp(n_m), 256, 0, st>>>(x->d_m_rows, x->d_m_off, x->d_m_pos, n_m, p->recv, p->value, p->ubm,
                                                            p->counters);
            DRONE_LAUNCH_CHECK("mp_apply_up_kernel");
        }
        if (n_down) {
            mp_pack_down_kernel<<<grid_mp(n_down), 256, 0, st>>>(x->d_down_rows, n_down, p->value, p->active, p->ubm, p->send,
                                                                p->counters);
            DRONE_LAUNCH_CHECK("mp_pack_down_kernel");
        }
    }
    if ((rc = mp_move(parts, false, local, st))) return rc;
    for (drone_mp *p : parts) {
        const drone_xplan *x = p->xplan;
        const int n_up = (int)x->up_rows.size();
        if (n_up) {
            mp_apply_down_kernel<<<grid_mp(n_up), 256, 0, st>>>(x->d_up_rows, n_up, p->recv, p->value, p->ubm, p->counters);
            DRONE_LAUNCH_CHECK("mp_apply_down_kernel");
        }
    }
    return DRONE_OK;
}

// One superstep of all given parts (one part over NCCL, or all parts of a partition held in this process).
static int mp_step(std::vector<drone_mp *> &parts, bool peval, int source_global, bool local, drone_pr_response *res,
                   cudaStream_t st) {
    using clock = std::chrono::steady_clock;
    const auto t0 = clock::now();
    int rc;
    for (drone_mp *p : parts)
        if (!peval && !p->started) return set_error(DRONE_E_STATE, "IncEVal called before PEVal");
    std::vector<MpReport> reports(parts.size());
    if ((rc = mp_local_runs(parts, peval, source_global, reports, st))) return rc;
    for (drone_mp *p : parts) p->started = true;
    const auto t1 = clock::now();
    if (parts[0]->xplan->nranks > 1) {
        if ((rc = mp_exchange(parts, local, st))) return rc;
        for (size_t i = 0; i < parts.size(); ++i)
            DRONE_CUDA(cudaMemcpyAsync(reports[i].counters, parts[i]->counters, sizeof(reports[i].counters), cudaMemcpyDeviceToHost, st));
        DRONE_CUDA(cudaStreamSynchronize(st));
    }
    const auto t2 = clock::now();
    for (size_t i = 0; i < parts.size(); ++i) {
        drone_pr_response &r = res[i];
        r.Mirror2MasterSendSize = reports[i].counters[0];
        r.Mirror2MasterRecvSize = reports[i].counters[1];
        r.Master2MirrorSendSize = reports[i].counters[2];
        r.Master2MirrorRecvSize = reports[i].counters[3];
        r.VisitedSize = reports[i].counters[4];
        r.LocalVertexSize = parts[i]->n_local;
        r.CalTime = std::chrono::duration<float>(t1 - t0).count();
        r.SendTime = std::chrono::duration<float>(t2 - t1).count();
    }
    return DRONE_OK;
}

static int mp_prepare(std::vector<drone_mp *> &parts) {
    for (drone_mp *p : parts) {
        DRONE_REQUIRE(p != nullptr, "NULL job handle");
        const int rc = xplan_ensure_device(p->xplan);
        if (rc) return rc;
    }
    return DRONE_OK;
}

}  // namespace drone

using namespace drone;

extern "C" {

int drone_mp_destroy(drone_mp *p);

int drone_mp_create(drone_mp **out, int kind, int n_local, int nnz, const int *d_index, const int *d_dst,
                    const float *d_edge_len, const int *d_local2global, drone_xplan *xplan, drone_comm *comm) {
    DRONE_REQUIRE(out != nullptr, "drone_mp_create: out is NULL");
    *out = nullptr;
    DRONE_REQUIRE(kind == DRONE_MP_CC || kind == DRONE_MP_SSSP, "drone_mp_create: kind=%d", kind);
    DRONE_REQUIRE(n_local >= 0 && nnz >= 0, "drone_mp_create: negative size");
    DRONE_REQUIRE(xplan != nullptr, "drone_mp_create: exchange plan is NULL");
    DRONE_REQUIRE(xplan->n_local == n_local, "drone_mp_create: the exchange plan was made for %d rows, the graph has %d",
                  xplan->n_local, n_local);
    DRONE_REQUIRE(xplan->nranks == 1 || comm == nullptr || (comm->nranks == xplan->nranks && comm->rank == xplan->rank),
                  "drone_mp_create: communicator and exchange plan disagree on rank / size");
    DRONE_REQUIRE(n_local == 0 || (d_index && d_local2global), "drone_mp_create: NULL graph array");
    DRONE_REQUIRE(nnz == 0 || d_dst != nullptr, "drone_mp_create: d_dst is NULL with nnz=%d", nnz);
    if (n_local > 0) {   // the relax kernels index the value arrays with d_dst: reject what would run out of bounds
        const int bad = validate_csr("drone_mp_create", d_index, d_dst, n_local, n_local, nnz, nullptr);
        if (bad) return bad;
    }
    drone_mp *p = new (std::nothrow) drone_mp();
    if (!p) return set_error(DRONE_E_INVALID, "drone_mp_create: out of host memory");
    p->kind = kind;
    p->n_local = n_local;
    p->nnz = nnz;
    p->index = d_index;
    p->dst = d_dst;
    p->len = d_edge_len;
    p->l2g = d_local2global;
    p->xplan = xplan;
    p->comm = comm;
    p->barrier_start = barrier_start();
    p->barrier_polls = barrier_polls();
    cudaError_t err = cudaGetDevice(&p->device);
    const size_t n1 = (size_t)(n_local > 0 ? n_local : 1);
    const size_t nb = std::max<size_t>(std::max(xplan->up_rows.size(), xplan->down_rows.size()), 1);
    p->block.add(&p->value, sizeof(unsigned) * n1);
    p->block.add(&p->state, sizeof(int) * (n1 + 3));      // read four at a time
    p->block.add(&p->active, sizeof(int) * n1);
    p->block.add(&p->ubm, sizeof(int) * n1);
    p->block.add(&p->send, sizeof(uint2) * nb);
    p->block.add(&p->recv, sizeof(uint2) * nb);
    p->block.add(&p->counters, sizeof(MpReport));
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, p->device);
    // every row above kWarpRow in the frontier at once: full pieces, and one partial piece per such row
    p->item_cap = nnz / kItemEdges + nnz / kWarpRow + 16;
    p->block.add(&p->items, sizeof(int4) * (size_t)p->item_cap);
    if (err == cudaSuccess) err = p->block.make();
    if (err != cudaSuccess) {
        drone_mp_destroy(p);
        return set_error(DRONE_E_CUDA, "drone_mp_create: %s", cudaGetErrorString(err));
    }
    *out = p;
    return DRONE_OK;
}

int drone_mp_destroy(drone_mp *p) {
    if (!p) return DRONE_OK;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(p->device);
    p->block.release();
    if (prev >= 0) cudaSetDevice(prev);
    delete p;
    return DRONE_OK;
}

static int mp_run(std::vector<drone_mp *> &parts, bool peval, int source_global, bool local, drone_pr_response *res,
                  void *stream) {
    DRONE_REQUIRE(res != nullptr, "Response pointer is NULL");
    OnDevice dev;
    int rc = dev.enter(parts[0]->device);      // calls may arrive on any host thread
    if (rc || (rc = mp_prepare(parts))) return rc;
    return mp_step(parts, peval, source_global, local, res, (cudaStream_t)stream);
}

int drone_mp_peval(drone_mp *p, int source_global_id, drone_pr_response *res, void *stream) {
    DRONE_REQUIRE(p != nullptr, "drone_mp_peval: NULL job");
    DRONE_REQUIRE(p->xplan->nranks == 1 || p->comm != nullptr, "drone_mp_peval: %d ranks but no communicator", p->xplan->nranks);
    std::vector<drone_mp *> parts{p};
    return mp_run(parts, true, source_global_id, false, res, stream);
}

int drone_mp_inceval(drone_mp *p, drone_pr_response *res, void *stream) {
    DRONE_REQUIRE(p != nullptr, "drone_mp_inceval: NULL job");
    DRONE_REQUIRE(p->xplan->nranks == 1 || p->comm != nullptr, "drone_mp_inceval: %d ranks but no communicator", p->xplan->nranks);
    std::vector<drone_mp *> parts{p};
    return mp_run(parts, false, -1, false, res, stream);
}

int drone_mp_step_local(int n_parts, drone_mp **jobs, int is_peval, int source_global_id, drone_pr_response *res,
                        void *stream) {
    DRONE_REQUIRE(n_parts >= 1 && jobs != nullptr, "drone_mp_step_local: no parts");
    std::vector<drone_mp *> parts(jobs, jobs + n_parts);
    for (int i = 0; i < n_parts; ++i) {
        DRONE_REQUIRE(parts[i] != nullptr, "drone_mp_step_local: part %d is NULL", i);
        DRONE_REQUIRE(parts[i]->xplan->nranks == n_parts && parts[i]->xplan->rank == i,
                      "drone_mp_step_local: part %d carries the plan of rank %d of %d", i, parts[i]->xplan->rank,
                      parts[i]->xplan->nranks);
        DRONE_REQUIRE(parts[i]->kind == parts[0]->kind && parts[i]->device == parts[0]->device,
                      "drone_mp_step_local: parts differ in kind or device");
    }
    return mp_run(parts, is_peval != 0, source_global_id, true, res, stream);
}

int drone_mp_device_arrays(drone_mp *p, void **d_value, int **d_active, int **d_update_by_message) {
    DRONE_REQUIRE(p != nullptr, "drone_mp_device_arrays: NULL job");
    if (d_value) *d_value = p->value;
    if (d_active) *d_active = p->active;
    if (d_update_by_message) *d_update_by_message = p->ubm;
    return DRONE_OK;
}

int drone_mp_values(drone_mp *p, void *h_out, void *stream) {
    DRONE_REQUIRE(p != nullptr && h_out != nullptr, "drone_mp_values: NULL argument");
    if (p->n_local == 0) return DRONE_OK;
    OnDevice dev;
    const int rc = dev.enter(p->device);
    if (rc) return rc;
    DRONE_CUDA(cudaMemcpyAsync(h_out, p->value, sizeof(unsigned) * (size_t)p->n_local, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    DRONE_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return DRONE_OK;
}

}  // extern "C"
