// A barrier over all blocks of a cooperative launch, for the kernels that run many steps in one launch.  It is bounded: a
// block whose wait runs out says so in `failed`, which ends every other block's wait too, and the kernel returns.
#pragma once

#include "common.cuh"

#include <cstdlib>

namespace drone {

struct GridBarrier {
    unsigned arrived;      // blocks that reached a barrier, over all barriers of the launch, counted modulo 2^32
    int failed;            // a wait ran out
};

// How often a block looks at the count before it gives up: kBarrierPolls (about five seconds), or DRONE_BARRIER_POLLS, read when
// a handle is made (0: every block gives up at its first barrier, which is how the failure is tested).
constexpr unsigned kBarrierPolls = 1u << 23;
inline unsigned barrier_polls() {
    const char *v = getenv("DRONE_BARRIER_POLLS");
    return v && *v ? (unsigned)strtoul(v, nullptr, 10) : kBarrierPolls;
}

// What `arrived` starts at: 0, or DRONE_BARRIER_START, read when a handle is made (a start just below 2^32 takes a short run
// over the end of the count, which otherwise 14 million iterations on a full grid reach).
inline unsigned barrier_start() {
    const char *v = getenv("DRONE_BARRIER_START");
    return v && *v ? (unsigned)strtoul(v, nullptr, 10) : 0u;
}

// The two halves of a barrier, for a block with work between them.  One thread of every block arrives, after a block-wide
// barrier behind what the others are to see; then every thread of the block waits, which is false when a wait ran out (in some
// block): then everybody returns.  `phase`: what `arrived` has to reach, at first its start.  The count only grows, so that a
// barrier is one atomic and one comparison modulo 2^32 (the blocks of a grid are far closer together than 2^31); a count of 64
// bits took 0.2 us more per barrier.
__device__ inline void grid_arrive(GridBarrier *b) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(&b->arrived) : "memory");
}
__device__ inline bool grid_wait(GridBarrier *b, unsigned &phase, unsigned poll_limit) {
    __shared__ int ok;
    phase += gridDim.x;
    if (threadIdx.x == 0) {
        int failed = 0;
        for (unsigned polls = 0;; ) {
            unsigned seen;
            if (polls >= poll_limit) {
                atomicExch(&b->failed, 1);
                failed = 1;
                break;
            }
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&b->arrived) : "memory");
            if ((int)(seen - phase) >= 0) break;
            if ((++polls & 255u) == 0 && (failed = *(volatile int *)&b->failed) != 0) break;
        }
        ok = failed ? 0 : 1;
    }
    __syncthreads();
    return ok != 0;
}

// Both at once.
__device__ inline bool grid_barrier(GridBarrier *b, unsigned &phase, unsigned poll_limit) {
    __syncthreads();
    if (threadIdx.x == 0) grid_arrive(b);
    return grid_wait(b, phase, poll_limit);
}

}  // namespace drone
