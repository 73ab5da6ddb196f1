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

constexpr unsigned kBarrierPolls = 1u << 23;   // about five seconds

// What `arrived` starts at: 0, or DRONE_BARRIER_START, read when a handle is made (a start just below 2^32 takes a short run
// over the end of the count, which otherwise 14 million iterations on a full grid reach).
inline unsigned barrier_start() {
    const char *v = getenv("DRONE_BARRIER_START");
    return v && *v ? (unsigned)strtoul(v, nullptr, 10) : 0u;
}

// Every thread of the grid arrives; false when a wait ran out (in some block), then everybody returns.  `phase`: what
// `arrived` has to reach, at first its start.  The count only grows, so that a barrier is one atomic and one comparison
// modulo 2^32 (the blocks of a grid are far closer together than 2^31); a count of 64 bits took 0.2 us more per barrier.
__device__ inline bool grid_barrier(GridBarrier *b, unsigned &phase) {
    __shared__ int ok;
    phase += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&b->arrived, 1u);
        unsigned seen = 0, polls = 0;
        int failed = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&b->arrived) : "memory");
            if (++polls >= kBarrierPolls) atomicExch(&b->failed, 1);
            if ((polls & 255u) == 0) failed = *(volatile int *)&b->failed;
        } while ((int)(seen - phase) < 0 && !failed);
        __threadfence();
        ok = failed ? 0 : 1;
    }
    __syncthreads();
    return ok != 0;
}

}  // namespace drone
