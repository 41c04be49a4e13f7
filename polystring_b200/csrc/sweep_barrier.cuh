// sweep_barrier.cuh -- the barrier in memory over the CTAs of one chain, for sweeps
// whose CTAs are all resident (cooperative launches).
#pragma once

#include "real_sweep.h"

namespace ps {

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Counts arrivals until target.  Returns false when the sweep must stop: this CTA has
// polled p.polls times in vain, which it tells the chains' other CTAs (p.err) and the
// host (p.notice), or another CTA has.
__device__ __forceinline__ bool chain_barrier(const RealProblem& p, unsigned* count, unsigned target) {
    __shared__ int stop;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        red_release_add(count, 1u);
        int spins = 0;
        const int polls = p.polls;
        while (ld_acquire(count) < target) {
            if ((spins & 63) == 63 && *((volatile int*)p.err)) { s = 1; break; }
            if (++spins > polls) {
                atomicExch(p.err, 2);
                *((volatile int*)p.notice) = 2;
                s = 1;
                break;
            }
        }
        stop = s;
    }
    __syncthreads();
    return stop == 0;
}

}  // namespace ps
