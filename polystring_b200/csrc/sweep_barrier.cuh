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
// polled kBarrierPolls times in vain, which it tells the chains' other CTAs (err) and the
// host (*notice), or another CTA has.  The limit is a constant and a launch that is to give
// up at once (hasty, a launch parameter) has a branch of its own: with the limit in a
// register or in shared memory a barrier takes 45 to 110 ns longer (32^3 OS2 5.85 us a
// step, 128 x 352 13.8 to 14.0; as here 5.71 and 13.57).
__device__ __forceinline__ bool chain_barrier(unsigned* count, int* err, int* const* notice, int hasty, unsigned target) {
    __shared__ int stop;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        red_release_add(count, 1u);
        long long spins = 0;
        if (hasty && ld_acquire(count) < target) {
            atomicExch(err, 2);
            *((volatile int*)*notice) = 2;
            s = 1;
        } else {
            while (ld_acquire(count) < target) {
                if ((spins & 63) == 63 && *((volatile int*)err)) { s = 1; break; }
                if (++spins > kBarrierPolls) {
                    atomicExch(err, 2);
                    *((volatile int*)*notice) = 2;
                    s = 1;
                    break;
                }
            }
        }
        stop = s;
    }
    __syncthreads();
    return stop == 0;
}

}  // namespace ps
