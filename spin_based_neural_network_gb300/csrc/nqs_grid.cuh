// Bounded grid-wide barrier of the cooperative kernels.
#pragma once
#include <stdint.h>

namespace nqs {

// Polls a grid barrier waits before it gives up (raising *err = 2).  A device variable (one per
// translation unit) so that graph replays read the current value; nqs_gpu_set_barrier_budget()
// lowers it for the tests of the timeout path.
static __device__ unsigned g_barrier_budget = 1u << 24;

// A monotonic arrival counter (bar[0], cleared at every launch): the arrival that returns
// old belongs to barrier instance old / count, which is passed once the counter reaches
// (old / count + 1) * count, so no reset and no second word is needed (a CTA can only
// arrive at the next instance after all arrivals of this one).  Ordering: the block
// barrier, then an acq_rel fence at GPU scope around the relaxed atomic and the polls.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, int *err, unsigned count) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned budget = *(volatile unsigned *)&g_barrier_budget;
        unsigned old;
        asm volatile("fence.acq_rel.gpu;\n\tatom.relaxed.gpu.global.add.u32 %0, [%1], 1;"
                     : "=r"(old) : "l"(bar) : "memory");
        const unsigned target = (old / count + 1u) * count;
        uint32_t it = 0;
        for (;;) {
            unsigned cur;
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(bar) : "memory");
            if ((int)(cur - target) >= 0) break;
            if (++it > budget) {
                atomicExch(err, 2);
                break;
            }
            if ((it & 31) == 0) {                       // the error word every 32nd poll only
                if (*((volatile int *)err)) break;
                if (it > 256) __nanosleep(32);
            }
        }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        s_ok = *((volatile int *)err) == 0;
    }
    __syncthreads();
    return s_ok != 0;                                 // one answer for the whole CTA
}

}  // namespace nqs
