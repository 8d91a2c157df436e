// grid_barrier.cuh -- a barrier among the CTAs of one cooperative launch (or a
// group of them), with a bounded wait.
#pragma once

#include <cstdint>

#include "ltl_kernels.h"

namespace ltl {

// State of a barrier in device memory.  `arrived` only ever grows: it is a
// multiple of the group's size whenever no launch uses it, so a launch needs no
// reset and a CTA finds the current round by rounding down what it reads before
// its own first arrival.  Zero it when the group's size changes.
struct GridBarrier {
    unsigned long long arrived;
};

// One CTA's view.  All threads of the CTA call wait(); it returns false once the
// wait has run out (the CTA should then return: the others will run out too), and
// sets *err.  That word stays set until the host has read it; the barrier is at some
// count in between then, and has to be zeroed before the next launch that uses it.
struct GridBarrierWait {
    unsigned long long* arrived;
    unsigned long long target;
    unsigned long long limit_ns;
    unsigned int ctas;

    __device__ __forceinline__ GridBarrierWait(GridBarrier* b, unsigned int ctas_, const BarrierLimit& limit)
        : arrived(&b->arrived), limit_ns(limit.ns), ctas(ctas_ > 1 ? ctas_ + limit.missing : 1u) {
        if (threadIdx.x == 0 && ctas > 1) {
            unsigned long long now;
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(arrived) : "memory");
            target = now - now % ctas;
        }
    }
    __device__ __forceinline__ bool wait(unsigned int* err) {
        int late = 0;
        __syncthreads();
        if (ctas > 1) {
            if (threadIdx.x == 0) {
                // release: this CTA's writes (ordered by the CTA barrier above) are
                // visible to whoever acquires the count
                asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(arrived) : "memory");
                target += ctas;
                unsigned long long now, t0 = 0, t;
                int tries = 0;
                while (true) {
                    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(arrived) : "memory");
                    if (now >= target) break;
                    if ((++tries & 1023) == 0) {
                        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                        if (t0 == 0) t0 = t;
                        if (t - t0 > limit_ns) {
                            *(volatile unsigned int*)err = 1u;
                            late = 1;
                            break;
                        }
                    }
                }
            }
            late = __syncthreads_or(late);
        }
        return late == 0;
    }
};

}  // namespace ltl
