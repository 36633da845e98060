// grid_barrier.cuh — barrier among the CTAs of a cooperative launch, with a bounded wait.
#pragma once

#include <cuda_runtime.h>

namespace shg {

// All CTAs that share *bar arrive and wait until it reaches target.  Every store before
// it (of any thread of any CTA) is visible to loads after it that read L2.  False when the wait
// ran out.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target, unsigned long long limit_ns) {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        unsigned v;
        asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned long long t0 = 0;
        for (unsigned it = 0;; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= target) break;
            if ((it & 255) == 255) {
                unsigned long long t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                if (!t0) t0 = t;
                if (t - t0 > limit_ns) {
                    ok = false;
                    break;
                }
            }
        }
    }
    return __syncthreads_and(ok);
}

}  // namespace shg
