// Bounded waits of kernels whose blocks wait on one another.
#pragma once

#include <cuda_runtime.h>

namespace afd {

constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // 2 s

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Every copy of this thread to shared memory (cp.async) has landed: before a
// block leaves early.
__device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Grid barrier on a counter that every block raises once per step; bounded
// like every wait. The fences make the step's stores visible to all blocks
// and drop the SM's cached copies of what they replaced.
__device__ __forceinline__ bool grid_barrier(unsigned int* bar, unsigned int target, int* flag) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned int v;
        int good = 1;
        unsigned long long t0 = 0;
        for (int n = 0;; ++n) {
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((n & 63) == 63) {
                const unsigned long long now = global_ns();
                if (t0 == 0) t0 = now;
                else if (now - t0 > kWaitLimitNs) {
                    good = 0;
                    atomicOr(flag, 2);
                    break;
                }
            }
        }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

}  // namespace afd
