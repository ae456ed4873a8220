// grid_barrier.cuh -- a barrier of all blocks of a cooperative launch.
#pragma once
#include "kernels.cuh"

namespace cudarl {

constexpr unsigned long long GRID_WAIT_NS = 2000000000ull;

// An arrival counter that only grows; the value it starts from is the launch's to know.  Bounded in time: a block that waits two seconds
// records the failure, and everybody leaves.
struct GridBarrier {
    unsigned* counter; Ctl* ctl; unsigned target; unsigned* s_flag;       // s_flag: a word of shared memory
    __device__ __forceinline__ void arrive() {      // this block's writes are visible to whoever sees the arrival
        __syncthreads();
        target += gridDim.x;
        if (threadIdx.x == 0u) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(counter) : "memory");
    }
    __device__ __forceinline__ bool wait() {
        if (threadIdx.x == 0u) {
            unsigned v, ok = 1u;
            unsigned long long t0 = 0ull;
            for (unsigned it = 1u;; ++it) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
                if ((int)(v - target) >= 0) break;
                if ((it & 1023u) == 0u) {
                    unsigned long long now; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                    if (t0 == 0ull) t0 = now;
                    else if (now - t0 > GRID_WAIT_NS) { atomicOr(&ctl->error, ERR_COPY_TIMEOUT); ok = 0u; break; }
                }
            }
            *s_flag = ok;
        }
        __syncthreads();
        return *s_flag != 0u;
    }
    __device__ __forceinline__ bool pass() { arrive(); return wait(); }
};

}  // namespace cudarl
