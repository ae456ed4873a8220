// global_table.cuh -- the Spaces of step_loop.cuh with the table and the counters in global memory: a barrier of the whole grid, or of one cluster.
#pragma once
#include "step_loop.cuh"
#include "grid_barrier.cuh"

namespace cudarl {

// The table and the counters in global memory.
struct GlobalTable {
    const Params& p;
    __device__ __forceinline__ float4 row(unsigned s) const { return p.Q[s]; }
    __device__ __forceinline__ unsigned moves(unsigned s) const { return __ldg(p.gp.mv + s); }
    __device__ __forceinline__ unsigned add(unsigned par, unsigned idx, unsigned n) const { return atomicAdd(p.gp.cnt[par] + idx, n); }
    __device__ __forceinline__ void count(unsigned par, unsigned idx, unsigned n) const { atomicAdd(p.gp.cnt[par] + idx, n); }
    __device__ __forceinline__ bool note(unsigned par, unsigned idx) const { return (atomicOr(p.gp.cnt[par] + idx, NOTED) & NOTED) != 0u; }
    __device__ __forceinline__ void clear(unsigned par, unsigned idx) const { p.gp.cnt[par][idx] = 0u; }
    __device__ __forceinline__ uint4 counts(unsigned par, unsigned s) const { return *reinterpret_cast<const uint4*>(p.gp.cnt[par] + 4u * s); }
    __device__ __forceinline__ void store(unsigned idx, float v) const { reinterpret_cast<float*>(p.Q)[idx] = v; }
};
struct GridSpace : GlobalTable {
    GridBarrier barrier;
    __device__ __forceinline__ GridSpace(const Params& q, unsigned* counter, unsigned base, unsigned* flag) : GlobalTable{q}, barrier{counter, q.ctl, base, flag} {}
    __device__ __forceinline__ void arrive() { barrier.arrive(); }
    __device__ __forceinline__ bool wait() { return barrier.wait(); }
};

// With all blocks in one cluster: its barrier takes 0.28 us.
struct ClusterSpace : GlobalTable {
    __device__ __forceinline__ void arrive() const { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
    __device__ __forceinline__ bool wait() const { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); return true; }
};

}  // namespace cudarl
