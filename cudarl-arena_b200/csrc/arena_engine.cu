// arena_engine.cu -- the fused train step for the smallest worlds: the whole world in the shared memory of one block, many steps per
// launch.
//
// A small world is latency, nothing else: in the gather engine (gather_engine.cu) a step is two barriers between blocks and several
// dependent accesses to L2.  Here the table, the counters and the move bytes lie in shared memory, the environments in registers, and
// the barrier is the block's.  The step itself is step_loop.cuh.
//
// What bounds it: one block's issue slots, about 300 instructions per warp and step.  B200, us per step, here / gather engine: one
// environment 0.59 / 3.0, 200 on 20 x 20 cells 1.1 / 4.7, 1,000 on 32 x 32 2.2 / 4.7; 4,096 on 64 x 64 16 / 4.7.  The same spread over
// the distributed shared memory of a cluster was no faster than L2 (4,096 on 64 x 64: 4.4 with 16 blocks; scattered 16-byte accesses to
// other blocks' shared memory are served one by one), nor with a copy of the table in every block (3.9: every update is then stored 8 times).
#include "step_loop.cuh"

namespace cudarl {

constexpr size_t ARENA_MOST = 226u * 1024u;      // dynamic shared memory of a block (227 KB less the static words of step_loop.cuh)
constexpr unsigned ARENA_ENVS = 1024u;
// rows (16 bytes a cell), two rows of counters by step parity (16 bytes each), a move byte
inline size_t arena_bytes(unsigned S) { return (size_t)S * 48u + (S + 15u) / 16u * 16u; }

struct ArenaSpace {
    static constexpr bool ALONE = true;
    float4* rows; unsigned* counters; const unsigned char* mv; unsigned S;
    __device__ __forceinline__ float4 row(unsigned s) const { return rows[s]; }
    __device__ __forceinline__ unsigned moves(unsigned s) const { return mv[s]; }
    __device__ __forceinline__ unsigned add(unsigned par, unsigned idx, unsigned n) const { return atomicAdd(counters + par * 4u * S + idx, n); }
    __device__ __forceinline__ void count(unsigned par, unsigned idx, unsigned n) const { atomicAdd(counters + par * 4u * S + idx, n); }
    __device__ __forceinline__ bool note(unsigned par, unsigned idx) const { return (atomicOr(counters + par * 4u * S + idx, NOTED) & NOTED) != 0u; }
    __device__ __forceinline__ void clear(unsigned par, unsigned idx) const { counters[par * 4u * S + idx] = 0u; }
    __device__ __forceinline__ uint4 counts(unsigned par, unsigned s) const { return reinterpret_cast<const uint4*>(counters)[par * S + s]; }
    __device__ __forceinline__ void store(unsigned idx, float v) const { reinterpret_cast<float*>(rows)[idx] = v; }
    __device__ __forceinline__ void arrive() const {}
    __device__ __forceinline__ bool wait() const { __syncthreads(); return true; }
};

template <unsigned AB, bool PLAIN>
__global__ void __launch_bounds__(AB, 1) k_arena_steps(const __grid_constant__ Params p, const __grid_constant__ StepLaunch l) {
    extern __shared__ __align__(16) unsigned char arena[];
    __shared__ unsigned s_flag;
    if (!may_start(p, &s_flag)) return;
    const unsigned S = p.S;
    float4* const rows = reinterpret_cast<float4*>(arena);
    uint4* const counters = reinterpret_cast<uint4*>(arena) + S;
    unsigned char* const moves = arena + (size_t)S * 48u;
    for (unsigned s = threadIdx.x; s < S; s += AB) {
        rows[s] = p.Q[s]; moves[s] = __ldg(p.gp.mv + s);
        counters[s] = make_uint4(0u, 0u, 0u, 0u); counters[S + s] = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();
    ArenaSpace space{rows, reinterpret_cast<unsigned*>(counters), moves, S};
    run_steps<Home::Registers, AB, PLAIN, true>(p, l, space, l.out, nullptr);
    __syncthreads();
    for (unsigned s = threadIdx.x; s < S; s += AB) p.Q[s] = rows[s];
}

template <unsigned AB>
static bool allow() {
    return cudaFuncSetAttribute((const void*)k_arena_steps<AB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ARENA_MOST) == cudaSuccess &&
           cudaFuncSetAttribute((const void*)k_arena_steps<AB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ARENA_MOST) == cudaSuccess;
}
// One block holds up to 1,024 environments at one per thread; twice that takes longer than the gather engine.
bool arena_plan(Params& p) {
    GatherP& gp = p.gp;
    const unsigned n = p.N ? p.N : 1u;
    if (n > ARENA_ENVS || arena_bytes(p.S) > ARENA_MOST) return false;
    gp.threads = n <= 32u ? 32u : n <= 256u ? 256u : 1024u;
    gp.chunk = gp.threads; gp.grid = 1u; gp.arena = 1u;
    return allow<32u>() && allow<256u>() && allow<1024u>();
}

template <unsigned AB>
static cudaError_t launch_one(const Params& p, const StepLaunch& l, cudaStream_t st) {
    if (plain(p, l)) k_arena_steps<AB, true><<<1, AB, arena_bytes(p.S), st>>>(p, l);
    else             k_arena_steps<AB, false><<<1, AB, arena_bytes(p.S), st>>>(p, l);
    return cudaGetLastError();
}
cudaError_t launch_arena_steps(const Params& p, const StepLaunch& l, cudaStream_t st) {
    return p.gp.threads == 32u ? launch_one<32u>(p, l, st) : p.gp.threads == 256u ? launch_one<256u>(p, l, st) : launch_one<1024u>(p, l, st);
}

}  // namespace cudarl
