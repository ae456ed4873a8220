// gather_engine.cu -- the fused train step for worlds whose table stays in L2: many steps per launch, one thread per environment.
//
// The tile engine (tile_engine.cu) streams the whole table through shared memory in every step, one warp per tile.  Where the table
// fits L2 that is not needed, and where the population bunches up -- everybody on the few paths to the goals, late in training -- a
// step lasts as long as the warp with the fullest tile: 256 x 256 cells with 65,536 environments went from 11 us a step to 116.
// Here the environments are spread evenly over the threads of ONE cooperative launch that runs many steps (step_loop.cuh), with the
// table, the counters and the barrier in global memory.
//
// A population that fits the threads stays in registers for the whole launch, a larger one is streamed from shared memory (24 bytes an
// environment), the largest from global memory.  Up to 16,384 environments run in the blocks of one cluster, whose barrier takes 0.28 us
// where one of the grid takes 1.3 - 2.4 (patch_engine.cu takes most worlds of up to 110,000, in launches of 16 or 32 steps and more).  Large populations are dealt to the
// blocks by cell every 64 steps (deal_by_cell), whether those are one call or many.
//
// What bounds it (B200): small populations, the chain of a step -- two barriers and four dependent accesses to L2 (300 - 500 ns each with
// the whole GPU at it): 256 x 256 cells with 65,536 environments 6.0 us a step.  Large ones, the rate of atomics on L2: about 117 G per
// second, 9 of the 22 us that 1,048,576 environments on 1024 x 1024 cells take (packing the counters into 16 or 8 bits changed little:
// it is atomics, not sectors).
//
// Reference semantics: those of tile_engine.cu.
#include "global_table.cuh"
#include <cstring>

namespace cudarl {

// Deal the environments to the blocks by cell: the records of l.in, sorted by lines of eight cells (128 bytes of the table) in the
// order of 8 x 8 tiles, into l.out.  The lanes of a warp then stand on a few lines instead of on 32: the rows, counters and move
// bytes they touch come in a few wide accesses.  A counting sort between barriers of the grid; the order within a line does not matter
// (nor does any order: results never depend on it).
template <unsigned THREADS>
__device__ bool deal_by_cell(const Params& p, const StepLaunch& l, GridSpace& space) {
    __shared__ unsigned s_warp[33], s_sum;
    const GatherP& gp = p.gp;
    const unsigned tid = threadIdx.x, first = min(blockIdx.x * l.chunk, p.N), last = min(first + l.chunk, p.N);
    const unsigned per = (gp.nbins + gridDim.x - 1u) / gridDim.x, b0 = min(blockIdx.x * per, gp.nbins), b1 = min(b0 + per, gp.nbins);
    auto key = [&](const int4 r) -> unsigned { return ((((unsigned)r.y >> 3) * gp.bins_x + ((unsigned)r.x >> 3)) << 3) | ((unsigned)r.y & 7u); };
    const unsigned lane = tid & 31u;
    for (unsigned i0 = first; i0 < last; i0 += THREADS) {          // one addition for all of a warp that stand on one line: everybody on
                                                                   // one start cell is 32 times fewer on one word (1,048,576, the first step 1,357 -> 647 us; 4,194,304 5,259 -> 2,559)
        const unsigned i = i0 + tid, k = i < last ? key(l.in[i]) : NOBODY;
        const unsigned mates = __match_any_sync(FULL, k), leader = (unsigned)__ffs((int)mates) - 1u;
        unsigned base = 0u;
        if (lane == leader && k != NOBODY) base = atomicAdd(gp.bins + k, (unsigned)__popc(mates));
        base = __shfl_sync(FULL, base, leader);
        if (k != NOBODY) gp.rank[i] = base + (unsigned)__popc(mates & ((1u << lane) - 1u));
    }
    space.arrive(); if (!space.wait()) return false;
    unsigned sum = 0u;
    for (unsigned k = b0 + tid; k < b1; k += THREADS) sum += gp.bins[k];
    if (tid == 0u) s_sum = 0u;
    __syncthreads();
    sum = __reduce_add_sync(FULL, sum);
    if ((tid & 31u) == 0u && sum) atomicAdd(&s_sum, sum);
    __syncthreads();
    if (tid == 0u) gp.part[blockIdx.x] = s_sum;
    space.arrive(); if (!space.wait()) return false;
    unsigned before = 0u;
    for (unsigned k = tid; k < blockIdx.x; k += THREADS) before += gp.part[k];
    if (tid == 0u) s_sum = 0u;
    __syncthreads();
    before = __reduce_add_sync(FULL, before);
    if ((tid & 31u) == 0u && before) atomicAdd(&s_sum, before);
    __syncthreads();
    unsigned carry = s_sum;
    for (unsigned k0 = b0; k0 < b1; k0 += THREADS) {
        const unsigned k = k0 + tid, v = k < b1 ? gp.bins[k] : 0u;
        unsigned total = 0u;
        const unsigned ex = block_scan_excl(v, s_warp, &total);
        if (k < b1) gp.bins[k] = carry + ex;
        carry += total;
    }
    space.arrive(); if (!space.wait()) return false;
    for (unsigned i = first + tid; i < last; i += THREADS) { const int4 r = l.in[i]; l.out[gp.bins[key(r)] + gp.rank[i]] = r; }
    space.arrive(); if (!space.wait()) return false;
    for (unsigned k = b0 + tid; k < b1; k += THREADS) gp.bins[k] = 0u;
    return true;
}

template <Home HOME, unsigned THREADS, bool PLAIN, bool OWNERS>
__global__ void __launch_bounds__(THREADS, 1) k_gather_steps(const __grid_constant__ Params p, const __grid_constant__ StepLaunch l) {
    extern __shared__ __align__(16) unsigned char arrays[];
    __shared__ unsigned s_flag;
    if (!may_start(p, &s_flag)) return;
    GridSpace space(p, p.gp.barrier, l.barrier_base, &s_flag);
    if (l.in != l.out && !deal_by_cell<THREADS>(p, l, space)) return;
    run_steps<HOME, THREADS, PLAIN, OWNERS>(p, l, space, l.out, arrays);
}
__global__ void __launch_bounds__(BLOCK) k_gather_export(Params p, const int4* __restrict__ work) {
    const unsigned i = blockIdx.x * BLOCK + threadIdx.x;
    if (i < p.N) { const int4 r = work[i]; if ((unsigned)r.w < p.N) p.st[r.w] = r; }
}

// The same with all blocks in one cluster: its barrier takes 0.28 us.
template <unsigned CB, bool PLAIN>
__global__ void __launch_bounds__(CB, 1) k_cluster_steps(const __grid_constant__ Params p, const __grid_constant__ StepLaunch l) {
    __shared__ unsigned s_flag;
    if (!may_start(p, &s_flag)) return;
    ClusterSpace space{p};
    run_steps<Home::Registers, CB, PLAIN, true>(p, l, space, l.out, nullptr);
}

// ------------------------------------------------------------------------------------------------
// The move byte of every cell (see MoveColumn in rules.cuh), row by row.
__global__ void __launch_bounds__(BLOCK) k_gather_moves(Params p, unsigned char* __restrict__ mv) {
    for (unsigned s = blockIdx.x * BLOCK + threadIdx.x; s < p.S; s += gridDim.x * BLOCK) {
        const int y = (int)(s / (unsigned)p.W), x = (int)(s - (unsigned)y * (unsigned)p.W);
        const unsigned own = p.cw[s];
        unsigned b = 0u;
        for (int a = 0; a < 4; ++a) {
            const int nx = x + (a == 1) - (a == 3), ny = y + (a == 2) - (a == 0);
            unsigned cls = CW_OBST;
            if (nx >= 0 && nx < p.W && ny >= 0 && ny < p.H) cls = p.cw[(unsigned)ny * (unsigned)p.W + (unsigned)nx];
            const bool blocked = (cls & CW_OBST) != 0u;
            if (blocked) b |= 1u << a;
            if ((blocked ? own : cls) & CW_GOAL) b |= 16u << a;
        }
        mv[s] = (unsigned char)b;
    }
}
void launch_gather_moves(const Params& p, cudaStream_t st) {
    const unsigned b = (p.S + BLOCK - 1u) / BLOCK;
    k_gather_moves<<<b < 2368u ? b : 2368u, BLOCK, 0, st>>>(p, p.gp.mv);
}

// How the population is spread over the launch: one environment per thread in registers while the blocks of one launch hold them all,
// else streamed from shared memory, or from global memory where that is too small.
constexpr unsigned SHARED_MOST = 200u * 1024u;
void gather_plan(Params& p) {
    GatherP& gp = p.gp;
    const unsigned n = p.N ? p.N : 1u, s = p.sms;
    if (n <= 16u * 1024u) {
        gp.cluster = 1u;
        gp.threads = n <= 16u * 256u ? 256u : n <= 16u * 512u ? 512u : 1024u;
        gp.chunk = gp.threads; gp.grid = (n + gp.chunk - 1u) / gp.chunk;
        return;
    }
    gp.threads = n <= 512u * s ? 512u : 1024u;
    gp.deal_every = gp.threads == 512u ? 0u : 64u;
    gp.home = gp.threads * s >= n ? 0u : 1u;
    gp.chunk = gp.home == 0u ? gp.threads : ((n + s - 1u) / s + 31u) / 32u * 32u;
    if (gp.home && (size_t)gp.chunk * STATE_BYTES > SHARED_MOST) gp.home = 2u;
    gp.grid = (n + gp.chunk - 1u) / gp.chunk;
    gp.bins_x = ((unsigned)p.W + 7u) / 8u; gp.nbins = gp.bins_x * (((unsigned)p.H + 7u) / 8u) * 8u;
}
unsigned gather_barriers(const StepLaunch& l) { return 2u * l.steps + (l.in != l.out ? 4u : 0u) + (l.eps_mode == 2 ? 1u : 0u); }
void launch_gather_export(const Params& p, const int4* work, cudaStream_t st) {
    if (p.N) k_gather_export<<<(p.N + BLOCK - 1u) / BLOCK, BLOCK, 0, st>>>(p, work);
}

template <unsigned CB, bool PLAIN>
static cudaError_t launch_cluster(const Params& p, const StepLaunch& l, cudaStream_t st) {
    auto* const fn = k_cluster_steps<CB, PLAIN>;
    cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(p.gp.grid); cfg.blockDim = dim3(CB); cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.gp.grid; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, p, l);
}
template <Home HOME, unsigned THREADS, bool OWNERS, bool PLAIN>
static cudaError_t launch_gather(const Params& p, const StepLaunch& l, cudaStream_t st) {
    const void* fn = (const void*)k_gather_steps<HOME, THREADS, PLAIN, OWNERS>;
    const size_t bytes = HOME == Home::Shared ? (size_t)p.gp.chunk * STATE_BYTES : 0u;
    if (HOME == Home::Shared) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SHARED_MOST);
        if (e != cudaSuccess) return e;
    }
    void* args[2] = {const_cast<Params*>(&p), const_cast<StepLaunch*>(&l)};
    return cudaLaunchCooperativeKernel(fn, dim3(p.gp.grid), dim3(THREADS), args, bytes, st);
}
template <bool PLAIN>
static cudaError_t launch(const Params& p, const StepLaunch& l, cudaStream_t st) {
    const GatherP& gp = p.gp;
    if (gp.cluster) return gp.threads == 256u ? launch_cluster<256u, PLAIN>(p, l, st) : gp.threads == 512u ? launch_cluster<512u, PLAIN>(p, l, st) : launch_cluster<1024u, PLAIN>(p, l, st);
    if (gp.threads == 512u) return launch_gather<Home::Registers, 512u, true, PLAIN>(p, l, st);
    return gp.home == 0u ? launch_gather<Home::Registers, 1024u, false, PLAIN>(p, l, st) : gp.home == 1u ? launch_gather<Home::Shared, 1024u, false, PLAIN>(p, l, st)
                                                                                       : launch_gather<Home::Global, 1024u, false, PLAIN>(p, l, st);
}
cudaError_t launch_gather_steps(const Params& p, const StepLaunch& l, cudaStream_t st) { return plain(p, l) ? launch<true>(p, l, st) : launch<false>(p, l, st); }

}  // namespace cudarl
