// rollout.cu -- the greedy rollout of every environment (evaluation): sm_100a kernels.
//
// The table does not change during a rollout, so the greedy policy is a map from cells to cells, and the length of an episode is
// the length of a path in that map.  Nobody has to walk it cell by cell:
//
//   k_rollout_tiles   one block per 64 x 64 (small grids: 32 x 32) cells folds the policy of its tile by pointer doubling in shared memory: for every
//                     cell the number of steps until the path ends on a goal or leaves the tile (and where), or "never" when it
//                     runs in a circle inside the tile.  One 4-byte word per cell.
//   k_rollout_walk    one thread per environment draws its start cell and hops from tile to tile over those words; a path that
//                     comes back to an earlier tile entry (Brent's cycle search over the hops) never ends.
//
// What bounds it: k_rollout_tiles streams the table once (16 bytes in, 4 out per cell) and looks up one word in shared memory per cell and round,
// until a round finds no path to end; k_rollout_walk makes a few scattered 4-byte look-ups per environment, one after the other.  B200,
// 4096 x 4096 cells, 4,194,304 environments, 1000 steps: the call 171 us, of which 94 + 74 under ncu (doubling to the last round 138 us; one environment per thread, start cells
// looked up in the cell words 89 us); the walk over single cells this replaces took 13.6 ms.  256 x 256 cells, 65,536 environments: one call after
// the other 17.8 us each (a call from Python with its own overhead 21), 24.4 with 64 x 64 tiles (16 blocks, 8 cells per thread and 3 more rounds than the 64 blocks of 32 x 32)
// and the walk started after the last fold had ended.
//
// Reference semantics: src/train.py:262-311 (evaluate), first-max argmax src/q_learning.cu:196-206.
#include "kernels.cuh"
#include "rules.cuh"
#include <cstring>

namespace cudarl {

// Word of a cell.  While the tile is folded: kind LIVE, bits 0-11 the cell reached after 2^round steps.  Final: EXIT with the number
// of steps in bits 0-12, the edge it leaves by (0 up, 1 right, 2 down, 3 left) in bits 22-23 and the place along it in bits 16-21;
// GOAL with the number of steps; or TRAPPED.  Bit 29: an obstacle or a goal, where no episode starts.  A path without a circle has at most 4096 steps inside a tile.
constexpr unsigned RT_ROWS = 8u;                 // rows of a tile that its threads take at a time
// Rows of tiles in a launch's second dimension, which ends at 65,535, while a grid's height ends at 2^28; the third takes the rest.
constexpr unsigned GRID_ROWS = 32768u;
constexpr unsigned KIND_LIVE = 0u, KIND_EXIT = 1u << 30, KIND_GOAL = 2u << 30, KIND_MASK = 3u << 30, TRAPPED = 3u << 30, NO_START = 1u << 29, STEPS_MASK = 0x1FFFu;

template <unsigned RT_SHIFT>
// (32 registers, so that an SM is full: with 38 it held three blocks of 64 x 64 cells instead of four, 4096 x 4096 cells 173 -> 180 us; 171 now)
__global__ void __launch_bounds__(RT_ROWS << RT_SHIFT, 2048u / (RT_ROWS << RT_SHIFT)) k_rollout_tiles(const __grid_constant__ Params p, unsigned* __restrict__ hop) {
    constexpr unsigned RT = 1u << RT_SHIFT, RT_CELLS = RT * RT, RT_THREADS = RT * RT_ROWS, RT_PER = RT_CELLS / RT_THREADS;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");       // the walk's blocks may take the slots that free up, and draw
    __shared__ unsigned s_w[RT_CELLS];
    const int x0 = (int)(blockIdx.x << RT_SHIFT), y0 = (int)((blockIdx.z * gridDim.y + blockIdx.y) << RT_SHIFT);
    unsigned cur[RT_PER];
    const unsigned lx = threadIdx.x & (RT - 1u), ly0 = threadIdx.x >> RT_SHIFT;          // a thread's cells lie below one another, 8 rows apart
    const int x = x0 + (int)lx;
    const float4* const q = p.Q + (size_t)(y0 + (int)ly0) * (size_t)p.W + (size_t)x;
    const MoveColumn moves(p, (unsigned)x);
    const unsigned short* const cw = p.cw + (size_t)(y0 + (int)ly0) * (size_t)p.W + (size_t)x;
    unsigned no_start = 0u;
    const bool inside = x0 + (int)RT <= p.W && y0 + (int)RT <= p.H;                       // the same for the whole block
#pragma unroll
    for (unsigned k = 0; k < RT_PER; ++k) {
        const unsigned ly = ly0 + k * RT_ROWS, ic = (ly << RT_SHIFT) | lx;
        const int y = y0 + (int)ly;
        unsigned w = KIND_LIVE | ic;
        if (inside || (x < p.W && y < p.H)) {
            const float4 row = __ldcs(q + (size_t)(k * RT_ROWS) * (size_t)p.W);
            const unsigned mvb = moves.at((unsigned)y);
            if (__ldcs(cw + (size_t)(k * RT_ROWS) * (size_t)p.W) & (CW_OBST | CW_GOAL)) no_start |= NO_START >> k;
            const unsigned a = (unsigned)argmax4(row), mv = mvb >> a;
            if (mv & 16u) w = KIND_GOAL | 1u;
            else if (!(mv & 1u)) {
                const unsigned mx = lx + (a == 1u) - (a == 3u), my = ly + (a == 2u) - (a == 0u);       // wraps when the move leaves the tile
                w = (mx | my) < RT ? (KIND_LIVE | (my << RT_SHIFT) | mx) : (KIND_EXIT | (a << 22) | (((a & 1u) ? ly : lx) << 16) | 1u);
            }
        }
        cur[k] = w; s_w[ic] = w;
    }
    __syncthreads();
    for (unsigned len = 1u; len <= RT_CELLS; len <<= 1) {
        bool found = false;
#pragma unroll
        for (unsigned k = 0; k < RT_PER; ++k) {
            if ((cur[k] & KIND_MASK) != KIND_LIVE) continue;
            const unsigned w = s_w[cur[k]], nw = (w & KIND_MASK) == KIND_LIVE ? w : w + len;
            found |= nw != w;
            cur[k] = nw;
        }
        // No path was found to end: none of the rest does.  (Had a live cell a way out, some cell on that way would be between 1 and 2 times
        // `len` steps from its end, and would have found it in this round.)
        if (!__syncthreads_or(found)) break;
#pragma unroll
        for (unsigned k = 0; k < RT_PER; ++k) s_w[k * RT_THREADS + threadIdx.x] = cur[k];
        __syncthreads();
    }
    unsigned* const out = hop + (size_t)(y0 + (int)ly0) * (size_t)p.W + (size_t)x;
#pragma unroll
    for (unsigned k = 0; k < RT_PER; ++k) {
        const unsigned w = ((cur[k] & KIND_MASK) == KIND_LIVE ? TRAPPED : cur[k]) | ((no_start << k) & NO_START);
        if (inside || (x < p.W && y0 + (int)(ly0 + k * RT_ROWS) < p.H)) out[(size_t)(k * RT_ROWS) * (size_t)p.W] = w;
    }
}

// (no read-only loads: the words are written while the walk's first instructions already run)
__device__ __forceinline__ unsigned ld_word(const unsigned* p) { unsigned v; asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p)); return v; }
// A start cell as sample_start draws it, and its word, which says whether an episode may start there.
__device__ __forceinline__ unsigned walk_start(const Params& p, const unsigned* __restrict__ hop, unsigned gi, unsigned long long nonce, unsigned& word) {
    if (p.start_mode == 2) {
#pragma unroll 1
        for (unsigned k = 0; k < 16u; ++k) {
            const U4 w = philox4x32_10(gi, k, (unsigned)nonce, (unsigned)(nonce >> 32), p.k0, p.k1 ^ TAG_EVAL);
            unsigned c;
            c = __umulhi(w.x, p.S); word = ld_word(hop + c); if (!(word & NO_START)) return c;
            c = __umulhi(w.y, p.S); word = ld_word(hop + c); if (!(word & NO_START)) return c;
            c = __umulhi(w.z, p.S); word = ld_word(hop + c); if (!(word & NO_START)) return c;
            c = __umulhi(w.w, p.S); word = ld_word(hop + c); if (!(word & NO_START)) return c;
        }
    }
    const unsigned c = p.start_mode == 2 ? p.fallback_start : p.start_cell;
    word = ld_word(hop + c);
    return c;
}

// EPT environments per thread: their first look-ups are on the way at the same time.
template <unsigned EPT, unsigned RT_SHIFT>
__global__ void __launch_bounds__(BLOCK) k_rollout_walk(const __grid_constant__ Params p, const unsigned* __restrict__ hop, unsigned max_steps,
                                                        unsigned long long nonce, Handover h) {
    constexpr unsigned RT = 1u << RT_SHIFT;
    __shared__ unsigned s_reached; __shared__ unsigned long long s_steps;
    if (threadIdx.x == 0) { s_reached = 0u; s_steps = 0ull; }
    __syncthreads();
    const unsigned i0 = blockIdx.x * (BLOCK * EPT) + threadIdx.x;
    unsigned cell[EPT], word[EPT];
#pragma unroll
    for (unsigned k = 0; k < EPT; ++k) {
        const unsigned i = i0 + k * BLOCK;
        cell[k] = p.start_mode == 2 ? __umulhi(philox4x32_10(p.env_offset + i, 0u, (unsigned)nonce, (unsigned)(nonce >> 32), p.k0, p.k1 ^ TAG_EVAL).x, p.S) : p.start_cell;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");                    // the words are written
#pragma unroll
    for (unsigned k = 0; k < EPT; ++k) word[k] = ld_word(hop + cell[k]);
    unsigned nr = 0u; unsigned long long sum = 0ull;
#pragma unroll
    for (unsigned k = 0; k < EPT; ++k) {
        const unsigned i = i0 + k * BLOCK;
        if (i >= p.N) continue;
        unsigned s = cell[k], w = word[k];
        if (p.start_mode == 2 && (w & NO_START)) s = walk_start(p, hop, p.env_offset + i, nonce, w);
        unsigned steps = 0u, y = s / (unsigned)p.W, x = s - y * (unsigned)p.W;
        unsigned cx = x, cy = y, hops = 0u, limit = 1u;      // the entry the path is compared with, moved up at 1, 3, 7, 15, ... hops
        for (;;) {
            if ((w & KIND_MASK) == TRAPPED) { steps = max_steps; break; }
            steps += w & STEPS_MASK;
            if ((w & KIND_MASK) == KIND_GOAL) { if (steps <= max_steps) ++nr; else steps = max_steps; break; }
            if (steps >= max_steps) { steps = max_steps; break; }
            const unsigned e = (w >> 22) & 3u, at = (w >> 16) & (RT - 1u), tx = x & ~(RT - 1u), ty = y & ~(RT - 1u);
            x = (e & 1u) ? (e == 1u ? tx + RT : tx - 1u) : tx + at;
            y = (e & 1u) ? ty + at : (e == 2u ? ty + RT : ty - 1u);
            if (x == cx && y == cy) { steps = max_steps; break; }
            if (++hops == limit) { cx = x; cy = y; hops = 0u; limit <<= 1; }
            w = ld_word(hop + (size_t)y * (size_t)p.W + (size_t)x);
        }
        sum += steps;
    }
    nr = __reduce_add_sync(FULL, nr);
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
    if ((threadIdx.x & 31u) == 0u) { if (nr) atomicAdd(&s_reached, nr); atomicAdd(&s_steps, sum); }
    __syncthreads();
    Ctl* const c = p.ctl;
    if (threadIdx.x == 0u) { if (s_reached) atomicAdd(&c->eval_reached, (unsigned long long)s_reached); atomicAdd(&c->eval_steps, s_steps); }
    if (last_to_finish<false>(p)) {                          // the totals go to the host, the counters back to zero
        box_put64(h, 1u, atomicExch(&c->eval_reached, 0ull)); box_put64(h, 3u, atomicExch(&c->eval_steps, 0ull));
        box_put_error(p, h);
    }
}

template <unsigned RT_SHIFT>
static cudaError_t launch_tiled(const Params& p, unsigned* hop, unsigned max_steps, unsigned long long nonce, Handover h, cudaStream_t st) {
    constexpr unsigned RT = 1u << RT_SHIFT;
    const unsigned tiles_x = ((unsigned)p.W + RT - 1u) / RT, tiles_y = ((unsigned)p.H + RT - 1u) / RT;
    const unsigned layers = (tiles_y + GRID_ROWS - 1u) / GRID_ROWS;
    const dim3 tiles(tiles_x, (tiles_y + layers - 1u) / layers, layers);     // (a tile beyond the last row has no cell of the grid in it)
    k_rollout_tiles<RT_SHIFT><<<tiles, RT * RT_ROWS, 0, st>>>(p, hop);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;                      // no walk over words that nobody has written
    // four environments per thread where the chip is full with that
    const unsigned ept = p.N >= 4u * 8u * BLOCK * p.sms ? 4u : 1u;
    cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((p.N + ept * BLOCK - 1u) / (ept * BLOCK)); cfg.blockDim = dim3(BLOCK); cfg.stream = st;
    cudaLaunchAttribute at;                              // the walk is set up, and draws its start cells, while the last tiles are folded
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization; at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, ept == 4u ? k_rollout_walk<4u, RT_SHIFT> : k_rollout_walk<1u, RT_SHIFT>, p, (const unsigned*)hop, max_steps, nonce, h);
}
cudaError_t launch_rollout(const Params& p, unsigned* hop, unsigned max_steps, unsigned long long nonce, Handover h, cudaStream_t st) {
    // A 64 x 64 tile takes 512 threads, four of them fill an SM.  Where they do not fill every SM (the chain of rounds in one block is then what
    // takes the time) tiles of a quarter of that size are folded by four times as many blocks; beyond, the larger tile saves hops.  A call from Python with 64 /
    // 32: 256^2 cells 24.0 / 20.4 us, 700^2 24.2 / 21.7, 1024^2 38.3 / 37.5, 1500^2 35.0 / 34.3, 2048^2 52.9 / 54.6.
    const unsigned big = (((unsigned)p.W + 63u) / 64u) * (((unsigned)p.H + 63u) / 64u);
    return big < 4u * p.sms ? launch_tiled<5u>(p, hop, max_steps, nonce, h, st) : launch_tiled<6u>(p, hop, max_steps, nonce, h, st);
}

}  // namespace cudarl
