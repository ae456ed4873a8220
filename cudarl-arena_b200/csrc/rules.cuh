// rules.cuh -- device-side rules shared by every kernel of the library: the counter-based random
// streams, the epsilon-greedy choice, the TD arithmetic and the seeded start cells.  One definition,
// so the kernels cannot drift apart.
//
// Reference semantics (paths relative to the CudaRL-Arena project root):
//   TD update   src/kernels.cu:96-114 (true max as in src/gpu/kernels.cu:36-45, src/train.py:134)
//   eps-greedy  src/train.py:101-108, first-max argmax src/q_learning.cu:196-206
//   reset       src/environment.cu:6-14
#pragma once
#include "kernels.cuh"

namespace cudarl {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr unsigned CROWDED_CELL = 24;       // a cell with more environments than this counts as "crowded" in the run statistics

// ------------------------------------------------------------------------------------------------
// Philox4x32-10, counter-based: no generator state is stored anywhere.
struct U4 { unsigned x, y, z, w; };

__device__ __forceinline__ U4 philox4x32_10(unsigned c0, unsigned c1, unsigned c2, unsigned c3,
                                            unsigned k0, unsigned k1) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const unsigned long long m0 = (unsigned long long)0xD2511F53u * c0, m1 = (unsigned long long)0xCD9E8D57u * c2;     // one wide multiply each
        const unsigned hi0 = (unsigned)(m0 >> 32), lo0 = (unsigned)m0, hi1 = (unsigned)(m1 >> 32), lo1 = (unsigned)m1;
        unsigned n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    return U4{c0, c1, c2, c3};
}

// The same with the round keys given (pairs).
__device__ __forceinline__ U4 philox4x32_10(unsigned c0, unsigned c1, unsigned c2, unsigned c3, const unsigned (&rk)[20]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const unsigned long long m0 = (unsigned long long)0xD2511F53u * c0, m1 = (unsigned long long)0xCD9E8D57u * c2;
        const unsigned n0 = (unsigned)(m1 >> 32) ^ c1 ^ rk[2 * r], n2 = (unsigned)(m0 >> 32) ^ c3 ^ rk[2 * r + 1];
        c0 = n0; c1 = (unsigned)m1; c2 = n2; c3 = (unsigned)m0;
    }
    return U4{c0, c1, c2, c3};
}

// Word pair {x, y} of the policy stream of one step: philox4x32_10(c0, 0, step, policy keys).  What the first two rounds make of the step
// and the keys alone is the same for every environment and comes from the host (policy_prefix): two of the twenty wide multiplies fewer.
__host__ __device__ __forceinline__ void policy_prefix(const unsigned (&rk)[20], unsigned long long step, unsigned (&pre)[4]) {
    const unsigned long long m1 = (unsigned long long)0xCD9E8D57u * (unsigned)step;
    const unsigned c0 = (unsigned)(m1 >> 32) ^ rk[0], c1 = (unsigned)m1;                  // first round, c1 = 0
    const unsigned long long m0 = (unsigned long long)0xD2511F53u * c0;
    pre[0] = (unsigned)(step >> 32) ^ rk[1]; pre[1] = c1 ^ rk[2]; pre[2] = (unsigned)(m0 >> 32) ^ rk[3]; pre[3] = (unsigned)m0 ^ rk[5];
}
__device__ __forceinline__ U4 policy_philox(unsigned env, const unsigned (&rk)[20], const unsigned (&pre)[4]) {
    unsigned long long m0 = (unsigned long long)0xD2511F53u * env;
    unsigned long long m1 = (unsigned long long)0xCD9E8D57u * ((unsigned)(m0 >> 32) ^ pre[0]);
    unsigned c0 = (unsigned)(m1 >> 32) ^ pre[1], c1 = (unsigned)m1, c2 = (unsigned)m0 ^ pre[2], c3 = 0u;
#pragma unroll
    for (int r = 2; r < 10; ++r) {
        m0 = (unsigned long long)0xD2511F53u * c0; m1 = (unsigned long long)0xCD9E8D57u * c2;
        const unsigned n0 = (unsigned)(m1 >> 32) ^ c1 ^ rk[2 * r], n2 = r == 2 ? (unsigned)(m0 >> 32) ^ pre[3] : (unsigned)(m0 >> 32) ^ c3 ^ rk[2 * r + 1];
        c0 = n0; c1 = (unsigned)m1; c2 = n2; c3 = (unsigned)m0;
    }
    return U4{c0, c1, c2, c3};
}

constexpr unsigned TAG_START = 0x53545254u, TAG_QINIT = 0x51494E49u, TAG_POLICY = 0x504F4C49u,
                   TAG_EVAL = 0x4556414Cu;

__device__ __forceinline__ float u01(unsigned w) { return (float)(w >> 8) * 5.9604644775390625e-08f; }

__device__ __forceinline__ unsigned cw_load(const unsigned short* cw, unsigned cell) { return cw[cell]; }

// The move bytes of the cells of a column (written tile by tile by k_te_cls, row by row by k_gather_moves, for the engine in use): bit a
// = a move in direction a is blocked, bit 4+a = the cell an environment stands on after choosing a is a goal.
struct MoveColumn {
    const unsigned char* at_x; unsigned tall, mask, shift;           // a row of tiles (or of cells) is `tall` bytes
    __device__ __forceinline__ MoveColumn(const Params& p, unsigned x) {
        const TileP& tp = p.tp;
        if (p.gp.mv) { at_x = p.gp.mv + x; tall = (unsigned)p.W; mask = 0u; shift = 0u; }
        else { mask = tp.T - 1u; shift = tp.tshift; tall = tp.tiles_x * tp.cls_stride; at_x = tp.tcls + (x >> shift) * tp.cls_stride + (x & mask); }
    }
    __device__ __forceinline__ unsigned at(unsigned y) const { return __ldg(at_x + ((y >> shift) * tall + ((y & mask) << shift))); }
};

__device__ __forceinline__ void box_put(const Handover& h, unsigned k, unsigned v) {
    *reinterpret_cast<volatile unsigned long long*>(&h.box->w[k]) = ((unsigned long long)h.ticket << 32) | v;
}
__device__ __forceinline__ void box_put64(const Handover& h, unsigned k, unsigned long long v) { box_put(h, k, (unsigned)v); box_put(h, k + 1u, (unsigned)(v >> 32)); }
__device__ __forceinline__ void box_put_error(const World& p, const Handover& h) { box_put(h, 0u, *reinterpret_cast<volatile unsigned*>(&p.ctl->error)); }
// To be called by all threads of every block, after their writes: true in one thread of the last block to get here, which sees what
// the other blocks have written -- and, when HOST, after which the host sees it too (arrays in the stage).
template <bool HOST>
__device__ __forceinline__ bool last_to_finish(const World& p) {
    __syncthreads();
    if (threadIdx.x != 0u) return false;
    if (HOST) __threadfence_system(); else __threadfence();
    if (gridDim.x == 1u) return true;
    if (atomicAdd(&p.ctl->done_blocks, 1u) + 1u != gridDim.x) return false;
    if (HOST) __threadfence_system(); else __threadfence();
    p.ctl->done_blocks = 0u;
    return true;
}

// Start cell of an episode.  CENTRE/FIXED: the configured cell (reference: src/environment.cu:9-10).
// RANDOM: first free non-goal cell among 64 seeded candidates, else the precomputed fallback cell.
template <class Closed>
__device__ __forceinline__ unsigned sample_start_if(const World& p, unsigned gi, unsigned long long nonce, unsigned tag, Closed closed) {
    if (p.start_mode != 2) return p.start_cell;
#pragma unroll 1            // restarts are rare: keep the inlined copies of this loop small (the step kernel's hot loop must fit the instruction cache)
    for (unsigned k = 0; k < 16; ++k) {
        U4 w = philox4x32_10(gi, k, (unsigned)nonce, (unsigned)(nonce >> 32), p.k0, p.k1 ^ tag);
        unsigned c;
        c = __umulhi(w.x, p.S); if (!closed(c)) return c;
        c = __umulhi(w.y, p.S); if (!closed(c)) return c;
        c = __umulhi(w.z, p.S); if (!closed(c)) return c;
        c = __umulhi(w.w, p.S); if (!closed(c)) return c;
    }
    return p.fallback_start;
}
__device__ __forceinline__ unsigned sample_start(const World& p, unsigned gi, unsigned long long nonce, unsigned tag) {
    return sample_start_if(p, gi, nonce, tag, [&](unsigned c) { return cw_load(p.cw, c) & (CW_OBST | CW_GOAL); });
}

// Reward of a step that does not end on a goal, for an agent at (x, y) whose action `a` was blocked: the step cost, or -- when
// the cell it walked into is a trap -- that trap's penalty (src/kernels.cu:47,61-63 of the reference: a trap is an obstacle, the
// agent stays where it is and is charged the cell's value).  Binary search in the sparse trap table.
__device__ __forceinline__ float blocked_step_reward(const World& p, int x, int y, int a) {
    if (!p.ntraps) return -0.01f;
    const int nx = x + (a == 1) - (a == 3), ny = y + (a == 2) - (a == 0);
    if (nx < 0 || nx >= p.W || ny < 0 || ny >= p.H) return -0.01f;
    const unsigned tgt = (unsigned)ny * (unsigned)p.W + (unsigned)nx;
    unsigned lo = 0, hi = p.ntraps;
    while (lo < hi) {
        const unsigned mid = (lo + hi) >> 1;
        const uint2 e = p.traps[mid];
        if (e.x == tgt) return __uint_as_float(e.y);
        if (e.x < tgt) lo = mid + 1u; else hi = mid;
    }
    return -0.01f;
}

__device__ __forceinline__ int argmax4(float4 r) {   // first maximum wins
    int b = 0; float bv = r.x;
    if (r.y > bv) { bv = r.y; b = 1; }
    if (r.z > bv) { bv = r.z; b = 2; }
    if (r.w > bv) { bv = r.w; b = 3; }
    return b;
}
// The same in two levels instead of three, for where it is part of a chain: the first of a pair unless the second is larger -- or, in the second pair, the first
// is no number (argmax4 passes over those, except in r.x).
__device__ __forceinline__ int argmax4_pairs(float4 r) {
    const bool y = r.y > r.x;
    const float lo = y ? r.y : r.x, hi = fmaxf(r.z, r.w);
    return hi > lo ? (r.z == hi ? 2 : 3) : (int)y;
}
__device__ __forceinline__ float max4(float4 r) {
    float m = r.x;
    m = r.y > m ? r.y : m; m = r.z > m ? r.z : m; m = r.w > m ? r.w : m;
    return m;
}
__device__ __forceinline__ float pick(float4 r, int a) { return a == 0 ? r.x : a == 1 ? r.y : a == 2 ? r.z : r.w; }
// One update of Q[s,a] toward `target`: q <- fma(lr, target - q, q), which is what nvcc makes of the reference's
// `q += lr * (target - q)` (src/kernels.cu:113-114).  Updates of the same (s,a) within a step are applied one
// after the other in ascending environment id, each seeing the value the previous one left (the targets come
// from Q_t), so any number of environments on one cell keeps the step a contraction.
__device__ __forceinline__ void fold(float4& r, int a, float lr, float target) {
    const float q = pick(r, a);
    const float v = __fmaf_rn(lr, __fsub_rn(target, q), q);
    r.x = a == 0 ? v : r.x; r.y = a == 1 ? v : r.y; r.z = a == 2 ? v : r.z; r.w = a == 3 ? v : r.w;
}

// Exclusive prefix of v over the block (any block size up to 1024); *total receives the block sum.
__device__ __forceinline__ unsigned block_scan_excl(unsigned v, unsigned* s_warp, unsigned* total) {
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned inc = v;
    for (int o = 1; o < 32; o <<= 1) { const unsigned t = __shfl_up_sync(FULL, inc, o); if (lane >= (unsigned)o) inc += t; }
    if (lane == 31u) s_warp[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const unsigned w = lane < nw ? s_warp[lane] : 0u; unsigned winc = w;
        for (int o = 1; o < 32; o <<= 1) { const unsigned t = __shfl_up_sync(FULL, winc, o); if (lane >= (unsigned)o) winc += t; }
        if (lane < nw) s_warp[lane] = winc - w;
        if (lane == 31u) s_warp[32] = winc;
    }
    __syncthreads();
    const unsigned r = s_warp[wid] + inc - v;
    *total = s_warp[32];
    __syncthreads();
    return r;
}

}  // namespace cudarl
