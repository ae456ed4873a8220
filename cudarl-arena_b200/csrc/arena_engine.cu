// arena_engine.cu -- the fused train step for the smallest worlds: the whole world in the shared memory of one block (k_arena_steps), up to 32
// environments in one warp (k_solo_steps), one in a thread (k_one_steps), many steps per launch.
//
// A small world is latency, nothing else: in the gather engine (gather_engine.cu) a step is two barriers between blocks and several
// dependent accesses to L2.  Here the table, the counters and the move bytes lie in shared memory, the environments in registers, and
// the barrier is the block's.  The step of k_arena_steps is step_loop.cuh; the other two, further down, have neither counters nor barriers.
//
// What bounds k_arena_steps: one block's issue slots, about 300 instructions per warp and step.  B200, us per step, here / gather engine: 200
// on 20 x 20 cells 1.1 / 4.7, 1,000 on 32 x 32 2.2 / 4.7; 4,096 on 64 x 64 16 / 4.7.  The same spread over
// the distributed shared memory of a cluster was no faster than L2 (4,096 on 64 x 64: 4.4 with 16 blocks; scattered 16-byte accesses to
// other blocks' shared memory are served one by one), nor with a copy of the table in every block (3.9: every update is then stored 8 times).
#include "step_loop.cuh"

namespace cudarl {

constexpr size_t ARENA_MOST = 226u * 1024u;      // dynamic shared memory of a block (227 KB less the static words of step_loop.cuh)
constexpr size_t SOLO_MOST = 216u * 1024u;       // 8.3 KB go to the draws
constexpr unsigned ARENA_ENVS = 1024u;
// rows (16 bytes a cell), two rows of counters by step parity (16 bytes each), a move byte
inline size_t solo_bytes(unsigned S) { return (size_t)S * 16u + (S + 15u) / 16u * 16u; }      // without the counters
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

// 2 to 32 environments: one warp steps them, without counters or a barrier in the step -- who stands on the same (cell, action) is found
// with a match across the warp, and the lowest of them applies the update for all.  A second warp makes the random draws, which depend
// on nothing, a chunk of steps ahead.  SHARED: the world in shared memory; else in global memory, where the rows the warp walks over stay in
// its first-level cache.
// What bounds it: the chain of dependent instructions of one step (B200, when it also ran a single environment: with the counters
// and barriers of the block's step 0.58 us a step, with the match but the draws in the same warp 0.46; as it is 0.36).
constexpr unsigned SOLO_CHUNK = 32u;

template <bool SHARED, bool PLAIN>
__global__ void __launch_bounds__(64, 1) k_solo_steps(const __grid_constant__ Params p, const __grid_constant__ StepLaunch l) {
    extern __shared__ __align__(16) unsigned char arena[];
    __shared__ unsigned s_flag, s_sum[5];
    __shared__ unsigned s_draw[2][SOLO_CHUNK][32];   // per step and environment: the 24 bits compared with epsilon, above them the action to explore
    __shared__ unsigned s_thr[2][SOLO_CHUNK];        // explore iff those 24 bits are below
    if (!may_start(p, &s_flag)) return;
    const unsigned tid = threadIdx.x, lane = tid & 31u, S = p.S, W = (unsigned)p.W;
    const bool walker = tid < 32u;
    if (tid < 5u) s_sum[tid] = 0u;
    float4* const rows = SHARED ? reinterpret_cast<float4*>(arena) : p.Q;
    unsigned char* const moves = SHARED ? arena + (size_t)S * 16u : p.gp.mv;
    if (SHARED) {
#pragma unroll 8
        for (unsigned s = tid; s < S; s += 64u) { rows[s] = p.Q[s]; moves[s] = __ldg(p.gp.mv + s); }
    }
    const unsigned tmax = p.max_steps > 0 ? (unsigned)p.max_steps : 0x7FFFFFFFu;
    const bool act = lane < p.N;
    Tally tally{0u, 0u, 0u, 0u, 0u};
    unsigned s = 0u, t = 0u, id = 0u, ended = 0u;
    if (act) { const int4 r = l.out[lane]; s = (unsigned)r.y * W + (unsigned)r.x; t = (unsigned)r.z; id = (unsigned)r.w; }
    EpsilonIndex eps_index(p, l, PLAIN);
    float eps = __ldg(p.eps_tab + eps_index.at);
    auto threshold = [](float e) -> unsigned { return !(e > 0.0f) ? 0u : e >= 1.0f ? (1u << 24) : (unsigned)ceilf(e * 16777216.0f); };
    unsigned thr = threshold(eps);
    auto make_draws = [&](unsigned first) {
        const unsigned b = (first / SOLO_CHUNK) & 1u, m = min(SOLO_CHUNK, l.steps - first);
        for (unsigned k = 0; k < m; ++k) {
            const unsigned long long g = p.step + first + k;
            const U4 r = philox4x32_10(p.env_offset + id, 0u, (unsigned)g, (unsigned)(g >> 32), p.policy_keys);
            s_draw[b][k][lane] = (r.x >> 8) | (r.y << 24);
        }
        if (lane < m) s_thr[b][lane] = threshold(__ldg(p.eps_tab + (l.eps_mode == 1 ? p.eps_idx + first + lane : p.eps_idx)));
    };
    if (!walker) make_draws(0u);
    __syncthreads();

    for (unsigned first = 0; first < l.steps; first += SOLO_CHUNK) {
        if (!walker) { if (first + SOLO_CHUNK < l.steps) make_draws(first + SOLO_CHUNK); }
        else {
            const unsigned b = (first / SOLO_CHUNK) & 1u, m = min(SOLO_CHUNK, l.steps - first);
            for (unsigned k = 0; k < m; ++k) {
                const float4 row = rows[s];
                unsigned mv = moves[s];
                const unsigned w = s_draw[b][k][lane];
                if (PLAIN || l.eps_mode != 2) thr = s_thr[b][k];
                const int a = (w & 0xFFFFFFu) < thr ? (int)(w >> 24) & 3 : argmax4(row);
                mv >>= a;                             // bit 0: the move is blocked, bit 4: it ends on a goal
                const unsigned cell = s, own = s * 4u + (unsigned)a, there = a == 0 ? s - W : a == 1 ? s + 1u : a == 2 ? s + W : s - 1u;
                const bool blocked = (mv & 1u) != 0u, done = (mv & 16u) != 0u;
                s = blocked ? s : there;
                float m4 = max4(rows[s]);
                const unsigned mates = __match_any_sync(FULL, act ? own : NOBODY), here = __match_any_sync(FULL, act ? cell : NOBODY);
                const unsigned n = (unsigned)__popc(mates), tot = act ? (unsigned)__popc(here) : 0u;
                const bool applies = act && lane == (unsigned)__ffs((int)mates) - 1u;
                if (tot > 1u) ++tally.conf;
                if (tot > CROWDED_CELL) { ++tally.on_crowded; if (lane == (unsigned)__ffs((int)here) - 1u) ++tally.crowded; }
                if (!PLAIN && p.legacy_clamp && m4 < 0.0f) m4 = 0.0f;
                float r = -0.01f;
                if (!PLAIN && p.ntraps && blocked) { const unsigned y = cell / W; r = blocked_step_reward(p, (int)(cell - y * W), (int)y, a); }     // a trap charges its penalty
                const float target = done ? 1.0f : __fmaf_rn(p.gamma, m4, r);
                __syncwarp();                         // every lane has taken its target from Q_t
                if (applies) reinterpret_cast<float*>(rows)[own] = apply_counted(pick(row, a), target, p.lr, n);
                if (!PLAIN && act && l.trace && first + k + 1u == l.steps) { p.tr_a[id] = a; p.tr_r[id] = done ? 1.0f : r; p.tr_d[id] = done ? 1 : 0; }
                t = min(t + 1u, STEP_SAT);
                const bool over = act && (done || t >= tmax);
                if (__any_sync(FULL, over)) {
                    if (over) {
                        s = sample_start(p, p.env_offset + id, p.step + first + k + 1ull, TAG_START); t = 0u;
                        if (done) ++tally.goals; else ++tally.timeouts;
                    }
                    if (!PLAIN && l.eps_mode == 2) {
                        ended += (unsigned)__popc(__ballot_sync(FULL, over));
                        if (first + k + 1u < l.steps) { eps_index.next(p, l, PLAIN, ended, true); eps = __ldg(p.eps_tab + eps_index.at); thr = threshold(eps); }
                    }
                }
                __syncwarp();                         // the entries are stored
            }
        }
        __syncthreads();
    }
    if (SHARED) for (unsigned k = tid; k < S; k += 64u) p.Q[k] = rows[k];
    if (walker && act) { const unsigned y = s / W; l.out[lane] = make_int4((int)(s - y * W), (int)y, (int)t, (int)id); }
    add_tallies(p, l, tally, s_sum, true, eps);
}

// One environment: one thread walks, a warp makes its draws ahead, a step per lane.  Nobody else changes the table, so the row an environment moves to is
// both its target's and the one it chooses from next: it is read once, and a step's chain is choice -> cell -> row.
// What bounds it: one thread's instructions, some 60 a step at about 6 cycles each.  B200, 10 x 10 cells, epsilon by episodes: 0.19 us a step, as one lane of
// k_solo_steps 0.36; 500 steps with table, state and statistics read back 229 -> 145 us (options as run-time tests, the maximum in three levels 168).
constexpr unsigned ONE_CHUNK = 128u;

template <bool SHARED, bool OPTIONS>       // OPTIONS: traps, the clamp, a trace
__global__ void __launch_bounds__(64, 1) k_one_steps(const __grid_constant__ Params p, const __grid_constant__ StepLaunch l) {
    extern __shared__ __align__(16) unsigned char arena[];
    __shared__ unsigned s_flag, s_sum[5];
    __shared__ unsigned s_draw[2][ONE_CHUNK + 1u], s_thr[2][ONE_CHUNK + 1u];       // by step; one more than are made is read ahead
    if (!may_start(p, &s_flag)) return;
    const unsigned tid = threadIdx.x, S = p.S, W = (unsigned)p.W;
    if (tid < 5u) s_sum[tid] = 0u;
    float4* const rows = SHARED ? reinterpret_cast<float4*>(arena) : p.Q;
    unsigned char* const moves = SHARED ? arena + (size_t)S * 16u : p.gp.mv;
    if (SHARED) {
#pragma unroll 8
        for (unsigned s = tid; s < S; s += 64u) { rows[s] = p.Q[s]; moves[s] = __ldg(p.gp.mv + s); }
    }
    const unsigned tmax = p.max_steps > 0 ? (unsigned)p.max_steps : 0x7FFFFFFFu;
    Tally tally{0u, 0u, 0u, 0u, 0u};
    const int4 r0 = l.out[0];
    const unsigned id = (unsigned)r0.w;
    unsigned s = (unsigned)r0.y * W + (unsigned)r0.x, t = (unsigned)r0.z;
    EpsilonIndex eps_index(p, l, false);
    float eps = __ldg(p.eps_tab + eps_index.at);
    auto threshold = [](float e) -> unsigned { return !(e > 0.0f) ? 0u : e >= 1.0f ? (1u << 24) : (unsigned)ceilf(e * 16777216.0f); };
    unsigned thr = threshold(eps);
    auto make_draws = [&](unsigned first) {
        const unsigned c = (first / ONE_CHUNK) & 1u, m = min(ONE_CHUNK, l.steps - first);
        for (unsigned k = tid & 31u; k < m; k += 32u) {
            const unsigned long long g = p.step + first + k;
            const U4 r = philox4x32_10(p.env_offset + id, 0u, (unsigned)g, (unsigned)(g >> 32), p.policy_keys);
            s_draw[c][k] = (r.x >> 8) | (r.y << 24);
            if (l.eps_mode == 1) s_thr[c][k] = threshold(__ldg(p.eps_tab + p.eps_idx + first + k));
        }
    };
    if (tid >= 32u) make_draws(0u);
    __syncthreads();
    float4 row = rows[s];
    unsigned mv = moves[s];
    for (unsigned first = 0; first < l.steps; first += ONE_CHUNK) {
        if (tid >= 32u) { if (first + ONE_CHUNK < l.steps) make_draws(first + ONE_CHUNK); }
        else if (tid == 0u) {
            const unsigned c = (first / ONE_CHUNK) & 1u, m = min(ONE_CHUNK, l.steps - first);
            unsigned next_w = s_draw[c][0], next_thr = l.eps_mode == 1 ? s_thr[c][0] : thr;
#pragma unroll 1
            for (unsigned k = 0; k < m; ++k) {
                const unsigned w = next_w;
                if (l.eps_mode == 1) { thr = next_thr; next_thr = s_thr[c][k + 1u]; }
                next_w = s_draw[c][k + 1u];
                const unsigned a = (w & 0xFFFFFFu) < thr ? (w >> 24) & 3u : (unsigned)argmax4_pairs(row);
                const unsigned bits = mv >> a;                // bit 0: the move is blocked, bit 4: it ends on a goal
                const bool blocked = (bits & 1u) != 0u, done = (bits & 16u) != 0u;
                const unsigned d = (a & 1u) ? 1u : W, to = blocked ? s : a - 1u < 2u ? s + d : s - d;
                float4 next = rows[to];
                mv = moves[to];
                const float q = pick(row, (int)a);
                float m4 = max4(next);
                if (OPTIONS && p.legacy_clamp && m4 < 0.0f) m4 = 0.0f;
                float r = -0.01f;
                if (OPTIONS && p.ntraps && blocked) { const unsigned y = s / W; r = blocked_step_reward(p, (int)(s - y * W), (int)y, (int)a); }     // a trap charges its penalty
                const float target = done ? 1.0f : __fmaf_rn(p.gamma, m4, r);
                const float v = __fmaf_rn(p.lr, __fsub_rn(target, q), q);
                reinterpret_cast<float*>(rows)[s * 4u + a] = v;
                if (blocked) { next.x = a == 0u ? v : next.x; next.y = a == 1u ? v : next.y; next.z = a == 2u ? v : next.z; next.w = a == 3u ? v : next.w; }
                row = next; s = to;
                if (OPTIONS && l.trace && first + k + 1u == l.steps) { p.tr_a[id] = (int)a; p.tr_r[id] = done ? 1.0f : r; p.tr_d[id] = done ? 1 : 0; }
                t = min(t + 1u, STEP_SAT);
                if (done || t >= tmax) {
                    s = sample_start(p, p.env_offset + id, p.step + first + k + 1ull, TAG_START); t = 0u;
                    row = rows[s]; mv = moves[s];
                    if (done) ++tally.goals; else ++tally.timeouts;
                    if (l.eps_mode == 2 && first + k + 1u < l.steps) { eps_index.next(p, l, false, tally.goals + tally.timeouts, true); eps = __ldg(p.eps_tab + eps_index.at); thr = threshold(eps); }
                }
            }
        }
        __syncthreads();
    }
    if (SHARED) for (unsigned k = tid; k < S; k += 64u) p.Q[k] = rows[k];
    if (tid == 0u) { const unsigned y = s / W; l.out[0] = make_int4((int)(s - y * W), (int)y, (int)t, (int)id); }
    add_tallies(p, l, tally, s_sum, true, eps);
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
    if (n <= 32u) {
        gp.threads = gp.chunk = 32u; gp.grid = 1u; gp.arena = 1u;
        return cudaFuncSetAttribute((const void*)k_one_steps<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLO_MOST) == cudaSuccess &&
               cudaFuncSetAttribute((const void*)k_one_steps<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLO_MOST) == cudaSuccess &&
               cudaFuncSetAttribute((const void*)k_solo_steps<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLO_MOST) == cudaSuccess &&
               cudaFuncSetAttribute((const void*)k_solo_steps<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLO_MOST) == cudaSuccess;
    }
    if (n > ARENA_ENVS || arena_bytes(p.S) > ARENA_MOST) return false;
    gp.threads = n <= 256u ? 256u : 1024u;
    gp.chunk = gp.threads; gp.grid = 1u; gp.arena = 1u;
    return allow<256u>() && allow<1024u>();
}

template <unsigned AB>
static cudaError_t launch_one(const Params& p, const StepLaunch& l, cudaStream_t st) {
    if (plain(p, l)) k_arena_steps<AB, true><<<1, AB, arena_bytes(p.S), st>>>(p, l);
    else             k_arena_steps<AB, false><<<1, AB, arena_bytes(p.S), st>>>(p, l);
    return cudaGetLastError();
}
cudaError_t launch_arena_steps(const Params& p, const StepLaunch& l, cudaStream_t st) {
    if (p.gp.threads == 32u) {
        const bool fits = solo_bytes(p.S) <= SOLO_MOST, pl = plain(p, l);
        if (p.N == 1u) {
            const size_t bytes = fits ? solo_bytes(p.S) : 0u;
            const bool options = p.ntraps || p.legacy_clamp || l.trace;
            (fits ? options ? k_one_steps<true, true> : k_one_steps<true, false> : options ? k_one_steps<false, true> : k_one_steps<false, false>)<<<1, 64, bytes, st>>>(p, l);
            return cudaGetLastError();
        }
        if (fits) { if (pl) k_solo_steps<true, true><<<1, 64, solo_bytes(p.S), st>>>(p, l); else k_solo_steps<true, false><<<1, 64, solo_bytes(p.S), st>>>(p, l); }
        else { if (pl) k_solo_steps<false, true><<<1, 64, 0, st>>>(p, l); else k_solo_steps<false, false><<<1, 64, 0, st>>>(p, l); }
        return cudaGetLastError();
    }
    return p.gp.threads == 256u ? launch_one<256u>(p, l, st) : launch_one<1024u>(p, l, st);
}

}  // namespace cudarl
