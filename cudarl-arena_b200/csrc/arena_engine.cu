// arena_engine.cu -- the fused train step for the smallest worlds, many steps per launch: the whole world in the shared memory of one block, one environment per
// thread (k_arena_steps, up to 1,024), or a single one in one thread (k_one_steps).  Where shared memory holds no counters beside the rows, up to 32 environments run
// in one warp without any (k_solo_steps).
//
// A small world is latency, nothing else: in the gather engine (gather_engine.cu) a step is two barriers between blocks and several
// dependent accesses to L2.  Here the table, the counters and the move bytes lie in shared memory, the environments in registers, and
// the barrier is the block's (or, in one warp, none):
//
//   count   every environment reads the row of its cell, chooses, counts itself in the (cell, action) counter, moves on, takes its TD target from Q_t;
//   apply   the first on a (cell, action) applies its update as often as it was counted.
//
// The draws depend on nothing: up to 512 environments as many threads again make them some steps ahead.
//
// What bounds it: one thread's instructions, some 120 a step at 5 - 6 cycles each, with 1,024 environments the block's issue slots.  B200, us a step, as an instance of the
// gather engine's loop (draws in the same thread, options tested where they are off) / here: 18 environments on 20 x 19 cells 0.87 / 0.59, 120 on 50 x 62 1.00 / 0.66,
// 200 on 20 x 20 1.10 / 0.84, 500 on 60 x 60 1.71 / 1.22, 1,000 on 32 x 32 2.23 / 1.85; and, with 33 bytes a cell instead of 49, on grids that no block held: 300 on 80 x 80
// 3.8 / 0.93, 1,000 on 70 x 70 3.9 / 1.7.  (4,096 on 64 x 64 took 16 in one block; spread over the distributed shared memory of a cluster 4.4: remote rows are
// served one by one.  patch_engine.cu, where environments move between the blocks instead, takes 2.7.)
#include "step_loop.cuh"

namespace cudarl {

constexpr size_t SOLO_MOST = 216u * 1024u;       // 8.3 KB go to the draws
constexpr unsigned ARENA_ENVS = 1024u;
inline size_t solo_bytes(unsigned S) { return (size_t)S * 16u + (S + 15u) / 16u * 16u; }      // rows and move bytes

// One environment per thread, WALK threads; with HELP as many again make the draws ahead, CHUNK steps of them.
template <unsigned WALK, bool HELP> struct Arena {
    static constexpr unsigned CHUNK = HELP ? (WALK <= 64u ? 32u : 2048u / WALK) : 1u, DRAWS = HELP ? 2u * CHUNK * WALK : 0u;
    // rows (16 bytes a cell), two copies of four 16-bit counters by step parity, a bit per cell where no episode starts, move bytes, draws
    static constexpr size_t MOST = 224u * 1024u;
    static size_t bytes(unsigned S) { return (size_t)S * 32u + (S + 31u) / 32u * 4u + (S + 15u) / 16u * 16u + DRAWS * 4u; }
    // the walkers' barrier: one warp needs none
    static __device__ __forceinline__ void sync() {
        if constexpr (WALK == 32u) __syncwarp();
        else if constexpr (HELP) asm volatile("barrier.cta.sync 1, %0;" :: "n"(WALK) : "memory");
        else __syncthreads();
    }
};

// PLAIN: no traps, no clamp, no trace, epsilon by step.
template <unsigned WALK, bool HELP, bool PLAIN>
__global__ void __launch_bounds__(HELP ? 2u * WALK : WALK, 1) k_arena_steps(const __grid_constant__ Params p, const __grid_constant__ StepLaunch l) {
    using A = Arena<WALK, HELP>;
    constexpr unsigned CHUNK = A::CHUNK, ALL = HELP ? 2u * WALK : WALK;
    extern __shared__ __align__(16) unsigned char arena[];
    __shared__ unsigned s_flag, s_sum[5], s_ended, s_thr[2][CHUNK];
    if (!may_start(p, &s_flag)) return;
    const unsigned tid = threadIdx.x, S = p.S, W = (unsigned)p.W;
    float4* const rows = reinterpret_cast<float4*>(arena);
    uint2* const counts = reinterpret_cast<uint2*>(rows + S);                        // [2][S]
    unsigned* const draws = reinterpret_cast<unsigned*>(counts + 2u * S);            // [2][CHUNK][WALK]: the 24 bits compared with epsilon, above them the action to explore
    unsigned* const closed = draws + A::DRAWS;
    unsigned char* const moves = reinterpret_cast<unsigned char*>(closed + (S + 31u) / 32u);
    if (tid < 5u) s_sum[tid] = 0u;
    if (tid == 5u) s_ended = 0u;
    for (unsigned s = tid; s < S; s += ALL) { rows[s] = p.Q[s]; moves[s] = __ldg(p.gp.mv + s); counts[s] = make_uint2(0u, 0u); counts[S + s] = make_uint2(0u, 0u); }
    map_closed(p, closed, S, tid, ALL);
    const unsigned slot = HELP && tid >= WALK ? tid - WALK : tid;
    const bool walker = !HELP || tid < WALK, act = slot < p.N;
    const unsigned tmax = p.max_steps > 0 ? (unsigned)p.max_steps : 0x7FFFFFFFu;
    Tally tally{0u, 0u, 0u, 0u, 0u};
    const int4 r0 = act ? l.out[slot] : make_int4(0, 0, 0, 0);
    const unsigned id = (unsigned)r0.w;
    unsigned s = (unsigned)r0.y * W + (unsigned)r0.x, t = (unsigned)r0.z, before = NOBODY;        // before: the (cell, action) applied in the last step
    EpsilonIndex eps_index(p, l, PLAIN);
    float eps = __ldg(p.eps_tab + eps_index.at);
    auto threshold = [](float e) -> unsigned { return !(e > 0.0f) ? 0u : e >= 1.0f ? (1u << 24) : (unsigned)ceilf(e * 16777216.0f); };
    unsigned thr = threshold(eps);
    auto draw = [&](unsigned long long g) -> unsigned {
        const U4 r = philox4x32_10(p.env_offset + id, 0u, (unsigned)g, (unsigned)(g >> 32), p.policy_keys);
        return (r.x >> 8) | (r.y << 24);
    };
    auto make_draws = [&](unsigned first) {
        const unsigned c = (first / CHUNK) & 1u, m = min(CHUNK, l.steps - first);
#pragma unroll 1
        for (unsigned k = 0; k < m; ++k) draws[(c * CHUNK + k) * WALK + slot] = draw(p.step + first + k);
        if (l.eps_mode == 1 && slot < m) s_thr[c][slot] = threshold(__ldg(p.eps_tab + p.eps_idx + first + slot));
    };
    if (HELP && !walker) make_draws(0u);
    __syncthreads();
#pragma unroll 1
    for (unsigned first = 0; first < l.steps; first += HELP ? CHUNK : l.steps) {
        if (HELP && !walker) { if (first + CHUNK < l.steps) make_draws(first + CHUNK); }
        else {
            const unsigned c = HELP ? (first / CHUNK) & 1u : 0u, m = HELP ? min(CHUNK, l.steps - first) : l.steps;
#pragma unroll 1
            for (unsigned k = 0; k < m; ++k) {
                const unsigned long long g = p.step + first + k;
                const unsigned par = (first + k) & 1u;
                if (l.eps_mode == 1) thr = HELP ? s_thr[c][k] : threshold(__ldg(p.eps_tab + p.eps_idx + k));
                unsigned own = NOBODY; float target = 0.0f, value = 0.0f;
                if (before != NOBODY) reinterpret_cast<unsigned short*>(counts + (par ^ 1u) * S)[before] = 0u;      // (everybody has read it; nobody uses that parity now)
                before = NOBODY;
                if (act) {
                    const unsigned w = HELP ? draws[(c * CHUNK + k) * WALK + slot] : draw(g);
                    const float4 row = rows[s];
                    unsigned mv = moves[s];
                    const unsigned a = (w & 0xFFFFFFu) < thr ? (w >> 24) & 3u : (unsigned)argmax4(row);
                    mv >>= a;                             // bit 0: the move is blocked, bit 4: it ends on a goal
                    own = s * 4u + a;
                    const unsigned sh = (a & 1u) * 16u, old = atomicAdd(reinterpret_cast<unsigned*>(counts + par * S) + (own >> 1), 1u << sh);
                    const unsigned d = (a & 1u) ? 1u : W, cell = s;
                    const bool blocked = (mv & 1u) != 0u, done = (mv & 16u) != 0u;
                    s = blocked ? s : a - 1u < 2u ? s + d : s - d;
                    float m4 = max4(rows[s]);
                    value = pick(row, (int)a);
                    if (!PLAIN && p.legacy_clamp && m4 < 0.0f) m4 = 0.0f;
                    float r = -0.01f;
                    if (!PLAIN && p.ntraps && blocked) { const unsigned y = cell / W; r = blocked_step_reward(p, (int)(cell - y * W), (int)y, (int)a); }     // a trap charges its penalty
                    target = done ? 1.0f : __fmaf_rn(p.gamma, m4, r);
                    if (!PLAIN && l.trace && first + k + 1u == l.steps) { p.tr_a[id] = (int)a; p.tr_r[id] = done ? 1.0f : r; p.tr_d[id] = done ? 1 : 0; }
                    t = min(t + 1u, STEP_SAT);
                    if (done || t >= tmax) {
                        s = sample_start_if(p, p.env_offset + id, g + 1ull, TAG_START, [&](unsigned cc) { return closed[cc >> 5] >> (cc & 31u) & 1u; }); t = 0u;
                        if (done) ++tally.goals; else ++tally.timeouts;
                        if (!PLAIN && l.eps_mode == 2) atomicAdd(&s_ended, 1u);
                    }
                    if ((old >> sh) & 0xFFFFu) own = NOBODY;      // the first on a (cell, action) applies its update
                }
                A::sync();
                if (own != NOBODY) {
                    const uint2 q = counts[par * S + (own >> 2)];
                    const unsigned a = own & 3u, n = ((a & 2u) ? q.y : q.x) >> ((a & 1u) * 16u) & 0xFFFFu, both = q.x + q.y, tot = (both & 0xFFFFu) + (both >> 16);
                    if (tot > 1u) tally.conf += n;
                    if (tot > CROWDED_CELL) {                     // the lowest chosen action speaks for the cell
                        const unsigned c0 = q.x & 0xFFFFu, c1 = q.x >> 16;
                        if ((a == 0u ? 0u : a == 1u ? c0 : a == 2u ? c0 + c1 : c0 + c1 + (q.y & 0xFFFFu)) == 0u) { ++tally.crowded; tally.on_crowded += tot; }
                    }
                    reinterpret_cast<float*>(rows)[own] = apply_counted(value, target, p.lr, n);
                    before = own;
                }
                if (!PLAIN && l.eps_mode == 2) {                  // (nobody adds to the ended episodes before the second barrier)
                    if (first + k + 1u < l.steps) { eps_index.next(p, l, PLAIN, *reinterpret_cast<volatile unsigned*>(&s_ended), true); eps = __ldg(p.eps_tab + eps_index.at); thr = threshold(eps); }
                }
                A::sync();
            }
        }
        if (HELP) __syncthreads();
    }
    __syncthreads();
    for (unsigned k = tid; k < S; k += ALL) p.Q[k] = rows[k];
    if (walker && act) { const unsigned y = s / W; l.out[slot] = make_int4((int)(s - y * W), (int)y, (int)t, (int)id); }
    add_tallies(p, l, tally, s_sum, true, eps);
}

// 2 to 32 environments on grids of more than 6,676 cells, and on others in launches of few steps: one warp steps them, without counters or a barrier in the step -- who stands on the same (cell, action) is found
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

template <unsigned WALK, bool HELP>
static cudaError_t launch_one(const Params& p, const StepLaunch& l, cudaStream_t st) {
    using A = Arena<WALK, HELP>;
    auto* const fn = plain(p, l) ? k_arena_steps<WALK, HELP, true> : k_arena_steps<WALK, HELP, false>;
    const cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)A::MOST);
    if (e != cudaSuccess) return e;
    fn<<<1, HELP ? 2u * WALK : WALK, A::bytes(p.S), st>>>(p, l);
    return cudaGetLastError();
}
// One block holds up to 1,024 environments at one per thread; twice that takes longer than the other engines.  Up to 512 half the threads make draws.
bool arena_plan(Params& p) {
    GatherP& gp = p.gp;
    const unsigned n = p.N ? p.N : 1u;
    gp.threads = n <= 32u ? 32u : n <= 64u ? 64u : n <= 128u ? 128u : n <= 256u ? 256u : n <= 512u ? 512u : 1024u;
    gp.chunk = gp.threads; gp.grid = 1u; gp.arena = 1u;
    if (n <= 32u) return true;
    return n <= ARENA_ENVS && (n <= 512u ? Arena<512u, true>::bytes(p.S) : Arena<1024u, false>::bytes(p.S)) <= Arena<1024u, false>::MOST;
}
cudaError_t launch_arena_steps(const Params& p, const StepLaunch& l, cudaStream_t st) {
    const bool pl = plain(p, l);
    // Up to 32 environments walk over few cells in few steps: not worth fetching the world into shared memory.  Us a step, 1 / 2 / 4 / 8 / 16 steps a call, fetched / not: 32 environments on 40 x 40
    // 7.0 / 6.2, 4.1 / 3.65, 2.1 / 2.6 ..; 60 x 60 10.3 / 6.2, 5.1 / 3.6, 2.6 / 2.6, 1.6 / 1.9 ..; 80 x 83 13.6 / 6.2, 7.2 / 3.5, 3.65 / 2.6, 2.1 / 1.9, 1.3 / 1.65; 110 x 110 (in one warp) 14.6 / 6.2 .. 1.8 / 1.65.
    const bool few = p.N > 1u && p.N <= 32u && l.steps * 800ull <= p.S;
    if (p.N == 1u || few || (p.N <= 32u && Arena<32u, true>::bytes(p.S) > Arena<32u, true>::MOST)) {
        const bool fits = !few && solo_bytes(p.S) <= SOLO_MOST, options = p.ntraps || p.legacy_clamp || l.trace;
        auto* const fn = p.N == 1u ? fits ? options ? k_one_steps<true, true> : k_one_steps<true, false> : options ? k_one_steps<false, true> : k_one_steps<false, false>
                                   : fits ? pl ? k_solo_steps<true, true> : k_solo_steps<true, false> : pl ? k_solo_steps<false, true> : k_solo_steps<false, false>;
        if (fits) { const cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLO_MOST); if (e != cudaSuccess) return e; }
        fn<<<1, 64, fits ? solo_bytes(p.S) : 0u, st>>>(p, l);
        return cudaGetLastError();
    }
    switch (p.gp.threads) {
        case 32u: return launch_one<32u, true>(p, l, st);
        case 64u: return launch_one<64u, true>(p, l, st);
        case 128u: return launch_one<128u, true>(p, l, st);
        case 256u: return launch_one<256u, true>(p, l, st);
        case 512u: return launch_one<512u, true>(p, l, st);
        default: return launch_one<1024u, false>(p, l, st);
    }
}

}  // namespace cudarl
