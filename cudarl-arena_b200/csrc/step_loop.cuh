// step_loop.cuh -- the fused train step with one thread per environment, many steps per launch, as the gather engine takes it (gather_engine.cu; patch_engine.cu where
// a patch overflows): table and counters in L2, a barrier of the grid or of one cluster.  And what all engines of many steps per launch share: the counted
// updates, the epsilon by episodes, the sums.
//
//   count   every environment reads the row of its cell, chooses its action, counts itself in the (cell, action) counter with an
//           atomic, moves on, and takes the TD target of its (cell, action) from Q_t;
//   -- barrier --
//   apply   the update of a (cell, action) is applied as many times as were counted, and the one table entry is stored;
//   -- barrier --
//
// All updates of one (cell, action) within a step are the same map, so only their number matters (see tile_engine.cu).  Who applies
// it: with OWNERS the first to count there, which needs the counter's old value -- right where latency counts and crowds are common;
// without, everybody who counted (all compute and store the same bits; of a crowd in a streamed population the first), so that the atomics need no answer -- right where their rate
// counts (1024 x 1024 cells, 1,048,576 environments: 25.0 -> 24.0 us a step; 1001 x 613, 150,001: 7.6 -> 6.8; but 64 x 64 with 4,096
// crowded ones 4.7 -> 5.5).  Counters alternate by step parity; who counted clears its counter in the next step's count phase, when
// everybody has read it and nobody uses that parity.
//
// A Space gives: row(s), moves(s), add(par, idx, n) -> old count, count(par, idx, n), note(par, idx) -> marked before, clear(par, idx),
// counts(par, s) -> uint4, store(idx, v), arrive(), wait() -> false when the launch has to be given up.
#pragma once
#include "kernels.cuh"
#include "rules.cuh"

namespace cudarl {

constexpr unsigned NOBODY = 0xFFFFFFFFu;
constexpr unsigned NOTED = 0x80000000u;     // a counter's mark: the crowded cell is in the statistics already

// What one environment needs between the two phases of a step, and what the launch sums up.
struct Tally { unsigned goals, timeouts, conf, crowded, on_crowded; };

// The update of (cell, action) `own` from the counted number of environments on it: the map q <- fma(lr, d - q, q) as often as counted.
// It is a contraction, so a long run ends at its fixed point: once the value stops changing it never changes again.
// Two at a time: a value that stands still shows at once, and half as many looks for one that does not.
__device__ __forceinline__ float apply_counted(float v, float d, float lr, unsigned n) {
    auto once = [&](float u) -> float { return __fmaf_rn(lr, __fsub_rn(d, u), u); };
    for (;;) {
        const float w = once(v);
        if (n == 1u || __float_as_uint(w) == __float_as_uint(v)) return w;
        const float x = once(w);
        if (n == 2u || __float_as_uint(x) == __float_as_uint(w)) return x;
        v = x; n -= 2u;
    }
}

// Whether a launch may start.  A context in which a wait has run out does nothing any more (its barrier counter is off); with a poll
// bound set (tests only) a wait that nothing can end runs out here.
__device__ __forceinline__ bool may_start(const Params& p, unsigned* s_flag) {
    if (threadIdx.x == 0u) {
        unsigned ok = (*reinterpret_cast<volatile unsigned*>(&p.ctl->error) & ERR_COPY_TIMEOUT) ? 0u : 1u;
        unsigned left = p.tp.wait_polls;
        while (left && *reinterpret_cast<volatile unsigned*>(&p.ctl->never) == 0u) --left;
        if (p.tp.wait_polls && left == 0u) { atomicOr(&p.ctl->error, ERR_COPY_TIMEOUT); ok = 0u; }
        *s_flag = ok;
    }
    __syncthreads();
    return *s_flag != 0u;
}

// A bit per cell into shared memory: no episode starts there.  32 cells at a time (the cell words are padded to 256 bytes): one after the other, a launch waited for one access to
// L2 per 32 cells and warp, 100 us for 168,000 cells.
__device__ __forceinline__ void map_closed(const World& p, unsigned* closed, unsigned cells, unsigned tid, unsigned threads) {
    for (unsigned k = tid; k < (cells + 31u) / 32u; k += threads) {
        const uint4* const q = reinterpret_cast<const uint4*>(p.cw) + 4u * k;
        unsigned w = 0u;
#pragma unroll
        for (unsigned j = 0; j < 4u; ++j) {
            const uint4 v = __ldg(q + j);
            const unsigned two[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (unsigned i = 0; i < 4u; ++i) {
                if (two[i] & (CW_OBST | CW_GOAL)) w |= 1u << (8u * j + 2u * i);
                if ((two[i] >> 16) & (CW_OBST | CW_GOAL)) w |= 2u << (8u * j + 2u * i);
            }
        }
        closed[k] = w;
    }
}

// The index of a step's epsilon in the table: fixed, by step, or by finished episodes -- it grows whenever their number passes the next
// multiple of the number of environments.
struct EpsilonIndex {
    unsigned at; unsigned long long ep0, ep_next;
    __device__ __forceinline__ EpsilonIndex(const Params& p, const StepLaunch& l, bool plain) : at(p.eps_idx), ep0(0ull), ep_next(~0ull) {
        if (plain || l.eps_mode != 2) return;
        ep0 = *reinterpret_cast<volatile unsigned long long*>(&p.ctl->episodes);
        const unsigned long long k = ep0 / p.N;
        at = (unsigned)min(k - l.eps_base_k, (unsigned long long)(l.eps_len - 1u));
        ep_next = (k + 1ull) * p.N;
    }
    // alone: `local` is the number of episodes finished in this launch, else the control block has all
    __device__ __forceinline__ void next(const Params& p, const StepLaunch& l, bool plain, unsigned local, bool alone) {
        if (l.eps_mode == 1) ++at;
        else if (!plain && l.eps_mode == 2) {
            const unsigned long long ep = alone ? ep0 + local : *reinterpret_cast<volatile unsigned long long*>(&p.ctl->episodes);
            while (ep >= ep_next) { ep_next += p.N; at = min(at + 1u, l.eps_len - 1u); }
        }
    }
};
// The sums of a launch: warp, block (s_sum: five zeroed words), control block.
__device__ __forceinline__ void add_tallies(const Params& p, const StepLaunch& l, const Tally& tally, unsigned* s_sum, bool episodes, float eps) {
    Ctl* const ctl = p.ctl;
    const unsigned tid = threadIdx.x;
    unsigned sums[5] = {tally.goals, tally.timeouts, tally.conf, tally.crowded, tally.on_crowded};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const unsigned v = __reduce_add_sync(FULL, sums[k]);
        if ((tid & 31u) == 0u && v) atomicAdd(&s_sum[k], v);
    }
    __syncthreads();
    if (tid == 0u) {
        if (s_sum[0]) atomicAdd(&ctl->goals, (unsigned long long)s_sum[0]);
        if (s_sum[1]) atomicAdd(&ctl->timeouts, (unsigned long long)s_sum[1]);
        if (episodes && s_sum[0] + s_sum[1]) atomicAdd(&ctl->episodes, (unsigned long long)(s_sum[0] + s_sum[1]));
        if (s_sum[2]) atomicAdd(&ctl->conflicts, (unsigned long long)s_sum[2]);
        if (s_sum[3]) atomicAdd(&ctl->long_chains, (unsigned long long)s_sum[3]);
        if (s_sum[4]) atomicAdd(&ctl->general, (unsigned long long)s_sum[4]);
        if (blockIdx.x == 0u && l.eps_mode == 2) ctl->eps_used = eps;
    }
}

// Where the state of the environments of a block lives during a launch.
enum class Home { Registers, Shared, Global };
// One environment of a block: cell, steps of the episode, number; the (cell, action) owned in this step, its TD target and value.
constexpr unsigned STATE_BYTES = 24u;

// The steps of one launch from step `skip` on, GB threads per block.  A block owns `count` slots of the records in `work` from `first` on: one per thread,
// in registers, or streamed turn by turn from shared (`arrays`: chunk x STATE_BYTES) or global memory (gp.state: N x STATE_BYTES).
// PLAIN: no traps, no clamp, no trace, epsilon by step -- the options are left out of the code, not skipped in it.
template <Home HOME, unsigned GB, bool PLAIN, bool OWNERS, class Space>
__device__ __forceinline__ void run_steps(const Params& p, const StepLaunch& l, Space& space, int4* __restrict__ work, unsigned char* arrays, unsigned skip = 0u) {
    __shared__ unsigned s_sum[5], s_ep;
    constexpr bool STREAM = HOME != Home::Registers;
    // Without OWNERS, who applies what a crowd has counted: with one turn a step everybody (all at the same time, and the answer to the question who came
    // first would take 0.6 us of the step's 7); with many turns the first to mark the counter, since the others' rounds would follow one another.
    // 1024 x 1024 cells, everybody on one start cell, everybody / the first, us a step: 1,048,576 environments at lr 0.1 160 / 108, at 0.001 1,963 /
    // 273, at 1e-5 107,000 / 10,170; 4,194,304 on 512 x 512, random starts 196 / 142.
    constexpr bool FIRST = !OWNERS && STREAM;
    const unsigned tid = threadIdx.x, first = blockIdx.x * l.chunk, count = first < p.N ? min(l.chunk, p.N - first) : 0u;
    Ctl* const ctl = p.ctl;
    const unsigned W = (unsigned)p.W;
    const unsigned tmax = p.max_steps > 0 ? (unsigned)p.max_steps : 0x7FFFFFFFu;
    if (tid < 5u) s_sum[tid] = 0u;
    if (tid == 5u) s_ep = 0u;
    __syncthreads();
    Tally tally{0u, 0u, 0u, 0u, 0u};
    unsigned s = 0u, t = 0u, id = 0u, own = NOBODY; float target = 0.f, value = 0.f;
    uint2 w = make_uint2(0u, 0u);                                  // the policy draw of the step at hand
    // streamed state, by slot of the block
    const size_t room = HOME == Home::Shared ? l.chunk : p.N, at0 = HOME == Home::Shared ? 0u : first;
    unsigned char* const base = HOME == Home::Shared ? arrays : p.gp.state;
    uint2* const m_pos = reinterpret_cast<uint2*>(base) + at0;
    float2* const m_tv = reinterpret_cast<float2*>(base + room * 8u) + at0;
    unsigned* const m_id = reinterpret_cast<unsigned*>(base + room * 16u) + at0;
    unsigned* const m_own = reinterpret_cast<unsigned*>(base + room * 20u) + at0;
    const unsigned end = STREAM ? (count + GB - 1u) / GB * GB : GB;      // slots, rounded up: whole warps take every turn
    auto draw = [&](unsigned i, unsigned long long g) -> uint2 {
        const U4 r = philox4x32_10(p.env_offset + i, 0u, (unsigned)g, (unsigned)(g >> 32), p.policy_keys);
        return make_uint2(r.x, r.y);
    };
    unsigned long long g = p.step + skip;
    for (unsigned j = tid; j < end; j += GB) {
        if (j >= count) continue;
        const int4 r = work[first + j];
        s = (unsigned)r.y * W + (unsigned)r.x; t = (unsigned)r.z; id = (unsigned)r.w;
        if (STREAM) { m_pos[j] = make_uint2(s, t); m_id[j] = id; m_own[j] = NOBODY; } else w = draw(id, g);
    }
    EpsilonIndex eps_index(p, l, PLAIN);
    if (l.eps_mode == 1) eps_index.at += skip;
    float eps = __ldg(p.eps_tab + eps_index.at);
    if (!PLAIN && l.eps_mode == 2) {       // every block has read the finished episodes before any adds those of the first step
        space.arrive();
        if (!space.wait()) return;
    }

    for (unsigned step = skip; step < l.steps; ++step, ++g) {
        const unsigned par = (unsigned)g & 1u;
        const unsigned thr = !(eps > 0.0f) ? 0u : eps >= 1.0f ? (1u << 24) : (unsigned)ceilf(eps * 16777216.0f);   // explore iff (w0 >> 8) < thr

        // ---- count ----
        for (unsigned j = tid; j < end; j += GB) {
            const bool act = j < count;
            if (STREAM) {
                unsigned before = NOBODY;
                if (act) { const uint2 q = m_pos[j]; s = q.x; t = q.y; id = m_id[j]; before = m_own[j]; }
                w = draw(id, g);
                if (before != NOBODY) space.clear(par ^ 1u, before);
            }
            unsigned mv = 0u; float4 row = make_float4(0.f, 0.f, 0.f, 0.f);
            if (act) { row = space.row(s); mv = space.moves(s); }
            if (!STREAM && own != NOBODY) space.clear(par ^ 1u, own);
            const int a = (w.x >> 8) < thr ? (int)(w.y & 3u) : argmax4(row);
            own = act ? s * 4u + (unsigned)a : NOBODY;
            mv >>= a;                                 // bit 0: the move is blocked, bit 4: it ends on a goal
            // a whole warp on one (cell, action) -- everybody at a common start cell -- counts once
            const bool common = __all_sync(FULL, own == __shfl_sync(FULL, own, 0));
            bool applies = act && !OWNERS;
            if (act && (!common || (tid & 31u) == 0u)) {
                const unsigned n = common ? 32u : 1u;
                if (OWNERS) applies = space.add(par, own, n) == 0u; else space.count(par, own, n);
            }
            const unsigned there = a == 0 ? s - W : a == 1 ? s + 1u : a == 2 ? s + W : s - 1u;
            s = (mv & 1u) ? s : there;
            float4 next = make_float4(0.f, 0.f, 0.f, 0.f);
            if (act) next = space.row(s);             // side by side with the atomic
            const bool done = (mv & 16u) != 0u;
            value = pick(row, a);
            float m = max4(next);
            if (!PLAIN && p.legacy_clamp && m < 0.0f) m = 0.0f;
            float r = -0.01f;
            if (!PLAIN && p.ntraps && (mv & 1u)) { const unsigned y = s / W; r = blocked_step_reward(p, (int)(s - y * W), (int)y, a); }     // a trap charges its penalty
            target = done ? 1.0f : __fmaf_rn(p.gamma, m, r);
            t = min(t + 1u, STEP_SAT);
            if (OWNERS && !applies) own = NOBODY;
            if (!act) continue;
            if (!PLAIN && l.trace && step + 1u == l.steps) { p.tr_a[id] = a; p.tr_r[id] = done ? 1.0f : r; p.tr_d[id] = done ? 1 : 0; }
            if (done || t >= tmax) {
                s = sample_start(p, p.env_offset + id, g + 1ull, TAG_START); t = 0u;
                if (done) ++tally.goals; else ++tally.timeouts;
                if (!PLAIN && l.eps_mode == 2) atomicAdd(&s_ep, 1u);
            }
            if (STREAM) {
                m_pos[j] = make_uint2(s, t);
                m_own[j] = own;
                if (applies) m_tv[j] = make_float2(target, value);
            }
        }
        if (!PLAIN && l.eps_mode == 2) {              // finished episodes of this step, before anybody can pass the barrier
            __syncthreads();
            if (tid == 0u && s_ep) { atomicAdd(&ctl->episodes, (unsigned long long)s_ep); s_ep = 0u; }
        }
        space.arrive();
        if (!STREAM) { w = draw(id, g + 1ull); asm volatile("" : "+r"(w.x), "+r"(w.y)); }      // behind the barrier's latency, and kept there
        if (!space.wait()) return;

        // ---- apply ----
        for (unsigned j = tid; j < end; j += GB) {
            if (STREAM) own = j < count ? m_own[j] : NOBODY;
            unsigned n = 0u;
            bool applies = own != NOBODY;
            if (applies) {
                if (STREAM) { const float2 q = m_tv[j]; target = q.x; value = q.y; }
                uint4 c = space.counts(par, own >> 2);
                const unsigned a = own & 3u;
                n = a == 0u ? c.x : a == 1u ? c.y : a == 2u ? c.z : c.w;
                const unsigned tot = c.x + c.y + c.z + c.w;
                if (tot > 1u) tally.conf += OWNERS ? n : 1u;
                if (tot > CROWDED_CELL) {             // (marks on the counters make the sum larger, or leave it as it is: it stays above)
                    unsigned marked = 0u;
                    if (!OWNERS) { marked = n & NOTED; c.x &= ~NOTED; c.y &= ~NOTED; c.z &= ~NOTED; n &= ~NOTED; ++tally.on_crowded; }
                    const unsigned below = a == 0u ? 0u : a == 1u ? c.x : a == 2u ? c.x + c.y : c.x + c.y + c.z;       // the lowest chosen action speaks for the cell
                    if (OWNERS) { if (below == 0u) { ++tally.crowded; tally.on_crowded += tot; } }
                    else if (!FIRST) { if (below == 0u && !space.note(par, own)) ++tally.crowded; }
                    else if (below == 0u || n > CROWDED_CELL) {
                        bool one = !marked;              // one lane of a warp tries
                        if (one && n > CROWDED_CELL) one = (tid & 31u) == (unsigned)__ffs((int)__match_any_sync(__activemask(), own)) - 1u;
                        one = one && !space.note(par, own);
                        if (one && below == 0u) ++tally.crowded;
                        applies = one || n <= CROWDED_CELL;
                    }
                }
            }
            if (FIRST) __syncwarp();                  // the lanes' rounds side by side, however they got here
            if (applies) space.store(own, apply_counted(value, target, p.lr, n));
        }
        eps_index.next(p, l, PLAIN, 0u, false);        // between the two barriers: nobody adds to the episodes before everybody has passed the second
        space.arrive();
        if (l.eps_mode && step + 1u < l.steps) eps = __ldg(p.eps_tab + eps_index.at);
        if (!space.wait()) return;
    }

    // ---- the last step's counters back to zero, the records out, the sums ----
    for (unsigned j = tid; j < end; j += GB) {
        if (j >= count) continue;
        if (STREAM) { const uint2 q = m_pos[j]; s = q.x; t = q.y; id = m_id[j]; own = m_own[j]; }
        if (own != NOBODY) space.clear(((unsigned)g & 1u) ^ 1u, own);
        const unsigned y = s / W;
        work[first + j] = make_int4((int)(s - y * W), (int)y, (int)t, (int)id);
    }
    add_tallies(p, l, tally, s_sum, l.eps_mode != 2, eps);
}

// Whether a launch needs none of the options PLAIN leaves out.
inline bool plain(const Params& p, const StepLaunch& l) { return !p.ntraps && !p.legacy_clamp && !l.trace && l.eps_mode != 2; }

}  // namespace cudarl
