// gather_engine.cu -- the fused train step for worlds whose table stays in L2: many steps per launch, one thread per environment.
//
// The tile engine (tile_engine.cu) streams the whole table through shared memory in every step, one warp per tile.  Where the table
// fits L2 that is not needed, and where the population bunches up -- everybody on the few paths to the goals, late in training -- a
// step lasts as long as the warp with the fullest tile: 256 x 256 cells with 65,536 environments went from 11 us a step to 116.
// Here the environments are spread evenly over the threads of ONE cooperative launch that runs many steps, and a step is
//
//   count   every environment reads the row of its cell, chooses its action, counts itself in the (cell, action) counter with an
//           atomic, and moves on; the first to count on a (cell, action) owns it and takes the TD target from Q_t;
//   -- barrier of the grid --
//   apply   the owner applies the update as many times as were counted, and stores the one table entry;
//   -- barrier of the grid --
//
// which is the tile engine's rule (all updates of one (cell, action) within a step are the same map, so only their number matters)
// with the counters in L2 instead of shared memory.  Counters alternate by step parity; the owner clears its counter in the next
// step's count phase, when everybody has read it and nobody uses that parity.
//
// A population that fits the threads stays in registers for the whole launch (EPT environments per thread); a larger one is
// streamed through in batches.  What bounds it: two grid barriers (1.3 - 1.7 us each) and four dependent L2 accesses per step while
// the population is small, scattered 32-byte sectors in L2 when it is large.
//
// Reference semantics: those of tile_engine.cu.
#include "kernels.cuh"
#include "rules.cuh"

namespace cudarl {

constexpr unsigned GB = 512u;                       // threads per block
constexpr unsigned NOBODY = 0xFFFFFFFFu;
constexpr unsigned long long GRID_WAIT_NS = 2000000000ull;

// A barrier of all blocks of the launch: an arrival counter that only ever grows (the host passes its value at the launch).  Bounded
// in time: a block that waits two seconds records the failure, and everybody leaves.
struct GridBarrier {
    unsigned* counter; unsigned target; unsigned blocks;
    __device__ __forceinline__ void arrive() {      // this block's writes are visible to whoever sees the arrival
        __syncthreads();
        target += blocks;
        if (threadIdx.x == 0u) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(counter) : "memory");
    }
    __device__ __forceinline__ bool wait(Ctl* ctl, unsigned* s_ok) {
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
            *s_ok = ok;
        }
        __syncthreads();
        return *s_ok != 0u;
    }
};

// What one environment needs between the two phases of a step, and what the launch sums up.
struct Tally { unsigned goals, timeouts, conf, crowded, on_crowded; };

// The update of (cell, action) `own` from the counted number of environments on it: the map q <- fma(lr, d - q, q) as often as counted.
// It is a contraction, so a long run ends at its fixed point: once the value stops changing it never changes again.
__device__ __forceinline__ float apply_counted(float v, float d, float lr, unsigned n) {
    for (unsigned i = 0; i < n; ++i) {
        const float w = __fmaf_rn(lr, __fsub_rn(d, v), v);
        if (__float_as_uint(w) == __float_as_uint(v)) break;
        v = w;
    }
    return v;
}

// EPT environments per thread and turn.  STREAM: a block owns `chunk` environments and takes them GB * EPT at a time, its state
// (records, ownership) in global memory; else chunk == GB * EPT and everything stays in registers for the whole launch.
template <int EPT, bool STREAM>
__global__ void __launch_bounds__(GB, STREAM ? 2 : 1) k_gather_steps(const __grid_constant__ Params p, const __grid_constant__ GatherLaunch l) {
    __shared__ unsigned s_ok, s_sum[5], s_ep;
    const unsigned tid = threadIdx.x, first = blockIdx.x * l.chunk, last = min(first + l.chunk, p.N);
    const GatherP& gp = p.gp;
    Ctl* const ctl = p.ctl;
    GridBarrier bar{gp.barrier, l.barrier_base, gridDim.x};
    if (tid < 5u) s_sum[tid] = 0u;
    if (tid == 5u) s_ep = 0u;
    if (tid == 6u) s_ok = (*reinterpret_cast<volatile unsigned*>(&ctl->error) & ERR_COPY_TIMEOUT) ? 0u : 1u;   // the barrier counter is off since then
    __syncthreads();
    if (s_ok == 0u) return;
    if (p.tp.wait_polls) {                           // tests only: a wait that nothing can end, bounded by a number of looks
        unsigned v = 0u;
        for (unsigned it = 0; it < p.tp.wait_polls; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(gp.barrier) : "memory");
            if ((int)(v - (bar.target + 0x40000000u)) >= 0) return;
        }
        if (tid == 0u) atomicOr(&ctl->error, ERR_COPY_TIMEOUT);
        return;
    }
    const unsigned tmax = p.max_steps > 0 ? (unsigned)p.max_steps : 0x7FFFFFFFu;
    const int dW = p.W;
    Tally tally{0u, 0u, 0u, 0u, 0u};
    int x[EPT], y[EPT]; unsigned t[EPT], own[EPT]; float dd[EPT], vv[EPT];
    U4 w[EPT];
    auto slot = [&](unsigned turn, int k) -> unsigned { return first + (turn * (unsigned)EPT + (unsigned)k) * GB + tid; };
    auto policy = [&](unsigned i, unsigned long long g) -> U4 { return philox4x32_10(p.env_offset + i, 0u, (unsigned)g, (unsigned)(g >> 32), p.k0, p.k1 ^ TAG_POLICY); };
    unsigned long long g = p.step;
    if (!STREAM) {
#pragma unroll
        for (int k = 0; k < EPT; ++k) {
            own[k] = NOBODY;
            const unsigned i = slot(0u, k);
            if (i < last) { const int4 r = p.st[i]; x[k] = r.x; y[k] = r.y; t[k] = (unsigned)r.z; w[k] = policy((unsigned)i, g); }
        }
    }
    unsigned eps_at = l.eps_mode == 2 ? *reinterpret_cast<volatile unsigned*>(&ctl->eps_idx) : p.eps_idx;
    float eps = 0.0f;

    for (unsigned step = 0; step < l.steps; ++step, ++g) {
        const unsigned par = (unsigned)(g & 1ull);
        unsigned* const cnt = gp.cnt[par]; unsigned* const cnt_old = gp.cnt[par ^ 1u];
        eps = __ldg(p.eps_tab + eps_at);
        const unsigned thr = !(eps > 0.0f) ? 0u : eps >= 1.0f ? (1u << 24) : (unsigned)ceilf(eps * 16777216.0f);   // explore iff (w0 >> 8) < thr
        const bool trace = l.trace && step + 1u == l.steps;

        // ---- count ----
        for (unsigned turn = 0; turn * (unsigned)EPT * GB < l.chunk; ++turn) {
            bool act[EPT]; unsigned s[EPT], mv[EPT], old[EPT], idx[EPT]; float4 row[EPT];
            if (STREAM) {
                unsigned before[EPT]; int4 r[EPT];
#pragma unroll
                for (int k = 0; k < EPT; ++k) {
                    const unsigned i = slot(turn, k);
                    before[k] = NOBODY;
                    if (i < last) { r[k] = p.st[i]; before[k] = step ? gp.own[i] : NOBODY; }
                }
#pragma unroll
                for (int k = 0; k < EPT; ++k) {
                    const unsigned i = slot(turn, k);
                    if (i < last) { x[k] = r[k].x; y[k] = r[k].y; t[k] = (unsigned)r[k].z; w[k] = policy(i, g); }
                    if (before[k] != NOBODY) cnt_old[before[k]] = 0u;
                }
            } else {
#pragma unroll
                for (int k = 0; k < EPT; ++k) if (own[k] != NOBODY) cnt_old[own[k]] = 0u;
            }
#pragma unroll
            for (int k = 0; k < EPT; ++k) {
                act[k] = slot(turn, k) < last;
                s[k] = 0u; mv[k] = 0u; row[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (act[k]) { s[k] = (unsigned)y[k] * (unsigned)dW + (unsigned)x[k]; row[k] = p.Q[s[k]]; mv[k] = __ldg(gp.mv + s[k]); }
            }
            float4 next[EPT]; int a[EPT]; bool blocked[EPT], done[EPT];
#pragma unroll
            for (int k = 0; k < EPT; ++k) {
                a[k] = argmax4(row[k]);
                if ((w[k].x >> 8) < thr) a[k] = (int)(w[k].y & 3u);
                blocked[k] = (mv[k] >> a[k]) & 1u; done[k] = (mv[k] >> (a[k] + 4)) & 1u;
                idx[k] = act[k] ? s[k] * 4u + (unsigned)a[k] : NOBODY;
                // a whole warp on one (cell, action) -- everybody at a common start cell -- counts once
                const unsigned lead = __shfl_sync(FULL, idx[k], 0);
                const bool common = __all_sync(FULL, idx[k] == lead);
                old[k] = 1u;
                if (act[k] && (!common || (tid & 31u) == 0u)) old[k] = atomicAdd(cnt + idx[k], common ? 32u : 1u);
                const int dx = blocked[k] ? 0 : (int)(signed char)(0xFF000100u >> (8 * a[k])), dy = blocked[k] ? 0 : (int)(signed char)(0x000100FFu >> (8 * a[k]));
                next[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (act[k]) {
                    x[k] += dx; y[k] += dy;
                    if (!STREAM && !done[k]) next[k] = p.Q[(unsigned)y[k] * (unsigned)dW + (unsigned)x[k]];      // everybody at once: one latency less
                }
            }
#pragma unroll
            for (int k = 0; k < EPT; ++k) {
                own[k] = NOBODY;
                if (!act[k]) continue;
                const unsigned i = slot(turn, k);
                if (old[k] == 0u) {
                    if (STREAM && !done[k]) next[k] = p.Q[(unsigned)y[k] * (unsigned)dW + (unsigned)x[k]];       // owners only: fewer sectors
                    own[k] = idx[k]; vv[k] = pick(row[k], a[k]);
                }
                float m = max4(next[k]);
                if (p.legacy_clamp && m < 0.0f) m = 0.0f;
                const float r = (blocked[k] && p.ntraps) ? blocked_step_reward(p, x[k], y[k], a[k]) : -0.01f;    // a trap charges its penalty
                dd[k] = done[k] ? 1.0f : __fmaf_rn(p.gamma, m, r);
                if (trace) { p.tr_a[i] = a[k]; p.tr_r[i] = done[k] ? 1.0f : r; p.tr_d[i] = done[k] ? 1 : 0; }
                t[k] = min(t[k] + 1u, STEP_SAT);
                if (done[k] || t[k] >= tmax) {
                    const unsigned c = sample_start(p, p.env_offset + i, g + 1ull, TAG_START);
                    y[k] = (int)(c / (unsigned)dW); x[k] = (int)(c - (unsigned)y[k] * (unsigned)dW); t[k] = 0u;
                    if (done[k]) ++tally.goals; else ++tally.timeouts;
                    if (l.eps_mode == 2) atomicAdd(&s_ep, 1u);
                }
                if (STREAM) {
                    p.st[i] = make_int4(x[k], y[k], (int)t[k], (int)i);
                    gp.own[i] = own[k];
                    if (own[k] != NOBODY) gp.dv[i] = make_float2(dd[k], vv[k]);
                }
            }
        }
        if (l.eps_mode == 2) {                        // finished episodes of this step, before anybody can pass the barrier
            __syncthreads();
            if (tid == 0u && s_ep) { atomicAdd(&ctl->episodes, (unsigned long long)s_ep); s_ep = 0u; }
        }
        bar.arrive();
        if (!STREAM) {
#pragma unroll
            for (int k = 0; k < EPT; ++k) w[k] = policy(slot(0u, k), g + 1ull);                                 // behind the barrier's latency
        }
        if (!bar.wait(ctl, &s_ok)) return;

        // ---- apply ----
        for (unsigned turn = 0; turn * (unsigned)EPT * GB < l.chunk; ++turn) {
            uint4 c[EPT];
            if (STREAM) {
#pragma unroll
                for (int k = 0; k < EPT; ++k) { const unsigned i = slot(turn, k); own[k] = i < last ? gp.own[i] : NOBODY; }
#pragma unroll
                for (int k = 0; k < EPT; ++k) if (own[k] != NOBODY) { const float2 q = gp.dv[slot(turn, k)]; dd[k] = q.x; vv[k] = q.y; }
            }
#pragma unroll
            for (int k = 0; k < EPT; ++k) if (own[k] != NOBODY) c[k] = *reinterpret_cast<const uint4*>(cnt + (own[k] & ~3u));
#pragma unroll
            for (int k = 0; k < EPT; ++k) {
                if (own[k] == NOBODY) continue;
                const unsigned a = own[k] & 3u, n = a == 0u ? c[k].x : a == 1u ? c[k].y : a == 2u ? c[k].z : c[k].w, tot = c[k].x + c[k].y + c[k].z + c[k].w;
                const unsigned below = a == 0u ? 0u : a == 1u ? c[k].x : a == 2u ? c[k].x + c[k].y : c[k].x + c[k].y + c[k].z;
                if (tot > 1u) tally.conf += n;
                if (tot > CROWDED_CELL && below == 0u) { ++tally.crowded; tally.on_crowded += tot; }             // the lowest chosen action speaks for the cell
                reinterpret_cast<float*>(p.Q)[own[k]] = apply_counted(vv[k], dd[k], p.lr, n);
            }
        }
        // the index of the next step's epsilon: by step, or by the episodes finished so far (read between the two barriers: nobody
        // adds to them before everybody has passed the second)
        if (l.eps_mode == 1) ++eps_at;
        else if (l.eps_mode == 2) {
            const unsigned long long kk = *reinterpret_cast<volatile unsigned long long*>(&ctl->episodes) / (unsigned long long)p.N;
            const unsigned long long rel = kk > ctl->eps_base_k ? kk - ctl->eps_base_k : 0ull;
            eps_at = (unsigned)(rel < (unsigned long long)(ctl->eps_len - 1u) ? rel : (unsigned long long)(ctl->eps_len - 1u));
        }
        bar.arrive();
        if (!bar.wait(ctl, &s_ok)) return;
    }

    // ---- the last step's counters back to zero, the records out, the sums ----
    unsigned* const cnt = gp.cnt[(unsigned)((g - 1ull) & 1ull)];
    for (unsigned turn = 0; turn * (unsigned)EPT * GB < l.chunk; ++turn) {
#pragma unroll
        for (int k = 0; k < EPT; ++k) {
            const unsigned i = slot(turn, k);
            if (i >= last) continue;
            if (STREAM) own[k] = gp.own[i]; else p.st[i] = make_int4(x[k], y[k], (int)t[k], (int)i);
            if (own[k] != NOBODY) cnt[own[k]] = 0u;
        }
    }
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
        if (l.eps_mode != 2 && s_sum[0] + s_sum[1]) atomicAdd(&ctl->episodes, (unsigned long long)(s_sum[0] + s_sum[1]));
        if (s_sum[2]) atomicAdd(&ctl->conflicts, (unsigned long long)s_sum[2]);
        if (s_sum[3]) { atomicAdd(&ctl->long_chains, (unsigned long long)s_sum[3]); atomicAdd(&ctl->general, (unsigned long long)s_sum[4]); }
        if (blockIdx.x == 0u && l.eps_mode == 2) { ctl->eps_used = eps; ctl->eps_idx = eps_at; }
    }
}

// ------------------------------------------------------------------------------------------------
// The move byte of every cell (see move_byte in rules.cuh), row by row.
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

// How the population is spread over the launch: as few environments per thread as let one block per SM hold them all in registers,
// else streamed by two blocks per SM.
void gather_plan(Params& p, int sms) {
    GatherP& gp = p.gp;
    const unsigned n = p.N ? p.N : 1u, s = (unsigned)(sms > 0 ? sms : 1);
    for (gp.ept = 1u; gp.ept <= 4u; gp.ept <<= 1) if ((n + GB * gp.ept - 1u) / (GB * gp.ept) <= s) break;
    if (gp.ept <= 4u) { gp.chunk = GB * gp.ept; gp.grid = (n + gp.chunk - 1u) / gp.chunk; gp.stream = 0u; return; }
    gp.ept = 2u; gp.stream = 1u;
    gp.chunk = ((n + 2u * s - 1u) / (2u * s) + 31u) / 32u * 32u;
    gp.grid = (n + gp.chunk - 1u) / gp.chunk;
}
unsigned gather_barriers(unsigned steps) { return 2u * steps; }

template <int EPT, bool STREAM>
static cudaError_t launch_one(const Params& p, const GatherLaunch& l, cudaStream_t st) {
    void* args[2] = {const_cast<Params*>(&p), const_cast<GatherLaunch*>(&l)};
    return cudaLaunchCooperativeKernel((const void*)k_gather_steps<EPT, STREAM>, dim3(p.gp.grid), dim3(GB), args, 0, st);
}
cudaError_t launch_gather_steps(const Params& p, const GatherLaunch& l, cudaStream_t st) {
    if (p.gp.stream) return launch_one<2, true>(p, l, st);
    switch (p.gp.ept) {
        case 1u: return launch_one<1, false>(p, l, st);
        case 2u: return launch_one<2, false>(p, l, st);
        default: return launch_one<4, false>(p, l, st);
    }
}

}  // namespace cudarl
