// kernels.cu -- sm_100a kernels of the batched grid-world + tabular Q-learning path other than the fused
// train step (tile_engine.cu) and the greedy rollout (rollout.cu): environment reset and caller-driven stepping, the
// ordered TD update of caller-supplied transitions (update_batch) and table initialisation.
//
// Data layout in HBM (per context = per GPU):
//   st [N]   environment state, one int4 {x, y, t, id} per environment (record k = environment k outside
//            train steps), one aligned 16-byte vector load/store per thread;
//   Q        the table, one float4 per grid cell (index y*W + x): one vector load is the whole action row;
//   cw       one 16-bit word per cell holding the cell's class bits (obstacle, goal);
//   ent / mailbox   collision entries and chain heads of update_batch.
//
// Reference semantics (paths relative to the CudaRL-Arena project root):
//   step        src/environment.cu:17-48, obstacle test src/kernels.cu:29-44, goal src/kernels.cu:56-59
//   reset       src/environment.cu:6-14
//   TD update   src/kernels.cu:96-114 (true max as in src/gpu/kernels.cu:36-45, src/train.py:134)
#include "kernels.cuh"
#include "rules.cuh"
#include <cstdio>

namespace cudarl {

// The cell `action` leads to from (x, y) if nothing is in the way there (its own at the edge of the grid, or for any action but 0..3).
__device__ __forceinline__ unsigned target_cell(const World& p, int x, int y, int action) {
    const int nx = x + (action == 1) - (action == 3), ny = y + (action == 2) - (action == 0);
    const bool inb = nx >= 0 && nx < p.W && ny >= 0 && ny < p.H;
    return inb ? (unsigned)ny * (unsigned)p.W + (unsigned)nx : (unsigned)y * (unsigned)p.W + (unsigned)x;
}

// chain heads are indexed by the low bits of the cell: neighbouring cells -> neighbouring slots
__device__ __forceinline__ unsigned mb_slot(const Params& p, unsigned cell) { return cell & (p.mb_slots - 1u); }

__global__ void k_reset_all(const __grid_constant__ World p) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.N) return;
    unsigned e = (unsigned)p.st[i].w;
    unsigned c = sample_start(p, p.env_offset + e, p.step, TAG_START);
    p.st[i] = make_int4((int)(c % (unsigned)p.W), (int)(c / (unsigned)p.W), 0, (int)e);
    if (p.reward) { p.reward[e] = 0.0f; p.done[e] = 0; }
}

__global__ void k_ids_identity(const __grid_constant__ World p) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.N) p.st[i].w = (int)i;
}
// overwrite x / y / t of environment-ordered records from caller arrays (any of them may be null)
__global__ void k_import_state(const __grid_constant__ World p, const int* x, const int* y, const int* t) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.N) return;
    int4 r = p.st[i];
    if (x) r.x = x[i];
    if (y) r.y = y[i];
    if (t) r.z = t[i];
    r.w = (int)i;
    p.st[i] = r;
}
// x[N] | y[N] | t[N] in environment order, into the spare copy or straight into the mapped stage
__global__ void k_export_state(const __grid_constant__ World p, int* __restrict__ out, Handover h) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.N) {
        const int4 r = p.st[i];
        out[r.w] = r.x; out[p.N + r.w] = r.y; out[2u * p.N + r.w] = r.z;
    }
    if (last_to_finish<true>(p)) box_put_error(p, h);
}
// Small results: device memory into mapped host memory, 16 bytes per thread and turn (both ends are 16-byte aligned, the tail is
// copied to the next multiple of 16: every buffer of the context and the stage have that room).
__global__ void k_copy_out(const __grid_constant__ World p, CopySpan a, CopySpan b, Handover h) {
    const unsigned n = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (unsigned i = i0; i * 16u < a.bytes; i += n) reinterpret_cast<uint4*>(a.dst)[i] = reinterpret_cast<const uint4*>(a.src)[i];
    for (unsigned i = i0; i * 16u < b.bytes; i += n) reinterpret_cast<uint4*>(b.dst)[i] = reinterpret_cast<const uint4*>(b.src)[i];
    if (last_to_finish<true>(p)) box_put_error(p, h);
}
__global__ void k_post(const __grid_constant__ World p, Handover h) {
    const unsigned long long* const c[6] = {&p.ctl->episodes, &p.ctl->goals, &p.ctl->timeouts, &p.ctl->conflicts, &p.ctl->long_chains, &p.ctl->general};
#pragma unroll
    for (unsigned k = 0; k < 6u; ++k) if (threadIdx.x == k) box_put64(h, 1u + 2u * k, *c[k]);       // one counter per lane
    if (threadIdx.x == 6u) box_put(h, 13u, __float_as_uint(p.ctl->eps_used));
    if (threadIdx.x == 7u) box_put_error(p, h);
}

// ------------------------------------------------------------------------------------------------
// Collision folding.
__device__ __forceinline__ void cswap(unsigned long long& ka, float& va, unsigned long long& kb, float& vb) {
    if (ka > kb) { unsigned long long tk = ka; ka = kb; kb = tk; float tv = va; va = vb; vb = tv; }
}

// Block-wide bitonic sort of n2 (power of two) key/value pairs in shared or global memory.
__device__ void block_bitonic(unsigned long long* keys, float* vals, unsigned n2) {
    for (unsigned k = 2; k <= n2; k <<= 1) {
        for (unsigned j = k >> 1; j > 0; j >>= 1) {
            for (unsigned i = threadIdx.x; i < n2; i += blockDim.x) {
                unsigned ixj = i ^ j;
                if (ixj > i) {
                    unsigned long long a = keys[i], b = keys[ixj];
                    bool up = (i & k) == 0;
                    if ((a > b) == up) { keys[i] = b; keys[ixj] = a; float t = vals[i]; vals[i] = vals[ixj]; vals[ixj] = t; }
                }
            }
            __syncthreads();
        }
    }
}

// Fold a sorted run (same cell) starting at index j of keys/vals; returns nothing, writes Q_{t+1}.
__device__ void apply_run(const Params& p, const unsigned long long* keys, const float* vals, unsigned j, unsigned n) {
    unsigned w0 = (unsigned)(keys[j] >> 32);
    unsigned cellp = w0 >> 2;              // (cell << 1) | parity
    unsigned cell = w0 >> 3;
    float4 row = __ldcg(p.Q + cell);
    for (; j < n; ++j) {
        unsigned wj = (unsigned)(keys[j] >> 32);
        if ((wj >> 2) != cellp) break;
        fold(row, (int)(wj & 3u), p.lr, vals[j]);
    }
    p.Q[cell] = row;          // in place: the targets were taken before this kernel started, and one thread owns the cell
}

constexpr unsigned LONG_SMEM = 1024;   // chain entries sorted in shared memory; longer chains use the global scratch
constexpr int SHORT_MAX = 8;           // chain entries folded in registers by one thread

// One long chain, whole block: count its entries (one hop per run), pick shared memory or a slice of the
// global scratch, copy the runs (one warp per run, batches of 256 runs), bitonic-sort by (cell, action, id)
// and let the first thread of every cell run fold it.
__device__ void process_long(const Params& p, unsigned head1, unsigned long long* s_keys, float* s_vals,
                             unsigned* s_bcast) {
    __shared__ unsigned s_run[BLOCK], s_off[BLOCK];
    if (threadIdx.x == 0) {
        unsigned q = head1, L = 0, hops = 0;
        while (q && hops <= p.ent_cap) {          // a chain can never have more runs than the entry array has slots
            L += (q >> LINK_POS_BITS) + 1u; ++hops;
            q = p.ent[(q & LINK_POS_MASK) - 1u].w;
        }
        unsigned n2 = 1; while (n2 < L) n2 <<= 1;
        unsigned base = 0xFFFFFFFFu;
        if (q || L > p.ent_cap) { atomicOr(&p.ctl->error, ERR_CHAIN_CYCLE); base = 0xFFFFFFFEu; }
        else if (L > LONG_SMEM) {
            base = atomicAdd(&p.ctl->scratch_cursor, n2);
            if (base + n2 > p.sc_cap) { atomicOr(&p.ctl->error, ERR_SCRATCH_OVERFLOW); base = 0xFFFFFFFEu; }
        }
        s_bcast[0] = L; s_bcast[1] = n2; s_bcast[2] = base;
    }
    __syncthreads();
    const unsigned L = s_bcast[0], n2 = s_bcast[1], base = s_bcast[2];
    if (base != 0xFFFFFFFEu) {
        unsigned long long* keys = (base == 0xFFFFFFFFu) ? s_keys : p.sc_key + base;
        float* vals = (base == 0xFFFFFFFFu) ? s_vals : p.sc_val + base;
        __shared__ unsigned s_q, s_nb, s_done_entries;
        if (threadIdx.x == 0) { s_q = head1; s_done_entries = 0; }
        __syncthreads();
        while (true) {                               // batches of up to 256 runs; ends when the chain is exhausted
            if (threadIdx.x == 0) {
                unsigned q = s_q, nb = 0, off = s_done_entries;
                while (q && nb < (unsigned)BLOCK) {
                    s_run[nb] = q; s_off[nb] = off; off += (q >> LINK_POS_BITS) + 1u; ++nb;
                    q = p.ent[(q & LINK_POS_MASK) - 1u].w;
                }
                s_q = q; s_nb = nb; s_done_entries = off;
            }
            __syncthreads();
            const unsigned nb = s_nb;
            if (nb == 0u) break;
            for (unsigned r = threadIdx.x >> 5; r < nb; r += BLOCK / 32) {
                const unsigned link = s_run[r], pos0 = (link & LINK_POS_MASK) - 1u, len = (link >> LINK_POS_BITS) + 1u;
                const unsigned j = threadIdx.x & 31u;
                if (j < len && s_off[r] + j < L) {
                    const uint4 e = p.ent[pos0 + j];
                    keys[s_off[r] + j] = ((unsigned long long)e.x << 32) | e.y; vals[s_off[r] + j] = __uint_as_float(e.z);
                }
            }
            __syncthreads();
        }
        for (unsigned i = L + threadIdx.x; i < n2; i += blockDim.x) { keys[i] = ~0ull; vals[i] = 0.0f; }
        __syncthreads();
        block_bitonic(keys, vals, n2);
        for (unsigned j = threadIdx.x; j < L; j += blockDim.x) {
            unsigned cp = (unsigned)(keys[j] >> 34);
            if (j == 0 || (unsigned)(keys[j - 1] >> 34) != cp) apply_run(p, keys, vals, j, L);
        }
    }
    __syncthreads();
}

constexpr unsigned MED_MAX = 32;                         // chain entries ranked by one warp with shuffles
constexpr unsigned MED_CHUNKS = LONG_SMEM / MED_MAX;     // medium chains a block can stage in shared memory

// One warp orders a staged chain of L <= 32 entries by (cell, action, index) with a shuffle ranking
// (indices are unique, so ranks are a permutation), then the first lane of every cell run folds it.
__device__ void process_medium(const Params& p, unsigned long long* keys, float* vals, unsigned L) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned long long key = lane < L ? keys[lane] : ~0ull;
    float val = lane < L ? vals[lane] : 0.0f;
    unsigned rank = 0;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        unsigned long long other = __shfl_sync(0xFFFFFFFFu, key, k);
        rank += (other < key) ? 1u : 0u;
    }
    __syncwarp();
    if (lane < L) { keys[rank] = key; vals[rank] = val; }
    __syncwarp();
    if (lane < L) {
        unsigned cp = (unsigned)(keys[lane] >> 34);
        if (lane == 0 || (unsigned)(keys[lane - 1] >> 34) != cp) apply_run(p, keys, vals, lane, L);
    }
    __syncwarp();
}

// Collision folding, one thread per ACTIVE mailbox slot (the producers list every slot they were the
// first to hook a chain into, so this kernel only visits slots that have work).  A slot's chain links
// RUNS of consecutive entries (one run = the lanes of one warp on one cell).  The owning thread gathers
// the chain's entries:
//   <= 8 entries   in registers, ordered by a sorting network and folded by that thread;
//   <= 32 entries  staged in shared memory by that thread, ordered and folded by one warp;
//   longer         queued for k_fix_long (one warp per chain up to 256 entries, then one block per chain).
__device__ __forceinline__ void flush_row(const Params& p, unsigned cellpar, const float4& row) { p.Q[cellpar >> 1] = row; }

__global__ void __launch_bounds__(BLOCK) k_fix(Params p) {
    __shared__ unsigned long long s_keys[LONG_SMEM];
    __shared__ float s_vals[LONG_SMEM];
    __shared__ unsigned s_medlen[MED_CHUNKS];
    __shared__ unsigned s_nmed;
    const unsigned nactive = p.ctl->active_count;      // slots that received a chain in this call
  for (unsigned tile = blockIdx.x; tile * BLOCK < nactive; tile += gridDim.x) {
    if (threadIdx.x == 0) s_nmed = 0;
    __syncthreads();
    const unsigned ai = tile * BLOCK + threadIdx.x;
    const unsigned slot = ai < nactive ? p.active[ai] : 0u;
    const unsigned head = ai < nactive ? p.mailbox[slot] : 0u;
    if (head) {
        p.mailbox[slot] = 0u;                          // leave the mailbox empty for the next call
        unsigned long long k8[SHORT_MAX]; float v8[SHORT_MAX];
        unsigned q = head, pos = 0, rem = 0; bool fresh = false;
#pragma unroll
        for (int j = 0; j < SHORT_MAX; ++j) {
            if (rem == 0u && q) { pos = (q & LINK_POS_MASK) - 1u; rem = (q >> LINK_POS_BITS) + 1u; fresh = true; }
            if (rem) {
                const uint4 e = __ldcg(p.ent + pos);
                k8[j] = ((unsigned long long)e.x << 32) | e.y; v8[j] = __uint_as_float(e.z);
                if (fresh) { q = e.w; fresh = false; }
                ++pos; --rem;
            } else { k8[j] = ~0ull; v8[j] = 0.0f; }
        }
        if (rem == 0u && q == 0u) {
            cswap(k8[0],v8[0],k8[1],v8[1]); cswap(k8[2],v8[2],k8[3],v8[3]); cswap(k8[4],v8[4],k8[5],v8[5]); cswap(k8[6],v8[6],k8[7],v8[7]);
            cswap(k8[0],v8[0],k8[2],v8[2]); cswap(k8[1],v8[1],k8[3],v8[3]); cswap(k8[4],v8[4],k8[6],v8[6]); cswap(k8[5],v8[5],k8[7],v8[7]);
            cswap(k8[1],v8[1],k8[2],v8[2]); cswap(k8[5],v8[5],k8[6],v8[6]); cswap(k8[0],v8[0],k8[4],v8[4]); cswap(k8[3],v8[3],k8[7],v8[7]);
            cswap(k8[1],v8[1],k8[5],v8[5]); cswap(k8[2],v8[2],k8[6],v8[6]);
            cswap(k8[1],v8[1],k8[4],v8[4]); cswap(k8[3],v8[3],k8[6],v8[6]);
            cswap(k8[2],v8[2],k8[4],v8[4]); cswap(k8[3],v8[3],k8[5],v8[5]);
            cswap(k8[3],v8[3],k8[4],v8[4]);
            unsigned curcp = 0xFFFFFFFFu; float4 row = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < SHORT_MAX; ++j) {
                if (k8[j] != ~0ull) {
                    const unsigned w0 = (unsigned)(k8[j] >> 32), cp = w0 >> 2;
                    if (cp != curcp) {
                        if (curcp != 0xFFFFFFFFu) flush_row(p, curcp, row);
                        curcp = cp; row = __ldcg(p.Q + (cp >> 1));
                    }
                    fold(row, (int)(w0 & 3u), p.lr, v8[j]);
                }
            }
            if (curcp != 0xFFFFFFFFu) flush_row(p, curcp, row);
        } else {
            const unsigned chunk = atomicAdd(&s_nmed, 1u);
            bool staged = false;
            if (chunk < MED_CHUNKS) {
                unsigned long long* mk = s_keys + chunk * MED_MAX; float* mv = s_vals + chunk * MED_MAX;
#pragma unroll
                for (int j = 0; j < SHORT_MAX; ++j) { mk[j] = k8[j]; mv[j] = v8[j]; }
                unsigned L = SHORT_MAX;
                while ((rem || q) && L < MED_MAX) {
                    if (rem == 0u) { pos = (q & LINK_POS_MASK) - 1u; rem = (q >> LINK_POS_BITS) + 1u; fresh = true; }
                    const uint4 e = __ldcg(p.ent + pos);
                    mk[L] = ((unsigned long long)e.x << 32) | e.y; mv[L] = __uint_as_float(e.z);
                    if (fresh) { q = e.w; fresh = false; }
                    ++pos; --rem; ++L;
                }
                staged = (rem == 0u && q == 0u);
                s_medlen[chunk] = staged ? L : 0u;
            }
            if (!staged) {                              // hand the chain to k_fix_long
                const unsigned li = atomicAdd(&p.ctl->long_count, 1u);
                p.longq[li] = head;
            }
        }
    }
    __syncthreads();
    {   // medium chains: one warp each
        const unsigned nmed = s_nmed < MED_CHUNKS ? s_nmed : MED_CHUNKS;
        for (unsigned c = threadIdx.x >> 5; c < nmed; c += BLOCK / 32) {
            const unsigned L = s_medlen[c];
            if (L) process_medium(p, s_keys + c * MED_MAX, s_vals + c * MED_MAX, L);
        }
    }
    __syncthreads();
  }

}

// Long chains (more than 32 entries: cells crowded with environments).  First tier: one WARP per chain for up
// to 256 entries -- lane 0 hops from run to run, all lanes copy the run's entries into the warp's slice of
// shared memory, a warp-wide bitonic sort orders them by (cell, action, id), the first lane of every cell run
// applies it.  Chains that do not fit are left to the block.
constexpr unsigned WARP_LONG = 256;

__device__ bool process_long_warp(const Params& p, unsigned head, unsigned long long* keys, float* vals) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned q = head, L = 0, hops = 0; bool fits = true;
    while (q && hops <= p.ent_cap) {                  // q is warp-uniform
        const unsigned pos0 = (q & LINK_POS_MASK) - 1u, len = (q >> LINK_POS_BITS) + 1u;
        if (L + len > WARP_LONG) { fits = false; break; }
        uint4 e = make_uint4(0u, 0u, 0u, 0u);
        if (lane < len) { e = __ldcg(p.ent + pos0 + lane); keys[L + lane] = ((unsigned long long)e.x << 32) | e.y; vals[L + lane] = __uint_as_float(e.z); }
        q = __shfl_sync(FULL, e.w, 0);                // the run's first entry carries the link to the next run
        L += len; ++hops;
    }
    if (!fits || q) return false;
    unsigned n2 = 32; while (n2 < L) n2 <<= 1;
    for (unsigned i = L + lane; i < n2; i += 32u) { keys[i] = ~0ull; vals[i] = 0.0f; }
    __syncwarp();
    for (unsigned k = 2; k <= n2; k <<= 1) {
        for (unsigned j = k >> 1; j > 0; j >>= 1) {
            for (unsigned i = lane; i < n2; i += 32u) {
                const unsigned ixj = i ^ j;
                if (ixj > i) {
                    const unsigned long long a = keys[i], b = keys[ixj];
                    const bool up = (i & k) == 0;
                    if ((a > b) == up) { keys[i] = b; keys[ixj] = a; const float t = vals[i]; vals[i] = vals[ixj]; vals[ixj] = t; }
                }
            }
            __syncwarp();
        }
    }
    for (unsigned j = lane; j < L; j += 32u) {
        const unsigned cp = (unsigned)(keys[j] >> 34);
        if (j == 0 || (unsigned)(keys[j - 1] >> 34) != cp) apply_run(p, keys, vals, j, L);
    }
    __syncwarp();
    return true;
}

// Eight chains at a time, one per warp; those too long for a warp are then taken one after the other by the whole block: any length,
// in shared memory up to 1024 entries, in the global scratch beyond.  The last kernel of an update_batch: it clears the call's counters
// and posts the box.
__global__ void __launch_bounds__(BLOCK) k_fix_long(Params p, Handover h) {
    constexpr unsigned WARPS = BLOCK / 32;
    __shared__ unsigned long long s_keys[WARPS * WARP_LONG];
    __shared__ float s_vals[WARPS * WARP_LONG];
    __shared__ unsigned s_left[WARPS], s_bcast[3];
    const unsigned n = p.ctl->long_count;
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    unsigned done = 0;
    for (unsigned c0 = blockIdx.x * WARPS; c0 < n; c0 += gridDim.x * WARPS) {
        const unsigned c = c0 + warp;
        unsigned left = 0u;
        if (c < n) {
            const unsigned head = p.longq[c];
            if (!process_long_warp(p, head, s_keys + warp * WARP_LONG, s_vals + warp * WARP_LONG)) left = head;
            ++done;
        }
        if (lane == 0u) s_left[warp] = left;
        __syncthreads();
        for (unsigned k = 0; k < WARPS; ++k) if (s_left[k]) process_long(p, s_left[k], s_keys, s_vals, s_bcast);
        __syncthreads();
    }
    if (lane == 0 && done) atomicAdd(&p.ctl->long_chains, (unsigned long long)done);
    if (last_to_finish<false>(p)) {
        p.ctl->active_count = 0u; p.ctl->long_count = 0u; p.ctl->scratch_cursor = 0u;
        box_put_error(p, h);
    }
}

// ------------------------------------------------------------------------------------------------
// Caller-driven step (no learning, sticky done, no auto-reset): Environment::step for all envs.
// actions / rewards / dones are indexed by environment id.
// The record of one environment after `a`, which leads towards cell `to`; cell words of its own cell and of `to`.  Reward and sticky done flag
// in `r` and `dn`.
__device__ __forceinline__ int4 stepped(const World& p, const int4 rec, int a, unsigned to, unsigned cw_own, unsigned cw_to, float& r, unsigned char& dn) {
    const unsigned s = (unsigned)rec.y * (unsigned)p.W + (unsigned)rec.x;
    const bool moved = to != s && !(cw_to & CW_OBST);
    r = (!moved && a >= 0 && a <= 3) ? blocked_step_reward(p, rec.x, rec.y, a) : -0.01f;    // a trap charges its penalty (src/kernels.cu:61-63)
    if ((moved ? cw_to : cw_own) & CW_GOAL) { r = 1.0f; dn = 1; }
    const unsigned s2 = moved ? to : s;
    return make_int4((int)(s2 % (unsigned)p.W), (int)(s2 / (unsigned)p.W), rec.z + 1, rec.w);
}
__global__ void k_step_actions(const __grid_constant__ World p, const int* __restrict__ actions, float* __restrict__ rewards, unsigned char* __restrict__ dones, Handover h) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.N) {
        const int4 rec = p.st[i];
        const unsigned e = (unsigned)rec.w;
        const int a = actions[e];
        float r; unsigned char dn = p.done[e];
        const unsigned to = target_cell(p, rec.x, rec.y, a);
        p.st[i] = stepped(p, rec, a, to, cw_load(p.cw, (unsigned)rec.y * (unsigned)p.W + (unsigned)rec.x), cw_load(p.cw, to), r, dn);
        p.reward[e] = r; p.done[e] = dn;
        if (rewards) rewards[e] = r;
        if (dones) dones[e] = dn;
    }
    if (h.box && last_to_finish<true>(p)) box_put_error(p, h);
}
// A context with one environment: the action comes with the launch, everything a caller asks for goes back in the box.  (x, y) is where the
// host last saw the environment: the cell words there are on their way while the record is, and nearly always the right ones.
__global__ void k_step_one(const __grid_constant__ World p, int action, bool reset, int x, int y, Handover h) {
    int4 rec = p.st[0];
    float r = 0.0f; unsigned char dn = 0;
    if (reset) {
        const unsigned c = sample_start(p, p.env_offset + (unsigned)rec.w, p.step, TAG_START);
        rec = make_int4((int)(c % (unsigned)p.W), (int)(c / (unsigned)p.W), 0, rec.w);
    } else {
        unsigned to = target_cell(p, x, y, action), own = cw_load(p.cw, (unsigned)y * (unsigned)p.W + (unsigned)x), there = cw_load(p.cw, to);
        dn = p.done[0];
        if (rec.x != x || rec.y != y) {
            to = target_cell(p, rec.x, rec.y, action);
            own = cw_load(p.cw, (unsigned)rec.y * (unsigned)p.W + (unsigned)rec.x); there = cw_load(p.cw, to);
        }
        rec = stepped(p, rec, action, to, own, there, r, dn);
    }
    p.st[0] = rec; p.reward[0] = r; p.done[0] = dn;
    box_put(h, 1u, (unsigned)rec.x); box_put(h, 2u, (unsigned)rec.y); box_put(h, 3u, __float_as_uint(r)); box_put(h, 4u, dn);
    box_put_error(p, h);
}

// The three words of a transition, all on their way at once: left to the compiler, the second waits behind the branch on the first, and a
// look-up across the link takes 2 us.
__device__ __forceinline__ void load_transition(const Transitions& tr, unsigned i, unsigned& at, unsigned& next, float& r) {
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(at) : "l"(tr.at + i));
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(next) : "l"(tr.next + i));
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(tr.r + i));
}
// The TD target of a transition, from the table as it is before the call.
__device__ __forceinline__ float transition_target(const World& p, unsigned at, unsigned next, float r) {
    float m = 0.0f;
    if (!(at >> 31)) {
        m = max4(__ldcg(p.Q + next));
        if (p.legacy_clamp && m < 0.0f) m = 0.0f;
    }
    return __fmaf_rn(p.gamma, m, r);
}

// update_batch, phase 1: the TD target of every transition; every transition becomes a collision entry (index order = fold order).
__global__ void k_update_main(Params p, unsigned n, Transitions tr) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned lane = threadIdx.x & 31u;
    bool first = false; unsigned slot = 0;
    if (i < n) {
        unsigned at, next; float r;
        load_transition(tr, i, at, next, r);
        const float d = transition_target(p, at, next, r);
        const unsigned cell = (at & 0x7FFFFFFFu) >> 2;
        slot = mb_slot(p, cell);
        const unsigned prev = atomicExch(p.mailbox + slot, i + 1u);              // a run of one entry
        p.ent[i] = make_uint4((cell << 3) | (at & 3u), i, __float_as_uint(d), prev);
        first = prev == 0u;
    }
    const unsigned fm = __ballot_sync(FULL, first);                  // list the slots that just became active
    if (fm) {
        unsigned base = 0;
        if (lane == __ffs(fm) - 1u) base = atomicAdd(&p.ctl->active_count, __popc(fm));
        base = __shfl_sync(FULL, base, __ffs(fm) - 1);
        if (first) p.active[base + __popc(fm & ((1u << lane) - 1u))] = slot;
    }
}

// update_batch of up to 1,024 transitions in one block: targets, a bitonic sort by (cell, action, index) -- strides below a warp by
// shuffle -- and the first of every run folds it.  One launch instead of three and nothing but latency: the inputs across the link, one
// look-up of the next rows, the sort, one read and write of the entries.  KEY: 32 bits hold cell, action and index of grids of up to
// 2^20 cells and halve the sort's shuffles.
template <class KEY>
__global__ void __launch_bounds__(UPDATE_SMALL) k_update_small(const __grid_constant__ World p, unsigned n, const __grid_constant__ Transitions tr, Handover h) {
    __shared__ KEY s_key[UPDATE_SMALL];
    __shared__ float s_target[UPDATE_SMALL];
    constexpr unsigned IDX = 10u, IDX_MASK = (1u << IDX) - 1u;
    static_assert(UPDATE_SMALL == 1u << IDX, "index bits of the key");
    const unsigned i = threadIdx.x;
    KEY key = ~(KEY)0;
    if (i < n) {
        unsigned at, next; float r;
        load_transition(tr, i, at, next, r);
        s_target[i] = transition_target(p, at, next, r);
        key = ((KEY)(at & 0x7FFFFFFFu) << IDX) | i;
    }
    for (unsigned k = 2u; k <= blockDim.x; k <<= 1)
        for (unsigned j = k >> 1; j; j >>= 1) {
            KEY other;
            if (j >= 32u) {
                __syncthreads();
                s_key[i] = key;
                __syncthreads();
                other = s_key[i ^ j];
            } else other = __shfl_xor_sync(FULL, key, j);
            const bool low = ((i & k) == 0u) == ((i & j) == 0u);     // this place keeps the smaller of the two
            key = (other < key) == low ? other : key;
        }
    __syncthreads();
    s_key[i] = key;
    __syncthreads();
    const KEY at = key >> IDX;
    if (key != ~(KEY)0 && (i == 0u || s_key[i - 1u] >> IDX != at)) {
        float* const q = reinterpret_cast<float*>(p.Q) + at;
        float v = *q;
        for (unsigned j = i; j < blockDim.x; ++j) {
            const KEY e = s_key[j];
            if (e >> IDX != at) break;
            v = __fmaf_rn(p.lr, __fsub_rn(s_target[(unsigned)e & IDX_MASK], v), v);      // each sees the value the one before it left
        }
        *q = v;
    }
    if (i == 0u) box_put_error(p, h);
}

// ------------------------------------------------------------------------------------------------
__global__ void k_q_init(const __grid_constant__ World p, int kind, float scale) {
    unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= p.S) return;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kind == 1) {
        U4 w = philox4x32_10(s, 0u, 0u, 0u, p.k0, p.k1 ^ TAG_QINIT);
        v.x = __fmul_rn(u01(w.x), scale); v.y = __fmul_rn(u01(w.y), scale);
        v.z = __fmul_rn(u01(w.z), scale); v.w = __fmul_rn(u01(w.w), scale);
    }
    p.Q[s] = v;
}
__global__ void k_cell_set(const __grid_constant__ World p, unsigned cell, unsigned cls, int clear_goals) {
    unsigned* w32 = reinterpret_cast<unsigned*>(p.cw);
    if (clear_goals) {
        unsigned n2 = (p.S + 1u) / 2u;
        for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += gridDim.x * blockDim.x)
            atomicAnd(w32 + i, ~0x00020002u);
    } else if (blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned sh = (cell & 1u) * 16u;
        atomicAnd(w32 + (cell >> 1), ~(7u << sh));
        if (cls) atomicOr(w32 + (cell >> 1), cls << sh);
    }
}

// ------------------------------------------------------------------------------------------------
static inline unsigned nblk(unsigned n) { return (n + BLOCK - 1) / BLOCK; }
static inline unsigned fix_blocks(const Params& p) { unsigned b = p.mb_slots / BLOCK; return b > 1184u ? 1184u : b; }
static inline unsigned sweep_blocks(unsigned S) { unsigned b = nblk((2u * S + 15u) / 16u); return b < 1u ? 1u : (b > 1184u ? 1184u : b); }

void launch_identity_ids(const Params& p, cudaStream_t st) { if (p.N) k_ids_identity<<<nblk(p.N), BLOCK, 0, st>>>(p); }
void launch_export_state(const Params& p, int* out, Handover h, cudaStream_t st) { k_export_state<<<p.N ? nblk(p.N) : 1u, BLOCK, 0, st>>>(p, out, h); }
void launch_copy_out(const Params& p, const CopySpan* spans, int n, Handover h, cudaStream_t st) {
    const CopySpan none{nullptr, nullptr, 0u}, a = n > 0 ? spans[0] : none, b = n > 1 ? spans[1] : none;
    const unsigned blocks = nblk(((a.bytes > b.bytes ? a.bytes : b.bytes) + 15u) / 16u);
    k_copy_out<<<blocks < 1u ? 1u : (blocks > 64u ? 64u : blocks), BLOCK, 0, st>>>(p, a, b, h);
}
void launch_post(const Params& p, Handover h, cudaStream_t st) { k_post<<<1, 32, 0, st>>>(p, h); }
void launch_import_state(const Params& p, const int* x, const int* y, const int* t, cudaStream_t st) { if (p.N) k_import_state<<<nblk(p.N), BLOCK, 0, st>>>(p, x, y, t); }
void launch_reset_all(const Params& p, cudaStream_t st) {
    if (p.N) k_reset_all<<<nblk(p.N), BLOCK, 0, st>>>(p);
}
void launch_step_actions(const Params& p, const int* a, float* r, unsigned char* d, Handover h, cudaStream_t st) {
    if (p.N) k_step_actions<<<nblk(p.N), BLOCK, 0, st>>>(p, a, r, d, h);
}
void launch_step_one(const Params& p, int action, bool reset, int x, int y, Handover h, cudaStream_t st) { k_step_one<<<1, 1, 0, st>>>(p, action, reset, x, y, h); }
void launch_update_batch(const Params& p, unsigned n, const Transitions& tr, Handover h, cudaStream_t st) {
    if (n <= UPDATE_SMALL) {
        unsigned threads = 32u; while (threads < n) threads <<= 1;
        // strictly below 2^20 cells: no key of 32 bits is the padding's all-ones word
        if (p.S < (1u << 20)) k_update_small<unsigned><<<1, threads, 0, st>>>(p, n, tr, h);
        else k_update_small<unsigned long long><<<1, threads, 0, st>>>(p, n, tr, h);
        return;
    }
    k_update_main<<<nblk(n), BLOCK, 0, st>>>(p, n, tr);
    k_fix<<<fix_blocks(p), BLOCK, 0, st>>>(p);
    k_fix_long<<<296, BLOCK, 0, st>>>(p, h);
}
void launch_q_init(const Params& p, int kind, float scale, cudaStream_t st) { k_q_init<<<nblk(p.S), BLOCK, 0, st>>>(p, kind, scale); }
void launch_cell_set(const Params& p, unsigned cell, unsigned cls, int clear_goals, cudaStream_t st) {
    k_cell_set<<<clear_goals ? sweep_blocks(p.S) : 1, BLOCK, 0, st>>>(p, cell, cls, clear_goals);
}

}  // namespace cudarl
