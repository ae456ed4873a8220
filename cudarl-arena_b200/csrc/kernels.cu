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
#include "grid_barrier.cuh"
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
// x | y | t in environment order (rows of `stride` >= N words, a multiple of 4), into the spare copy or straight into the mapped stage: four
// environments per thread, whole 16-byte words out.
__global__ void k_export_state(const __grid_constant__ World p, int* __restrict__ out, unsigned stride, Handover h) {
    const unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) * 4u;
    if (i < p.N) {
        const int4 r0 = p.st[i], r1 = p.st[min(i + 1u, p.N - 1u)], r2 = p.st[min(i + 2u, p.N - 1u)], r3 = p.st[min(i + 3u, p.N - 1u)];
        *reinterpret_cast<int4*>(out + i) = make_int4(r0.x, r1.x, r2.x, r3.x);
        *reinterpret_cast<int4*>(out + stride + i) = make_int4(r0.y, r1.y, r2.y, r3.y);
        *reinterpret_cast<int4*>(out + 2u * stride + i) = make_int4(r0.z, r1.z, r2.z, r3.z);
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

// Fold a sorted run (same cell) starting at index j of keys/vals; returns nothing, writes Q_{t+1}.
__device__ void apply_run(const Params& p, const unsigned long long* keys, const float* vals, unsigned j, unsigned n) {
    const unsigned cell = (unsigned)(keys[j] >> 34);
    float4 row = __ldcg(p.Q + cell);
    for (; j < n; ++j) {
        unsigned wj = (unsigned)(keys[j] >> 32);
        if ((wj >> 2) != cell) break;
        fold(row, (int)(wj & 3u), p.lr, vals[j]);
    }
    p.Q[cell] = row;          // in place: the targets were taken before this kernel started, and one thread owns the cell
}

constexpr unsigned STAGE_ENTRIES = 1024;   // chain entries a block stages in shared memory
constexpr unsigned LONG_MARK = 0xFFFFFFFFu;   // in a mailbox slot: its chain is long
constexpr int SHORT_MAX = 8;           // chain entries folded in registers by one thread

constexpr unsigned MED_MAX = 32;                         // chain entries ranked by one warp with shuffles
constexpr unsigned MED_CHUNKS = STAGE_ENTRIES / MED_MAX;     // medium chains a block can stage in shared memory

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
// first to hook a chain into, so this kernel only visits slots that have work).  The owning thread gathers
// the chain's entries:
//   <= 8 entries   in registers, ordered by a sorting network and folded by that thread;
//   <= 32 entries  staged in shared memory by that thread, ordered and folded by one warp;
//   longer         marked, and left to k_fix_long.
__global__ void __launch_bounds__(BLOCK) k_fix(Params p) {
    __shared__ unsigned long long s_keys[STAGE_ENTRIES];
    __shared__ float s_vals[STAGE_ENTRIES];
    __shared__ unsigned s_medlen[MED_CHUNKS];
    __shared__ unsigned s_nmed;
    const unsigned nactive = p.ctl->active_count;      // slots that received a chain in this call
    // few slots are spread over all blocks, a warp's worth each: a block stages no more than 32 chains of medium length
    const unsigned per = min((unsigned)BLOCK, ((nactive + gridDim.x - 1u) / gridDim.x + 31u) & ~31u);
  for (unsigned tile = blockIdx.x; tile * per < nactive; tile += gridDim.x) {
    if (threadIdx.x == 0) s_nmed = 0;
    __syncthreads();
    const unsigned ai = threadIdx.x < per ? tile * per + threadIdx.x : nactive;
    const unsigned slot = ai < nactive ? p.active[ai] : 0u;
    const unsigned head = ai < nactive ? p.mailbox[slot] : 0u;
    if (head) {
        p.mailbox[slot] = 0u;                          // leave the mailbox empty for the next call
        unsigned long long k8[SHORT_MAX]; float v8[SHORT_MAX];
        unsigned q = head;                             // index of the next entry + 1
#pragma unroll
        for (int j = 0; j < SHORT_MAX; ++j) {
            if (q) {
                const uint4 e = __ldcg(p.ent + (q - 1u));
                k8[j] = ((unsigned long long)e.x << 32) | e.y; v8[j] = __uint_as_float(e.z);
                q = e.w;
            } else { k8[j] = ~0ull; v8[j] = 0.0f; }
        }
        if (q == 0u) {
            cswap(k8[0],v8[0],k8[1],v8[1]); cswap(k8[2],v8[2],k8[3],v8[3]); cswap(k8[4],v8[4],k8[5],v8[5]); cswap(k8[6],v8[6],k8[7],v8[7]);
            cswap(k8[0],v8[0],k8[2],v8[2]); cswap(k8[1],v8[1],k8[3],v8[3]); cswap(k8[4],v8[4],k8[6],v8[6]); cswap(k8[5],v8[5],k8[7],v8[7]);
            cswap(k8[1],v8[1],k8[2],v8[2]); cswap(k8[5],v8[5],k8[6],v8[6]); cswap(k8[0],v8[0],k8[4],v8[4]); cswap(k8[3],v8[3],k8[7],v8[7]);
            cswap(k8[1],v8[1],k8[5],v8[5]); cswap(k8[2],v8[2],k8[6],v8[6]);
            cswap(k8[1],v8[1],k8[4],v8[4]); cswap(k8[3],v8[3],k8[6],v8[6]);
            cswap(k8[2],v8[2],k8[4],v8[4]); cswap(k8[3],v8[3],k8[5],v8[5]);
            cswap(k8[3],v8[3],k8[4],v8[4]);
            unsigned cur = 0xFFFFFFFFu; float4 row = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < SHORT_MAX; ++j) {
                if (k8[j] != ~0ull) {
                    const unsigned w0 = (unsigned)(k8[j] >> 32), cell = w0 >> 2;
                    if (cell != cur) {
                        if (cur != 0xFFFFFFFFu) p.Q[cur] = row;
                        cur = cell; row = __ldcg(p.Q + cell);
                    }
                    fold(row, (int)(w0 & 3u), p.lr, v8[j]);
                }
            }
            if (cur != 0xFFFFFFFFu) p.Q[cur] = row;
        } else {
            const unsigned chunk = atomicAdd(&s_nmed, 1u);
            bool staged = false;
            if (chunk < MED_CHUNKS) {
                unsigned long long* mk = s_keys + chunk * MED_MAX; float* mv = s_vals + chunk * MED_MAX;
#pragma unroll
                for (int j = 0; j < SHORT_MAX; ++j) { mk[j] = k8[j]; mv[j] = v8[j]; }
                unsigned L = SHORT_MAX;
                for (; q && L < MED_MAX; ++L) {
                    const uint4 e = __ldcg(p.ent + (q - 1u));
                    mk[L] = ((unsigned long long)e.x << 32) | e.y; mv[L] = __uint_as_float(e.z);
                    q = e.w;
                }
                staged = q == 0u;
                s_medlen[chunk] = staged ? L : 0u;
            }
            if (!staged) {                              // leave the chain's cells to k_fix_long
                const unsigned li = atomicAdd(&p.ctl->long_count, 1u);
                p.longq[li] = slot;
                p.mailbox[slot] = LONG_MARK;
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

// Entries of long chains (more than 32: cells crowded with transitions).  Following such a chain is one look-up after the other -- 10,000
// transitions of a cell took 5 ms -- so it is not followed: the entries of marked slots are picked out of the entry array in order, sorted
// by cell and action with a stable radix sort, which keeps the order of the transitions, and every (cell, action) is folded by one warp.
// One cooperative launch; without long chains it ends at once.  The last kernel of an update_batch: it clears the call's counters and posts
// the box.
// What bounds it: the sort's three barriers per pass of 9 bits and three sweeps over the entries, then the longest (cell, action) at about
// 10 cycles a transition.
constexpr unsigned SORT_THREADS = 512u, SORT_WARPS = SORT_THREADS / 32u, SORT_BITS = 9u, SORT_BINS = 1u << SORT_BITS;
static_assert(SORT_BINS == SORT_THREADS, "one bin per thread");

__device__ void fold_crowded(const Params& p, unsigned n, GridBarrier& bar) {
    __shared__ unsigned s_count[SORT_WARPS][SORT_BINS];
    __shared__ unsigned s_base[SORT_BINS], s_warp[33];
    const SortP& so = p.so;
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, lt = (1u << lane) - 1u, blocks = gridDim.x, b = blockIdx.x;
    auto share = [&](unsigned m, unsigned& first, unsigned& last) { const unsigned per = (m + blocks - 1u) / blocks; first = min(b * per, m); last = min(first + per, m); };
    unsigned first, last, total = 0u;

    // ---- pick out, in order ----
    share(n, first, last);
    auto chosen = [&](unsigned i, uint4& e) -> bool { if (i >= last) return false; e = p.ent[i]; return p.mailbox[mb_slot(p, e.x >> 2)] == LONG_MARK; };
    unsigned mine = 0u; uint4 e;
    for (unsigned i = first + tid; i < last; i += SORT_THREADS) if (chosen(i, e)) ++mine;
    block_scan_excl(mine, s_warp, &total);
    if (tid == 0u) so.part[b] = total;
    if (!bar.pass()) return;
    unsigned before = 0u, all = 0u;
    for (unsigned k = tid; k < blocks; k += SORT_THREADS) { const unsigned v = so.part[k]; all += v; if (k < b) before += v; }
    block_scan_excl(before, s_warp, &before);
    block_scan_excl(all, s_warp, &all);
    for (unsigned i0 = first; i0 < last; i0 += SORT_THREADS) {
        const bool take = chosen(i0 + tid, e);
        const unsigned at = before + block_scan_excl(take ? 1u : 0u, s_warp, &total);
        if (take) so.a[at] = make_uint2(e.x, e.z);
        before += total;
    }
    if (!bar.pass()) return;
    for (unsigned k = b * SORT_THREADS + tid; k < p.ctl->long_count; k += blocks * SORT_THREADS) p.mailbox[p.longq[k]] = 0u;

    // ---- sort, least significant digit first ----
    uint2 *from = so.a, *to = so.b;
    const unsigned key_bits = 32u - (unsigned)__clz((int)(p.S * 4u - 1u)), passes = (key_bits + SORT_BITS - 1u) / SORT_BITS, bits = (key_bits + passes - 1u) / passes;
    share(all, first, last);
    for (unsigned pass = 0; pass < passes; ++pass) {
        const unsigned shift = pass * bits, mask = (1u << bits) - 1u;
        s_base[tid] = 0u;
        __syncthreads();
        for (unsigned i = first + tid; i < last; i += SORT_THREADS) atomicAdd(&s_base[(from[i].x >> shift) & mask], 1u);
        __syncthreads();
        so.hist[tid * blocks + b] = s_base[tid];
        if (!bar.pass()) return;
        for (unsigned d = b * SORT_WARPS + warp; d < SORT_BINS; d += blocks * SORT_WARPS) {       // a warp per digit: where each block's part of it starts
            unsigned run = 0u;
            for (unsigned k0 = 0; k0 < blocks; k0 += 32u) {
                const unsigned k = k0 + lane, v = k < blocks ? so.hist[d * blocks + k] : 0u;
                unsigned inc = v;
                for (int o = 1; o < 32; o <<= 1) { const unsigned u = __shfl_up_sync(FULL, inc, o); if (lane >= (unsigned)o) inc += u; }
                if (k < blocks) so.hist[d * blocks + k] = run + inc - v;
                run += __shfl_sync(FULL, inc, 31);
            }
            if (lane == 0u) so.total[d] = run;
        }
        if (!bar.pass()) return;
        const unsigned start = block_scan_excl(so.total[tid], s_warp, &total) + so.hist[tid * blocks + b];
        s_base[tid] = start;
        for (unsigned i0 = first; i0 < last; i0 += SORT_THREADS) {
            for (unsigned w = 0; w < SORT_WARPS; ++w) s_count[w][tid] = 0u;
            __syncthreads();
            const unsigned i = i0 + tid;
            const bool act = i < last;
            const uint2 v = act ? from[i] : make_uint2(0u, 0u);
            const unsigned d = act ? (v.x >> shift) & mask : SORT_BINS;
            const unsigned mates = __match_any_sync(FULL, d), rank = __popc(mates & lt);
            if (act && rank == 0u) s_count[warp][d] = __popc(mates);
            __syncthreads();
            unsigned run = s_base[tid];
            for (unsigned w = 0; w < SORT_WARPS; ++w) { const unsigned c = s_count[w][tid]; s_count[w][tid] = run; run += c; }
            s_base[tid] = run;
            __syncthreads();
            if (act) to[s_count[warp][d] + rank] = v;
            __syncthreads();
        }
        uint2* const t = from; from = to; to = t;
        if (!bar.pass()) return;
    }

    // ---- fold: the warp whose window a (cell, action) starts in takes all of it ----
    unsigned crowded = 0u;
    for (unsigned i0 = (b * SORT_WARPS + warp) * 32u; i0 < all; i0 += blocks * SORT_WARPS * 32u) {
        const unsigned i = i0 + lane, key = i < all ? from[i].x : 0xFFFFFFFFu, prev = i && i < all ? from[i - 1u].x : 0xFFFFFFFFu;
        if (i < all && (key >> 2) != (prev >> 2) && i + 32u < all && (from[i + 32u].x >> 2) == (key >> 2)) ++crowded;      // a cell with more than 32 transitions
        unsigned starts = __ballot_sync(FULL, i < all && key != prev);
        while (starts) {
            const unsigned l = (unsigned)__ffs((int)starts) - 1u, k = __shfl_sync(FULL, key, l);
            starts &= starts - 1u;
            float q = reinterpret_cast<const float*>(p.Q)[k];
            unsigned j = i0 + l + lane;
            uint2 cur = j < all ? from[j] : make_uint2(0xFFFFFFFFu, 0u);
            for (;;) {
                const unsigned m = __ballot_sync(FULL, cur.x == k), cnt = m == FULL ? 32u : (unsigned)__ffs((int)~m) - 1u;
                const float target = __uint_as_float(cur.y);
                j += 32u;
                cur = cnt == 32u && j < all ? from[j] : make_uint2(0xFFFFFFFFu, 0u);          // on its way while these are folded
                for (unsigned u = 0; u < cnt; ++u) q = __fmaf_rn(p.lr, __fsub_rn(__shfl_sync(FULL, target, u), q), q);      // each sees the value the one before it left
                if (cnt < 32u) break;
            }
            if (lane == 0u) reinterpret_cast<float*>(p.Q)[k] = q;
        }
    }
    crowded = __reduce_add_sync(FULL, crowded);
    if (lane == 0u && crowded) atomicAdd(&p.ctl->long_chains, (unsigned long long)crowded);
}
__global__ void __launch_bounds__(SORT_THREADS) k_fix_long(const __grid_constant__ Params p, unsigned n, Handover h) {
    __shared__ unsigned s_flag;
    GridBarrier bar{p.so.barrier, p.ctl, 0u, &s_flag};
    if (p.ctl->long_count && !(*reinterpret_cast<volatile unsigned*>(&p.ctl->error) & ERR_COPY_TIMEOUT)) fold_crowded(p, n, bar);
    if (last_to_finish<false>(p)) {
        p.ctl->active_count = 0u; p.ctl->long_count = 0u; *p.so.barrier = 0u;
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
__device__ __forceinline__ void step_record(const World& p, unsigned i, int a, float& r, unsigned char& dn) {
    const int4 rec = p.st[i];                               // record i is environment i
    dn = p.done[i];
    const unsigned to = target_cell(p, rec.x, rec.y, a);
    p.st[i] = stepped(p, rec, a, to, cw_load(p.cw, (unsigned)rec.y * (unsigned)p.W + (unsigned)rec.x), cw_load(p.cw, to), r, dn);
}
// VEC: four environments per thread, so that what crosses the link does so in 16-byte words a thread; else any alignment.
template <bool VEC>
__global__ void k_step_actions(const __grid_constant__ World p, const int* __restrict__ actions, float* __restrict__ rewards, unsigned char* __restrict__ dones, Handover h) {
    const unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) * (VEC ? 4u : 1u);
    if (VEC && i + 4u <= p.N) {
        const int4 a = *reinterpret_cast<const int4*>(actions + i);
        float4 r; uchar4 d = *reinterpret_cast<const uchar4*>(p.done + i);
        const int acts[4] = {a.x, a.y, a.z, a.w};
        int4 rec[4]; unsigned to[4], own[4], there[4]; float rr[4]; unsigned char dd[4] = {d.x, d.y, d.z, d.w};
        // all loads of one kind before the first store: the four environments' look-ups are on their way together
#pragma unroll
        for (unsigned k = 0; k < 4u; ++k) rec[k] = p.st[i + k];
#pragma unroll
        for (unsigned k = 0; k < 4u; ++k) { to[k] = target_cell(p, rec[k].x, rec[k].y, acts[k]); own[k] = cw_load(p.cw, (unsigned)rec[k].y * (unsigned)p.W + (unsigned)rec[k].x); there[k] = cw_load(p.cw, to[k]); }
#pragma unroll
        for (unsigned k = 0; k < 4u; ++k) p.st[i + k] = stepped(p, rec[k], acts[k], to[k], own[k], there[k], rr[k], dd[k]);
        r = make_float4(rr[0], rr[1], rr[2], rr[3]); d = make_uchar4(dd[0], dd[1], dd[2], dd[3]);
        *reinterpret_cast<float4*>(p.reward + i) = r; *reinterpret_cast<uchar4*>(p.done + i) = d;
        if (rewards) *reinterpret_cast<float4*>(rewards + i) = r;
        if (dones) *reinterpret_cast<uchar4*>(dones + i) = d;
    } else for (unsigned e = i; e < p.N && e < i + (VEC ? 4u : 1u); ++e) {
        float r; unsigned char dn;
        step_record(p, e, actions[e], r, dn);
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
        const unsigned own = at & 0x7FFFFFFFu;                                   // cell * 4 + action
        slot = mb_slot(p, own >> 2);
        const unsigned prev = atomicExch(p.mailbox + slot, i + 1u);
        p.ent[i] = make_uint4(own, i, __float_as_uint(d), prev);
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

// update_batch of up to 1,024 transitions in one block, one launch, nothing but latency: the inputs across the link, one look-up of the next
// rows, one read and write of the entries.  Transitions of one (cell, action) find each other in a hash table in shared memory; the first
// there folds their list, by index, when no list is longer than 8 -- else the block sorts them all (bitonic by (cell, action, index), strides
// below a warp by shuffle) and the first of every run folds it.  KEY: 32 bits hold cell, action and index of grids of up to 2^20 cells and
// halve the sort's shuffles.
constexpr unsigned UPDATE_SLOTS = 2u * UPDATE_SMALL, UPDATE_LIST = 8u;
template <class KEY>
__global__ void __launch_bounds__(UPDATE_SMALL) k_update_small(const __grid_constant__ World p, unsigned n, const __grid_constant__ Transitions tr, Handover h) {
    __shared__ KEY s_key[UPDATE_SMALL];
    __shared__ float s_target[UPDATE_SMALL];
    __shared__ unsigned s_slot[UPDATE_SLOTS], s_head[UPDATE_SLOTS], s_next[UPDATE_SMALL];       // (cell, action) + 1; list of its transitions: index + 1, 0 = end
    constexpr unsigned IDX = 10u, IDX_MASK = (1u << IDX) - 1u;
    static_assert(UPDATE_SMALL == 1u << IDX, "index bits of the key");
    const unsigned i = threadIdx.x;
    KEY key = ~(KEY)0;
    unsigned at = 0u, next = 0u; float r = 0.0f;
    if (i < n) load_transition(tr, i, at, next, r);
    for (unsigned k = i; k < UPDATE_SLOTS; k += blockDim.x) { s_slot[k] = 0u; s_head[k] = 0u; }
    __syncthreads();
    bool first = false; unsigned slot = 0u;
    if (i < n) {
        const unsigned own = at & 0x7FFFFFFFu;
        key = ((KEY)own << IDX) | i;
        slot = (own * 0x9E3779B1u) >> (32u - IDX - 1u);
        for (;; slot = (slot + 1u) & (UPDATE_SLOTS - 1u)) {
            const unsigned was = atomicCAS(&s_slot[slot], 0u, own + 1u);
            first = was == 0u;
            if (first || was == own + 1u) break;
        }
        s_next[i] = atomicExch(&s_head[slot], i + 1u);
    }
    float v = 0.0f;
    float* const q = reinterpret_cast<float*>(p.Q) + (at & 0x7FFFFFFFu);
    if (first) v = *q;
    if (i < n) s_target[i] = transition_target(p, at, next, r);
    __syncthreads();
    unsigned list[UPDATE_LIST], len = 0u;
    if (first) {
        unsigned e = s_head[slot];
#pragma unroll
        for (unsigned k = 0; k < UPDATE_LIST; ++k) { list[k] = e ? e : 0xFFFFFFFFu; if (e) { ++len; e = s_next[e - 1u]; } }
        if (e) len = UPDATE_LIST + 1u;
    }
    if (!__syncthreads_or(len > UPDATE_LIST)) {
        if (first) {
            for (unsigned last = 0u; len; --len) {
                unsigned m = list[0] > last ? list[0] : 0xFFFFFFFFu;
#pragma unroll
                for (unsigned k = 1; k < UPDATE_LIST; ++k) if (list[k] > last && list[k] < m) m = list[k];
                v = __fmaf_rn(p.lr, __fsub_rn(s_target[m - 1u], v), v);          // each sees the value the one before it left
                last = m;
            }
            *q = v;
        }
        if (i == 0u) box_put_error(p, h);
        return;
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
    const KEY own = key >> IDX;
    if (key != ~(KEY)0 && (i == 0u || s_key[i - 1u] >> IDX != own)) {
        float* const entry = reinterpret_cast<float*>(p.Q) + own;
        float u = *entry;
        for (unsigned j = i; j < blockDim.x; ++j) {
            const KEY e = s_key[j];
            if (e >> IDX != own) break;
            u = __fmaf_rn(p.lr, __fsub_rn(s_target[(unsigned)e & IDX_MASK], u), u);
        }
        *entry = u;
    }
    // a cell with more than 32 transitions
    const KEY cell = key >> (IDX + 2u);
    if (key != ~(KEY)0 && (i == 0u || s_key[i - 1u] >> (IDX + 2u) != cell) && i + 32u < blockDim.x && s_key[i + 32u] != ~(KEY)0 && s_key[i + 32u] >> (IDX + 2u) == cell)
        atomicAdd(&p.ctl->long_chains, 1ull);
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
static inline unsigned fix_blocks(const Params& p) { const unsigned b = p.mb_slots / 32u; return b > 1184u ? 1184u : b; }
static inline unsigned sweep_blocks(unsigned S) { unsigned b = nblk((2u * S + 15u) / 16u); return b < 1u ? 1u : (b > 1184u ? 1184u : b); }

void launch_identity_ids(const Params& p, cudaStream_t st) { if (p.N) k_ids_identity<<<nblk(p.N), BLOCK, 0, st>>>(p); }
void launch_export_state(const Params& p, int* out, unsigned stride, Handover h, cudaStream_t st) { k_export_state<<<p.N ? nblk((p.N + 3u) / 4u) : 1u, BLOCK, 0, st>>>(p, out, stride, h); }
void launch_copy_out(const Params& p, const CopySpan* spans, int n, Handover h, cudaStream_t st) {
    const CopySpan none{nullptr, nullptr, 0u}, a = n > 0 ? spans[0] : none, b = n > 1 ? spans[1] : none;
    const unsigned blocks = nblk(((a.bytes > b.bytes ? a.bytes : b.bytes) + 15u) / 16u);
    k_copy_out<<<blocks < 1u ? 1u : (blocks > 296u ? 296u : blocks), BLOCK, 0, st>>>(p, a, b, h);
}
void launch_post(const Params& p, Handover h, cudaStream_t st) { k_post<<<1, 32, 0, st>>>(p, h); }
void launch_import_state(const Params& p, const int* x, const int* y, const int* t, cudaStream_t st) { if (p.N) k_import_state<<<nblk(p.N), BLOCK, 0, st>>>(p, x, y, t); }
void launch_reset_all(const Params& p, cudaStream_t st) {
    if (p.N) k_reset_all<<<nblk(p.N), BLOCK, 0, st>>>(p);
}
void launch_step_actions(const Params& p, const int* a, float* r, unsigned char* d, Handover h, cudaStream_t st) {
    if (!p.N) return;
    const bool vec = (((uintptr_t)a | (uintptr_t)r) & 15u) == 0u && ((uintptr_t)d & 3u) == 0u;
    // results that go across the link; within the device one environment per thread is the better spread: 4,194,304 environments 57 us, four per thread 62
    if (vec && h.box) k_step_actions<true><<<nblk((p.N + 3u) / 4u), BLOCK, 0, st>>>(p, a, r, d, h);
    else k_step_actions<false><<<nblk(p.N), BLOCK, 0, st>>>(p, a, r, d, h);
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
    void* args[3] = {const_cast<Params*>(&p), &n, &h};
    const unsigned blocks = (n + 2u * SORT_THREADS - 1u) / (2u * SORT_THREADS);
    cudaLaunchCooperativeKernel((const void*)k_fix_long, dim3(blocks < p.so.blocks ? blocks : p.so.blocks), dim3(SORT_THREADS), args, 0, st);
}
void launch_q_init(const Params& p, int kind, float scale, cudaStream_t st) { k_q_init<<<nblk(p.S), BLOCK, 0, st>>>(p, kind, scale); }
void launch_cell_set(const Params& p, unsigned cell, unsigned cls, int clear_goals, cudaStream_t st) {
    k_cell_set<<<clear_goals ? sweep_blocks(p.S) : 1, BLOCK, 0, st>>>(p, cell, cls, clear_goals);
}

}  // namespace cudarl
