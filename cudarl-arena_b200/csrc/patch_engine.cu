// patch_engine.cu -- the fused train step for worlds of a few thousand environments: cut into patches, one per block of a cluster, many steps per launch.
//
// In the gather engine (gather_engine.cu) the table and the counters of a step lie in L2, and a step is two barriers and four dependent accesses there.
// Here every block of one cluster owns a patch of the grid and the environments that stand on it: their rows, counters, move bytes and records are
// in its shared memory.  What blocks have to tell one another in a step they write into one another's shared memory:
//
//   * the environments that walk out of a patch, or whose next episode starts on another, as 8-byte records;
//   * max_a Q of the cells along the patches' edges, for the TD targets of moves across them.
//
// One barrier of the cluster a step, and no access to L2:
//
//   look      every environment draws, reads its row, chooses, reads the row it moves to; one that goes gets its place in the receiver's list    (while the barrier is under way)
//   commit    every environment counts itself, and is put back or sent
//   apply     the first on a (cell, action) applies its update as often as it was counted; edge values out
//
// Cells are numbered by bands: bands of 8 or more rows (a power of two), in a band column by column, in a column downwards.  A patch is a range of
// that numbering, a place in it is a cell's index in shared memory, and the ranges are cut at the beginning of a launch so that cells and
// environments weigh the same for every block.  (The population bunches up on the paths to the goals.)
//
// What does not fit -- more environments on a patch than its block has slots for, more records in a step than the receiver has room for -- ends
// the launch's patches with that step, for all blocks at the same one: the records go back to environment order, the rows into the table, and
// the rest of the steps runs as in the gather engine, which no crowd can overrun.
//
// What bounds it: the chain of one step, thread by thread some 350 instructions at about 6 cycles each (look, commit, apply, edge values), the longest of them in the
// block next to a goal, where most arrivals and restarts are.  Hence one environment a thread in straight code, a loop only for what is left over (with
// everything in one loop 3.1 us where it is 2.7 now; 1,024 threads, whose 64 registers spill, 5.3 where 768 take 3.4), residents and arrivals in
// different warps, an arrival looked at as soon as it is there, and remote atomics whose answer nobody waits for.  B200, us a step, gather engine's cluster / here: 600
// environments on 32 x 150 cells 3.7 / 1.8, 1,500 on 80 x 80 3.9 / 2.1, 4,096 on 64 x 64 with an untrained table 4.0 / 2.4, after 6,000 steps 4.0 / 2.7,
// 8,192 on 100 x 100 4.5 / 3.4 and on 250 x 250 4.9 / 3.0, 12,000 on 200 x 200 5.7 / 4.1.
//
// (The same with a patch on every multiprocessor, records and edge values as words in L2 that carry the number of their step: 65,536 on 256 x 256 5.7, the gather
// engine 6.1; 150,001 on 1001 x 613 6.7 / 6.8; 1,048,576 on 1024 x 1024 21 / 22.  Not worth a second engine.)
//
// Reference semantics: those of tile_engine.cu.
#include "global_table.cuh"
#include <algorithm>
#include <cstring>

namespace cudarl {

constexpr unsigned AWAY = 0x80000000u;           // a destination on another patch: block << 16 | cell of that patch
constexpr unsigned NO_CELL = 0xFFFFFFFFu, HOLE = 0xFFFFFFFFu;

// An environment on a patch, 8 bytes: number (26 bits), cell (14), steps of the episode (24).
__device__ __forceinline__ uint2 patch_rec(unsigned id, unsigned loc, unsigned t) { return make_uint2(id | loc << 26, t << 8 | loc >> 6); }
__device__ __forceinline__ unsigned rec_id(uint2 r) { return r.x & 0x3FFFFFFu; }
__device__ __forceinline__ unsigned rec_loc(uint2 r) { return r.x >> 26 | (r.y & 0xFFu) << 6; }
__device__ __forceinline__ unsigned rec_t(uint2 r) { return r.y >> 8; }

// Shared memory of another block of the cluster: the address there of what lies at p here.
__device__ __forceinline__ unsigned at_block(const void* p, unsigned rank) {
    unsigned a; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void put_there(unsigned a, unsigned v) { asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void put_there(unsigned a, uint2 v) { asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" :: "r"(a), "l"((unsigned long long)v.y << 32 | v.x) : "memory"); }      // in one piece
__device__ __forceinline__ unsigned add_there(unsigned a, unsigned v) { unsigned o; asm volatile("atom.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory"); return o; }

// What the patches of a launch are cut from: records sorted by cell number / 8 into pp.dealt, cut[] = the first such bin of each block's patch,
// s_first[] = the first record of it.  A counting sort, as in the gather engine.
template <unsigned THREADS>
__device__ void cut_patches(const Params& p, const StepLaunch& l, const PatchP& pp, ClusterSpace& space, unsigned* s_cut, unsigned* s_first) {
    __shared__ unsigned s_warp[33], s_sum;
    const unsigned tid = threadIdx.x, lane = tid & 31u, G = gridDim.x, b = blockIdx.x;
    const unsigned share = (p.N + G - 1u) / G, first = min(b * share, p.N), last = min(first + share, p.N);
    const unsigned per = (pp.bins + G - 1u) / G, b0 = min(b * per, pp.bins), b1 = min(b0 + per, pp.bins);
    auto bin = [&](const int4 r) -> unsigned {
        return (((((unsigned)r.y >> pp.shift) * (unsigned)p.W + (unsigned)r.x) << pp.shift) | ((unsigned)r.y & ((1u << pp.shift) - 1u))) >> 3;
    };
    for (unsigned i = first + tid; i < last; i += THREADS) pp.rank[i] = atomicAdd(pp.count + bin(l.in[i]), 1u);
    space.arrive(); space.wait();
    unsigned sum = 0u;
    for (unsigned k = b0 + tid; k < b1; k += THREADS) sum += pp.count[k];
    if (tid == 0u) s_sum = 0u;
    __syncthreads();
    sum = __reduce_add_sync(FULL, sum);
    if (lane == 0u && sum) atomicAdd(&s_sum, sum);
    __syncthreads();
    if (tid == 0u) pp.part[b] = s_sum;
    space.arrive(); space.wait();
    unsigned carry = 0u;
    for (unsigned k = 0; k < b; ++k) carry += pp.part[k];
    // patch j starts behind the bin in which the weight of all before it passes j parts of G
    const unsigned long long weight = (unsigned long long)pp.w_env * p.N + (unsigned long long)PT_BIN_WEIGHT * pp.bins;
#pragma unroll 1
    for (unsigned k0 = b0; k0 < b1; k0 += THREADS) {
        const unsigned k = k0 + tid, v = k < b1 ? pp.count[k] : 0u;
        unsigned total = 0u;
        const unsigned ex = carry + block_scan_excl(v, s_warp, &total);
        if (k < b1) {
            pp.count[k] = ex;
            const unsigned long long w0 = (unsigned long long)pp.w_env * ex + (unsigned long long)PT_BIN_WEIGHT * k;
            const unsigned long long w1 = w0 + (unsigned long long)pp.w_env * v + PT_BIN_WEIGHT;
#pragma unroll 1
            for (unsigned j = (unsigned)(w0 * G / weight); j < G; ++j) {
                const unsigned long long at = j * weight / G;
                if (at > w1) break;
                if (at > w0) pp.cut[j] = k + 1u;
            }
        }
        carry += total;
    }
    if (b == 0u && tid == 0u) { pp.cut[0] = 0u; pp.cut[G] = pp.bins; }
    space.arrive(); space.wait();
    for (unsigned i = first + tid; i < last; i += THREADS) { const int4 r = l.in[i]; pp.dealt[pp.count[bin(r)] + pp.rank[i]] = r; }
    for (unsigned j = tid; j <= G; j += THREADS) { const unsigned c = pp.cut[j]; s_cut[j] = c; s_first[j] = c < pp.bins ? pp.count[c] : p.N; }
    space.arrive(); space.wait();
    for (unsigned k = b0 + tid; k < b1; k += THREADS) pp.count[k] = 0u;
}

// What an environment finds out before it is counted.
struct Look {
    unsigned id, t, own, dest, ghost, mv, at;    // own: cell * 4 + action; dest: where it goes, and its place in the list there; ghost: the edge value its move needs, or NO_CELL
    float m;                                     // max_a Q of the cell it moves to, if that is on the patch
};
constexpr unsigned OVER = 0x100u;                // in mv: the episode ends

template <unsigned THREADS, bool PLAIN>
__global__ void __launch_bounds__(THREADS, 1) k_patch_steps(const __grid_constant__ Params p, const __grid_constant__ StepLaunch l, const __grid_constant__ PatchP pp) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned s_cut[PT_BLOCKS + 1u], s_first[PT_BLOCKS + 1u], s_sum[5], s_flag;
    __shared__ unsigned s_mailed[3], s_stop[2], s_news[2][PT_BLOCKS];      // written by the other blocks: records sent here (by step modulo 3), whether a block stops, episodes each has ended (by parity)
    __shared__ unsigned s_taken, s_holes, s_full, s_over, s_edges;   // this step: slots given to arrivals, slots left, a record without room, episodes that ended here; edge values owed
    const bool may = may_start(p, &s_flag);                         // (the same for every block: nothing sets the error word while the cluster runs)
    const unsigned tid = threadIdx.x, b = blockIdx.x, G = gridDim.x, W = (unsigned)p.W;
    const unsigned LB = pp.shift, B = 1u << LB, BM = B - 1u, band = W << LB;
    ClusterSpace space{p};
    if (tid < 5u) s_sum[tid] = 0u;
    if (tid < 3u) s_mailed[tid] = 0u;
    if (tid < 2u) s_stop[tid] = 0u;
    if (tid < 2u * PT_BLOCKS) (&s_news[0][0])[tid] = 0u;
    if (tid == 0u) s_taken = s_holes = s_full = s_over = s_edges = 0u;
    if (!may) return;
    cut_patches<THREADS>(p, l, pp, space, s_cut, s_first);

    // ---- the patch into shared memory ----
    float4* const rows = reinterpret_cast<float4*>(smem);
    uint2* const counts = reinterpret_cast<uint2*>(rows + pp.cells);                 // four 16-bit counters a cell
    uint2* const mail = counts + pp.cells;                                           // three lists of arrivals, by step modulo 3; HOLE: not come yet
    uint2* const rec = mail + 3u * THREADS;                                          // slots
    uint2* const owned = rec + pp.slots;                                             // per slot and then per arrival: the (cell, action) it applies and the target
    unsigned* const from = reinterpret_cast<unsigned*>(owned + pp.slots + THREADS);  // per edge value: block << 16 | cell of that block, or NO_CELL
    float* const ghost = reinterpret_cast<float*>(from + pp.ghosts);                 // the edge values, twice, by parity of the step
    unsigned* const edge = reinterpret_cast<unsigned*>(ghost + 2u * pp.ghosts);      // the edge values owed to others: cell | block << 14 | place there << 18
    unsigned* const closed = edge + pp.ghosts;                                       // a bit per cell of the grid (pp.bits: all or none): no episode starts there
    unsigned short* const holes = reinterpret_cast<unsigned short*>(closed + (pp.bits + 31u) / 32u);         // a ring of free slots
    unsigned char* const moves = reinterpret_cast<unsigned char*>(holes + pp.slots);
    const unsigned k0 = s_cut[b] << 3, cells = (s_cut[b + 1u] << 3) - k0, u0 = k0 >> LB, cols = cells ? ((k0 + cells - 1u) >> LB) - u0 + 1u : 0u;
    const unsigned gdown = 2u * B + cols, nghost = gdown + cols;
    bool fits = true;                                                                // the same for every block
    for (unsigned j = tid; j < G; j += THREADS) {
        const unsigned c = s_cut[j + 1u] - s_cut[j];
        fits = fits && c * 8u <= pp.cells && s_first[j + 1u] - s_first[j] <= pp.limit;
    }
    fits = !__syncthreads_or(!fits);
    unsigned step = 0u;
    if (fits) {
        Tally tally{0u, 0u, 0u, 0u, 0u};
        EpsilonIndex eps_index(p, l, PLAIN);
        float eps = __ldg(p.eps_tab + eps_index.at);
        auto find = [&](unsigned key) -> unsigned {                // the block a cell belongs to
            unsigned lo = 0u, hi = G;
#pragma unroll 1
            while (hi - lo > 1u) { const unsigned mid = (lo + hi) >> 1; if (s_cut[mid] <= key >> 3) lo = mid; else hi = mid; }
            return lo;
        };
        auto place = [&](unsigned key) -> unsigned { const unsigned d = find(key), loc = key - (s_cut[d] << 3); return d == b ? loc : AWAY | d << 16 | loc; };
        auto key_of = [&](unsigned x, unsigned y) -> unsigned { return (((y >> LB) * W + x) << LB) | (y & BM); };
        auto over_w = [&](unsigned n) -> unsigned { const unsigned q = __umulhi(n, pp.w_rcp); return n - q * W >= W ? q + 1u : q; };      // n / W
        auto cell_of = [&](unsigned key, unsigned& x, unsigned& y) { const unsigned u = key >> LB, r = over_w(u); x = u - r * W; y = (r << LB) | (key & BM); };
        // The cell of the patch a move leads to (beyond it: `cells` or more), and the edge value of that cell.
        auto moved = [&](unsigned loc, unsigned a) -> unsigned {
            const unsigned far_side = a == 0u ? 0u : BM;           // up from a band's first row, down from its last
            unsigned d = (a & 1u) ? B : 1u;
            if (!(a & 1u) && ((k0 + loc) & BM) == far_side) d = band - BM;
            return a - 1u < 2u ? loc + d : loc - d;
        };
        auto ghost_of = [&](unsigned loc, unsigned a) -> unsigned {
            const unsigned u = ((k0 + loc) >> LB) - u0;
            return a == 0u ? 2u * B + u : a == 1u ? 2u * B + loc - cells : a == 2u ? gdown + u : loc;
        };
        for (unsigned k = tid; k < nghost; k += THREADS) from[k] = NO_CELL;
        for (unsigned k = tid; k < 3u * THREADS; k += THREADS) mail[k] = make_uint2(0u, HOLE);
#pragma unroll 1
        for (unsigned c0 = tid & ~31u; c0 < pp.bits; c0 += THREADS) {
            const unsigned c = c0 + (tid & 31u), w = __ballot_sync(FULL, c < pp.bits && (cw_load(p.cw, c) & (CW_OBST | CW_GOAL)));
            if ((tid & 31u) == 0u) closed[c0 >> 5] = w;
        }
        __syncthreads();
#pragma unroll 1
        for (unsigned k = tid; k < cells; k += THREADS) {
            unsigned x, y; cell_of(k0 + k, x, y);
            counts[k] = make_uint2(0u, 0u);
            if (y >= (unsigned)p.H) { rows[k] = make_float4(0.f, 0.f, 0.f, 0.f); moves[k] = 0x0Fu; continue; }       // below the last band's last row
            const unsigned s = y * W + x;
            rows[k] = p.Q[s]; moves[k] = __ldg(p.gp.mv + s);
            for (unsigned a = 0; a < 4u; ++a) {
                const bool there = a == 0u ? y > 0u : a == 1u ? x + 1u < W : a == 2u ? y + 1u < (unsigned)p.H : x > 0u;
                const unsigned n = moved(k, a);
                if (!there || n < cells) continue;
                const unsigned g = ghost_of(k, a), f = place(k0 + n) & ~AWAY;
                from[g] = f;                                       // and its block is told that the value is wanted here
                put_there(at_block(edge + add_there(at_block(&s_edges, f >> 16), 1u), f >> 16), (f & 0x3FFFu) | b << 14 | g << 18);
            }
        }
        unsigned hi = s_first[b + 1u] - s_first[b], head = 0u, free_slots = 0u;     // slots in use, the ring of holes among them
        for (unsigned j = tid; j < hi; j += THREADS) {
            const int4 r = pp.dealt[s_first[b] + j];
            rec[j] = patch_rec((unsigned)r.w, key_of((unsigned)r.x, (unsigned)r.y) - k0, (unsigned)r.z);
        }
        space.arrive(); space.wait();
        const unsigned edges = s_edges;
        const unsigned my_edge = tid < edges ? edge[tid] : 0u;     // the first of them: where it goes does not change
        const unsigned my_edge_at = tid < edges ? at_block(ghost + (my_edge >> 18), (my_edge >> 14) & 15u) : 0u;
        auto edges_out = [&](unsigned par) {
            if (tid < edges) put_there(my_edge_at + par * pp.ghosts * 4u, __float_as_uint(max4(rows[my_edge & 0x3FFFu])));
#pragma unroll 1
            for (unsigned k = tid + THREADS; k < edges; k += THREADS) {
                const unsigned e = edge[k];
                put_there(at_block(ghost + par * pp.ghosts + (e >> 18), (e >> 14) & 15u), __float_as_uint(max4(rows[e & 0x3FFFu])));
            }
        };
        edges_out(0u);
        space.arrive();
        const unsigned tmax = p.max_steps > 0 ? (unsigned)p.max_steps : 0x7FFFFFFFu;
        const bool early = PLAIN || l.eps_mode != 2;               // the epsilon of a step is known before the others have arrived
        unsigned long long g = p.step;
        unsigned ended = 0u;                                       // episodes finished in this launch, by all
        const unsigned i = THREADS - 1u - tid;                     // the arrival this thread takes: those that have least to do take the first
        auto leave = [&](unsigned j) { unsigned at = head + free_slots + atomicAdd(&s_holes, 1u); if (at >= pp.slots) at -= pp.slots; if (at >= pp.slots) at -= pp.slots; holes[at] = (unsigned short)j; };
        uint2 arr;                                                 // the arrival, as it came

        unsigned turn = 0u;                                        // the step modulo 3
        for (bool over = false; !over; ++step, ++g, turn = turn == 2u ? 0u : turn + 1u) {
            const unsigned par = step & 1u, next = par ^ 1u;
            uint2* const here = mail + turn * THREADS;             // this step's arrivals
            const unsigned there = turn == 2u ? 0u : turn + 1u;    // the list of the next step's
            const bool last = step == l.steps;
            unsigned thr = !(eps > 0.0f) ? 0u : eps >= 1.0f ? (1u << 24) : (unsigned)ceilf(eps * 16777216.0f);
            unsigned pre[4];
            policy_prefix(p.policy_keys, g, pre);
            uint2 mine = make_uint2(0u, HOLE); unsigned slot = 0u;         // an arrival that stays, and its slot

            auto look = [&](const uint2 r, Look& o) {
                const unsigned id = rec_id(r), loc = rec_loc(r);
                const U4 w = policy_philox(p.env_offset + id, p.policy_keys, pre);
                const float4 row = rows[loc];
                unsigned mv = moves[loc];
                const unsigned a = (w.x >> 8) < thr ? w.y & 3u : (unsigned)argmax4(row);
                mv >>= a;                                 // bit 0: the move is blocked, bit 4: it ends on a goal
                o.id = id; o.own = loc * 4u + a; o.mv = mv; o.t = min(rec_t(r) + 1u, STEP_SAT);
                o.dest = (mv & 1u) ? loc : moved(loc, a);
                o.ghost = NO_CELL; o.m = 0.0f;
                if (o.dest < cells) o.m = max4(rows[o.dest]);
                else { o.ghost = ghost_of(loc, a); o.dest = AWAY | from[o.ghost]; }
                if ((mv & 16u) || o.t >= tmax) {
                    const unsigned s = sample_start_if(p, p.env_offset + id, g + 1ull, TAG_START, [&](unsigned c) { return pp.bits ? closed[c >> 5] >> (c & 31u) & 1u : cw_load(p.cw, c) & (CW_OBST | CW_GOAL); }), y = over_w(s);
                    o.dest = place(key_of(s - y * W, y)); o.t = 0u; o.mv |= OVER;
                }
                if (o.dest & AWAY) o.at = add_there(at_block(s_mailed + there, (o.dest >> 16) & 15u), 1u);      // (the answer is not waited for here)
            };
            // Counts the environment; what it applies, and whether its slot j is free.
            auto commit = [&](const Look& o, bool arrival, unsigned j, bool& left) -> uint2 {
                const unsigned sh = (o.own & 1u) * 16u, old = atomicAdd(reinterpret_cast<unsigned*>(counts) + (o.own >> 1), 1u << sh);
                float m = o.ghost != NO_CELL ? ghost[par * pp.ghosts + o.ghost] : o.m;
                if (!PLAIN && p.legacy_clamp && m < 0.0f) m = 0.0f;
                float rw = -0.01f;
                if (!PLAIN && p.ntraps && (o.mv & 1u)) { unsigned x, y; cell_of(k0 + (o.own >> 2), x, y); rw = blocked_step_reward(p, (int)x, (int)y, (int)(o.own & 3u)); }
                const bool done = (o.mv & 16u) != 0u;
                const float target = done ? 1.0f : __fmaf_rn(p.gamma, m, rw);
                if (!PLAIN && l.trace && step + 1u == l.steps) { p.tr_a[o.id] = (int)(o.own & 3u); p.tr_r[o.id] = done ? 1.0f : rw; p.tr_d[o.id] = done ? 1 : 0; }
                if (o.mv & OVER) {
                    if (done) ++tally.goals; else ++tally.timeouts;
                    if (!PLAIN && l.eps_mode == 2) atomicAdd(&s_over, 1u);
                }
                const uint2 now = patch_rec(o.id, o.dest & 0xFFFFu, o.t);
                left = false;
                if (o.dest & AWAY) {
                    const unsigned d = (o.dest >> 16) & 15u;
                    if (o.at < THREADS) put_there(at_block(mail + there * THREADS + o.at, d), now);
                    else {                                         // no room: everybody stops after this step, and this is where it stands then
                        unsigned x, y; cell_of((s_cut[d] << 3) + rec_loc(now), x, y);
                        p.st[o.id] = make_int4((int)x, (int)y, (int)o.t, (int)o.id);
                        s_full = 1u;
                    }
                    if (!arrival) { rec[j].y = HOLE; left = true; }
                } else if (!arrival) rec[j] = now;
                else {                                             // (its slot may be one that another thread has not yet passed over)
                    const unsigned k = atomicAdd(&s_taken, 1u);
                    if (k < free_slots) { unsigned at = head + k; if (at >= pp.slots) at -= pp.slots; slot = holes[at]; } else slot = hi + (k - free_slots);
                    mine = now;
                }
                return make_uint2(((old >> sh) & 0xFFFFu) == 0u ? o.own : NOBODY, __float_as_uint(target));
            };
            auto apply = [&](const uint2 duty) {
                const uint2 c = counts[duty.x >> 2];
                float* const q = reinterpret_cast<float*>(rows) + duty.x;
                const float v = *q;
                const unsigned a = duty.x & 3u, n = ((a & 2u) ? c.y : c.x) >> ((a & 1u) * 16u) & 0xFFFFu, both = c.x + c.y, tot = (both & 0xFFFFu) + (both >> 16);     // (no field overflows: a patch has fewer than 32,768 environments)
                if (tot > 1u) tally.conf += n;
                if (tot > CROWDED_CELL) {                          // the lowest chosen action speaks for the cell
                    const unsigned c0 = c.x & 0xFFFFu, c1 = c.x >> 16;
                    if ((a == 0u ? 0u : a == 1u ? c0 : a == 2u ? c0 + c1 : c0 + c1 + (c.y & 0xFFFFu)) == 0u) { ++tally.crowded; tally.on_crowded += tot; }
                }
                *q = apply_counted(v, __uint_as_float(duty.y), p.lr, n);
            };

            // ---- this thread's first: the environment of its slot, or an arrival that is here already, as most are ----
            // Looked at while the barrier is under way.  (Should everybody stop before this step, it is still where it was.)
            const bool resident = tid < hi;
            uint2 r = make_uint2(0u, HOLE);
            if (early && !last) {
                if (resident) r = rec[tid];
                else { const unsigned long long v = *reinterpret_cast<volatile unsigned long long*>(here + i); r = make_uint2((unsigned)v, (unsigned)(v >> 32)); }
            }
            Look first;
            const bool act = r.y != HOLE;
            if (act) look(r, first);
            __syncwarp();
            space.wait();
            if (tid == 0u) s_taken = s_holes = 0u;                 // (the last step's were read before the barrier; nobody adds before the next __syncthreads)
            const unsigned arrived = min(s_mailed[turn], THREADS);
            arr = i < arrived ? here[i] : make_uint2(0u, HOLE);
            over = last || s_stop[par] != 0u;
            if (!PLAIN && l.eps_mode == 2 && step) {
                for (unsigned k = 0; k < G; ++k) ended += s_news[par][k];
                eps_index.next(p, l, PLAIN, ended, true);
                if (!over) { eps = __ldg(p.eps_tab + eps_index.at); thr = !(eps > 0.0f) ? 0u : eps >= 1.0f ? (1u << 24) : (unsigned)ceilf(eps * 16777216.0f); }
            }
            if (over) break;
            __syncthreads();
            uint2 duty = make_uint2(NOBODY, 0u);
            bool left = false;
            if (act) duty = commit(first, !resident, tid, left);
            // ---- the others, if any: more slots than threads, an arrival that came late or to a thread that had a slot's ----
            bool late = i < arrived && !(act && !resident);
            unsigned j = early ? tid + THREADS : tid;
#pragma unroll 1
            while (j < hi || late) {
                const bool arrival = j >= hi;
                r = arrival ? arr : rec[j];
                uint2 more = make_uint2(NOBODY, 0u);
                if (r.y != HOLE) {
                    Look o; bool gone = false;
                    look(r, o);
                    more = commit(o, arrival, j, gone);
                    if (gone) leave(j);
                }
                owned[arrival ? pp.slots + i : j] = more;
                if (arrival) break;
                j += THREADS;
            }
            __syncthreads();

            // ---- apply ----
            const unsigned taken = s_taken, new_hi = hi + (taken > free_slots ? taken - free_slots : 0u);
            if (duty.x != NOBODY) apply(duty);
#pragma unroll 1
            for (j = early ? tid + THREADS : tid; j < hi || late; j += THREADS) {
                const bool arrival = j >= hi;
                const uint2 more = owned[arrival ? pp.slots + i : j];
                if (more.x != NOBODY) apply(more);
                if (arrival) break;
            }
            if (mine.y != HOLE) rec[slot] = mine;
            if (left) leave(tid);
            if (tid < G) {
                if (s_full != 0u || new_hi > pp.limit) put_there(at_block(s_stop + next, tid), 1u);
                if (!PLAIN && l.eps_mode == 2) put_there(at_block(&s_news[next][b], tid), s_over);
            }
            __syncthreads();
            edges_out(next);
            for (unsigned k = tid; k < cells / 2u; k += THREADS) reinterpret_cast<uint4*>(counts)[k] = make_uint4(0u, 0u, 0u, 0u);
            if (tid == 0u) { s_mailed[turn] = 0u; s_over = 0u; }   // (the next to add to this list do so after the barrier)
            if (i < arrived) here[i].y = HOLE;
            const unsigned used = min(taken, free_slots);
            head += used; if (head >= pp.slots) head -= pp.slots;
            free_slots += s_holes - used;
            hi = new_hi;
            __syncwarp();
            space.arrive();
            if (l.eps_mode == 1) { ++eps_index.at; if (step + 1u < l.steps) eps = __ldg(p.eps_tab + eps_index.at); }
        }
        {                                                          // back to environment order
            auto put = [&](const uint2 r) { unsigned x, y; cell_of(k0 + rec_loc(r), x, y); p.st[rec_id(r)] = make_int4((int)x, (int)y, (int)rec_t(r), (int)rec_id(r)); };
#pragma unroll 1
            for (unsigned j = tid; j < hi; j += THREADS) if (rec[j].y != HOLE) put(rec[j]);
            if (arr.y != HOLE) put(arr);
        }
        // the rows back into the table, along its rows
#pragma unroll 1
        for (unsigned k = tid; k < cols << LB; k += THREADS) {
            const unsigned yb = k / cols, u = u0 + (k - yb * cols), loc = ((u << LB) | yb) - k0;
            if (loc >= cells) continue;
            const unsigned r = over_w(u), y = (r << LB) | yb;
            if (y < (unsigned)p.H) p.Q[y * W + (u - r * W)] = rows[loc];
        }
        add_tallies(p, l, tally, s_sum, true, eps);
    }
    space.arrive(); space.wait();                                  // (nobody leaves while others may still write into its shared memory)
    if (step < l.steps) {                                          // the same for every block
        int4* const work = fits ? p.st : pp.dealt;
        run_steps<Home::Registers, THREADS, PLAIN, true>(p, l, space, work, nullptr, step);
        if (!fits) {
            __syncthreads();
            const unsigned first = b * l.chunk, n = first < p.N ? min(l.chunk, p.N - first) : 0u;
            if (tid < n) { const int4 r = work[first + tid]; p.st[r.w] = r; }
        }
    }
}

// ------------------------------------------------------------------------------------------------
constexpr size_t PT_SHARED = 218u * 1024u;       // dynamic shared memory of a block: 227 KB less the static words here and in step_loop.cuh
static size_t patch_shared(const PatchP& pp) {
    return 25 * (size_t)pp.cells + 18 * (size_t)pp.slots + 32 * (size_t)pp.threads + 16 * (size_t)pp.ghosts + (size_t)(pp.bits + 31u) / 32u * 4u + 16;
}
// Whether the patches of a world fit the blocks' shared memory, and how it is shared out.  Not where episodes start on one cell, and everybody passes through one
// patch: 12,000 on 200 x 190 cells 3.9 / 5.2 (us a step, gather engine's cluster / here).  Up to one environment a thread, and on crowded grids threads left for
// the arrivals: 12,000 on 200 x 200 5.7 / 4.1, on 100 x 100 5.2 / 5.3, 10,000 there 5.2 / 4.6; 16,384 on 128 x 128 5.3 / 5.7.
bool patch_plan(const Params& p, PatchP& pp) {
    pp = PatchP{};
    const size_t S = p.S, N = p.N;
    if (N > PT_MOST_ENVS || (N > PT_DENSE_ENVS && S < 2 * N) || p.start_mode != 2) return false;
    const unsigned G = (unsigned)std::min<size_t>(PT_BLOCKS, std::max<size_t>(1, (std::max(S, N) + 63) / 64));
    pp.blocks = G;
    unsigned sh = 3u;
    while (sh < 7u && ((size_t)2 << (2u * sh)) <= S / G) ++sh;       // bands about as high as a patch is wide
    while (sh > 3u && (((size_t)p.H + (1u << sh) - 1u) >> sh << sh) * 8u > (size_t)p.H * 9u) --sh;      // (and no more than an eighth of the last one empty)
    pp.shift = sh;
    pp.w_rcp = p.W > 1 ? (unsigned)((1ull << 32) / (unsigned)p.W) : 0xFFFFFFFFu;
    const size_t keys = ((((size_t)p.H + (1u << sh) - 1u) >> sh) << sh) * (size_t)p.W;
    if (keys > (size_t)G * 16384u) return false;
    pp.bins = (unsigned)keys / 8u;
    const size_t avg_n = (N + G - 1) / G;
    pp.threads = avg_n <= 128u ? 256u : avg_n <= 256u ? 512u : 768u;        // residents and arrivals in different warps
    pp.limit = (unsigned)(avg_n * 2u + 256u);
    pp.slots = pp.limit + pp.threads;
    // an environment weighs as much as w_env / 16 cells: the more the better the blocks' work is balanced, and the larger the patches where nobody is
    for (unsigned w = 128u; w >= 8u; w -= (w + 3u) / 4u) {
        pp.w_env = w;
        pp.cells = (unsigned)((keys + (N * w + 15) / 16 + G - 1) / G + 23u) & ~7u;
        pp.ghosts = 2u * (1u << sh) + 2u * (pp.cells / (1u << sh) + 2u);
        pp.bits = (unsigned)S;                           // (without, a restart takes an access to L2 or two)
        if (patch_shared(pp) > PT_SHARED) pp.bits = 0u;
        pp.shared = (unsigned)patch_shared(pp);
        if (pp.cells <= 16384u && pp.ghosts <= 16384u && pp.shared <= PT_SHARED) return true;
    }
    return false;
}
template <unsigned THREADS, bool PLAIN>
static cudaError_t launch(const Params& p, const StepLaunch& l, const PatchP& pp, cudaStream_t st) {
    auto* const fn = k_patch_steps<THREADS, PLAIN>;
    cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PT_SHARED);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(pp.blocks); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = pp.shared; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = pp.blocks; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, p, l, pp);
}
cudaError_t launch_patch_steps(const Params& p, const StepLaunch& l, const PatchP& pp, cudaStream_t st) {
    const bool pl = plain(p, l);
    if (pp.threads == 256u) return pl ? launch<256u, true>(p, l, pp, st) : launch<256u, false>(p, l, pp, st);
    if (pp.threads == 768u) return pl ? launch<768u, true>(p, l, pp, st) : launch<768u, false>(p, l, pp, st);
    return pl ? launch<512u, true>(p, l, pp, st) : launch<512u, false>(p, l, pp, st);
}

}  // namespace cudarl
