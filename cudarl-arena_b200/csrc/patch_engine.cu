// patch_engine.cu -- the fused train step for worlds that fit the shared memory of several blocks: cut into patches, one per block, many steps per launch.
//
// In the gather engine (gather_engine.cu) the table and the counters of a step lie in L2, and a step is two barriers and four dependent accesses there.
// Here every block owns a patch of the grid and the environments that stand on it: their rows, counters, move bytes and records are in its shared
// memory.  What blocks have to tell one another in a step is little:
//
//   * the environments that walk out of a patch, or whose next episode starts on another, as 8-byte records;
//   * max_a Q of the cells along the patches' edges, for the TD targets of moves across them.
//
//   look      every environment draws, reads its row, chooses, reads the row it moves to; one that goes gets its place in the receiver's list    (while the barrier is under way)
//   commit    every environment counts itself, and is put back or sent
//   apply     the first on a (cell, action) applies its update as often as it was counted; edge values out
//
// Up to 8,192 environments the blocks are one cluster and write into one another's shared memory: one barrier of the cluster a step, and no access to L2.
//
// More of them take a patch on every multiprocessor (GRID).  Records and edge values then travel through L2 as 8-byte words that carry the number of the step
// they are for, and the blocks wait for one another at a counter that orders nothing: when everybody has arrived, what was sent is there or about to be, and
// a word is read again until its number is right.  That takes 0.85 us, a barrier that publishes the others' writes 1.3, behind 448 atomics and stores of a block 2.3.
// (Words alone, one from every block, without the counter: 1.8, and with the edge values 8: many warps that read again and again hold up the words themselves.)
//
// Cells are numbered by bands: bands of 8 or more rows (a power of two), in a band column by column, in a column downwards.  A patch is a range of
// that numbering, a place in it is a cell's index in shared memory, and the ranges are cut at the beginning of a launch so that cells and
// environments weigh the same for every block.  (The population bunches up on the paths to the goals.)
//
// What does not fit -- more environments on a patch than its block has slots for, more records in a step than the receiver has room for -- ends
// the launch's patches with that step, for all blocks at the same one: the records go back to environment order, the rows into the table, and
// the rest of the steps runs as in the gather engine, which no crowd can overrun.  Two launches in a row that end so in their first eighth, and the host hears of it and leaves the next
// steps to the gather engine.  (In their first half: 43,788 environments on 484 x 698 cells, 1,041 steps and results 5.5 -> 7.2 ms, patches being worth that much until then.)
//
// What bounds it: the chain of one step, thread by thread some 350 instructions at about 6 cycles each (look, commit, apply, edge values), the longest of them in the
// block next to a goal, where most arrivals and restarts are (256 x 256 cells, 65,536 environments: 24 cells with 486 environments, 214 arrivals and 204 restarts a
// step, half of all blocks have 35 and none).  Hence one environment a thread in straight code, a loop only for what is left over (4,096 on 64 x 64 with
// everything in one loop 3.1 us, now 2.7; 1,024 threads, whose 64 registers spill, 8,192 on 100 x 100 5.3, 768 take 3.4), residents and arrivals in
// different warps, an arrival looked at as soon as it is there, and atomics whose answer nobody waits for.  B200, us a step, gather engine / here, with trained
// tables: in a cluster 1,500 environments on 80 x 80 cells 3.9 / 2.1, 4,096 on 64 x 64 4.0 / 2.7, 8,192 on 91 x 91 4.3 / 3.4 and on 250 x 250 4.6 / 2.9; on the whole GPU 3,000 on
// 350 x 350 3.8 / 2.6, 10,240 on 202 x 202 5.4 / 3.3, 16,000 on 300 x 300 6.1 / 3.1, 30,000 on 150 x 150 5.9 / 4.3, 100,000 on 300 x 290 7.6 / 7.0, 65,536 on 256 x 256 with eight goals 6.1 / 4.3 after
// 12,000 steps of a falling epsilon and 5.1 after 40,000, but 6.0 / 6.2 with epsilon 0.1 from the beginning, when all paths lead to the goals.
//
// Reference semantics: those of tile_engine.cu.
#include "global_table.cuh"
#include <algorithm>
#include <cstring>
#include <type_traits>

namespace cudarl {

constexpr unsigned AWAY = 0x80000000u;           // a destination on another patch: block << 16 | cell of that patch
constexpr unsigned NO_CELL = 0xFFFFFFFFu, HOLE = 0xFFFFFFFFu;
constexpr unsigned PT_AT_ONCE = 256u;            // GRID: arrivals of a step that are fetched before their number is known

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

// Across the whole GPU: 32 bits under the number of the step they are for.
typedef unsigned long long Word;
__device__ __forceinline__ void send_word(Word* q, unsigned v, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(q), "l"((Word)v << 32 | tag) : "memory");
}
__device__ __forceinline__ Word look_word(const Word* q) { Word v; asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(q) : "memory"); return v; }
// The word when it has come; false after two seconds.
__device__ __noinline__ bool wait_word(const Word* q, unsigned tag, unsigned& v) {
    unsigned long long t0 = 0ull;
    for (unsigned it = 1u;; ++it) {
        const Word w = look_word(q);
        if ((unsigned)w == tag) { v = (unsigned)(w >> 32); return true; }
        if ((it & 1023u) == 0u) {
            unsigned long long now; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0ull) t0 = now;
            else if (now - t0 > GRID_WAIT_NS) return false;
        }
    }
}

// What the patches of a launch are cut from: records sorted by cell number / 8 into pp.dealt, cut[] = the first such bin of each block's patch,
// s_first[] = the first record of it.  A counting sort, as in the gather engine.
template <unsigned THREADS, class Space>
__device__ bool cut_patches(const Params& p, const StepLaunch& l, const PatchP& pp, Space& space, unsigned* s_cut, unsigned* s_first) {
    __shared__ unsigned s_warp[33], s_sum;
    const unsigned tid = threadIdx.x, lane = tid & 31u, G = gridDim.x, b = blockIdx.x;
    const unsigned share = (p.N + G - 1u) / G, first = min(b * share, p.N), last = min(first + share, p.N);
    const unsigned per = (pp.bins + G - 1u) / G, b0 = min(b * per, pp.bins), b1 = min(b0 + per, pp.bins);
    auto bin = [&](const int4 r) -> unsigned {
        return (((((unsigned)r.y >> pp.shift) * (unsigned)p.W + (unsigned)r.x) << pp.shift) | ((unsigned)r.y & ((1u << pp.shift) - 1u))) >> 3;
    };
    for (unsigned i = first + tid; i < last; i += THREADS) pp.rank[i] = atomicAdd(pp.count + bin(l.in[i]), 1u);
    space.arrive(); if (!space.wait()) return false;
    unsigned sum = 0u;
    for (unsigned k = b0 + tid; k < b1; k += THREADS) sum += pp.count[k];
    if (tid == 0u) s_sum = 0u;
    __syncthreads();
    sum = __reduce_add_sync(FULL, sum);
    if (lane == 0u && sum) atomicAdd(&s_sum, sum);
    __syncthreads();
    if (tid == 0u) pp.part[b] = s_sum;
    space.arrive(); if (!space.wait()) return false;
    unsigned carry = 0u;
    for (unsigned k = tid; k < b; k += THREADS) carry += pp.part[k];
    block_scan_excl(carry, s_warp, &carry);
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
    space.arrive(); if (!space.wait()) return false;
    for (unsigned i = first + tid; i < last; i += THREADS) { const int4 r = l.in[i]; pp.dealt[pp.count[bin(r)] + pp.rank[i]] = r; }
    for (unsigned j = tid; j <= G; j += THREADS) { const unsigned c = pp.cut[j]; s_cut[j] = c; s_first[j] = c < pp.bins ? pp.count[c] : p.N; }
    space.arrive(); if (!space.wait()) return false;
    for (unsigned k = b0 + tid; k < b1; k += THREADS) pp.count[k] = 0u;
    return true;
}

// What an environment finds out before it is counted.
struct Look {
    unsigned id, t, own, dest, ghost, mv, at;    // own: cell * 4 + action; dest: where it goes, and its place in the list there; ghost: the edge value its move needs, or NO_CELL
    float m;                                     // max_a Q of the cell it moves to, if that is on the patch
};
constexpr unsigned OVER = 0x100u;                // in mv: the episode ends

// GRID: a patch on every multiprocessor, else in a cluster.
template <unsigned THREADS, bool PLAIN, bool GRID>
__global__ void __launch_bounds__(THREADS, 1) k_patch_steps(const __grid_constant__ Params p, const __grid_constant__ StepLaunch l, const __grid_constant__ PatchP pp) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr unsigned BLOCKS = GRID ? PT_MOST_BLOCKS : PT_BLOCKS;
    __shared__ unsigned s_cut[BLOCKS + 1u], s_first[BLOCKS + 1u], s_sum[5], s_flag, s_in;
    __shared__ Word s_word;                                        // GRID: the counter as everybody has arrived
    __shared__ unsigned s_mailed[3], s_stop[2], s_news[2][PT_BLOCKS];      // written by the other blocks: records sent here (by step modulo 3), whether a block stops, episodes each has ended (by parity)
    __shared__ unsigned s_taken, s_holes, s_full, s_over, s_edges;   // this step: slots given to arrivals, slots left, a record without room, episodes that ended here; edge values owed
    const bool may = may_start(p, &s_flag);                         // (the same for every block: nothing sets the error word while the cluster runs)
    const unsigned tid = threadIdx.x, b = blockIdx.x, G = gridDim.x, W = (unsigned)p.W;
    const unsigned LB = pp.shift, B = 1u << LB, BM = B - 1u, band = W << LB;
    using Space = std::conditional_t<GRID, GridSpace, ClusterSpace>;
    Space space = [&]() -> Space { if constexpr (GRID) return GridSpace(p, pp.barrier, 0u, &s_flag); else return ClusterSpace{p}; }();
    if (tid < 5u) s_sum[tid] = 0u;
    if (tid < 3u) s_mailed[tid] = 0u;
    if (tid < 2u) s_stop[tid] = 0u;
    if (tid < 2u * PT_BLOCKS) (&s_news[0][0])[tid] = 0u;
    if (tid == 0u) s_taken = s_holes = s_full = s_over = s_edges = 0u;
    if (!may) return;
    if (!cut_patches<THREADS>(p, l, pp, space, s_cut, s_first)) return;

    // ---- the patch into shared memory ----
    float4* const rows = reinterpret_cast<float4*>(smem);
    uint2* const counts = reinterpret_cast<uint2*>(rows + pp.cells);                 // four 16-bit counters a cell
    uint2* const mail = counts + pp.cells;                                           // three lists of arrivals, by step modulo 3; HOLE: not come yet
    uint2* const rec = mail + (GRID ? 0u : 3u * THREADS);                                          // slots
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
        unsigned kept = 0u;                                        // GRID: records this thread has written back
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
        if (!GRID) for (unsigned k = tid; k < 3u * THREADS; k += THREADS) mail[k] = make_uint2(0u, HOLE);
        map_closed(p, closed, pp.bits, tid, THREADS);
#pragma unroll 4
        for (unsigned k = tid; k < cells; k += THREADS) {
            unsigned x, y; cell_of(k0 + k, x, y);
            const bool real = y < (unsigned)p.H;                   // not below the last band's last row
            const unsigned s = real ? y * W + x : 0u;
            const float4 row = p.Q[s]; const unsigned char mv = __ldg(p.gp.mv + s);
            rows[k] = row; moves[k] = real ? mv : 0x0Fu;
            counts[k] = make_uint2(0u, 0u);
        }
        __syncthreads();
#pragma unroll 1
        for (unsigned k = tid; k < cells; k += THREADS) {
            unsigned x, y; cell_of(k0 + k, x, y);
            if (y >= (unsigned)p.H) continue;
            bool outside = false;
            for (unsigned a = 0; a < 4u; ++a) {
                const bool there = a == 0u ? y > 0u : a == 1u ? x + 1u < W : a == 2u ? y + 1u < (unsigned)p.H : x > 0u;
                const unsigned n = moved(k, a);
                if (!there || n < cells) continue;
                const unsigned g = ghost_of(k, a), f = place(k0 + n) & ~AWAY;
                from[g] = f;
                outside = true;
                if constexpr (!GRID) put_there(at_block(edge + add_there(at_block(&s_edges, f >> 16), 1u), f >> 16), (f & 0x3FFFu) | b << 14 | g << 18);     // its block is told that the value is wanted here
            }
            if (GRID && outside) edge[atomicAdd(&s_edges, 1u)] = k;
        }
        unsigned hi = s_first[b + 1u] - s_first[b], head = 0u, free_slots = 0u;     // slots in use, the ring of holes among them
        for (unsigned j = tid; j < hi; j += THREADS) {
            const int4 r = pp.dealt[s_first[b] + j];
            rec[j] = patch_rec((unsigned)r.w, key_of((unsigned)r.x, (unsigned)r.y) - k0, (unsigned)r.z);
        }
        if constexpr (GRID) __syncthreads(); else { space.arrive(); space.wait(); }
        const unsigned edges = s_edges;
        unsigned tag = l.epoch;                                    // GRID: the number of the step
        auto ghost_word = [&](unsigned k) -> const Word* { const unsigned f = from[k]; return f == NO_CELL ? nullptr : pp.edge + (s_cut[f >> 16] << 3) + (f & 0xFFFFu); };
        const Word* const my_ghost = GRID && tid < nghost ? ghost_word(tid) : nullptr;
        const unsigned my_edge = tid < edges ? edge[tid] : 0u;     // the first of them: where it goes does not change
        const unsigned my_edge_at = !GRID && tid < edges ? at_block(ghost + (my_edge >> 18), (my_edge >> 14) & 15u) : 0u;
        auto edges_out = [&](unsigned par) {
            if constexpr (GRID) {
                Word* const m = pp.edge + (size_t)par * pp.keys + k0;
#pragma unroll 1
                for (unsigned k = tid; k < edges; k += THREADS) { const unsigned c = edge[k]; send_word(m + c, __float_as_uint(max4(rows[c])), tag); }
                return;
            }
            if (tid < edges) put_there(my_edge_at + par * pp.ghosts * 4u, __float_as_uint(max4(rows[my_edge & 0x3FFFu])));
#pragma unroll 1
            for (unsigned k = tid + THREADS; k < edges; k += THREADS) {
                const unsigned e = edge[k];
                put_there(at_block(ghost + par * pp.ghosts + (e >> 18), (e >> 14) & 15u), __float_as_uint(max4(rows[e & 0x3FFFu])));
            }
        };
        // GRID: the blocks wait for one another at a counter that orders nothing; what was sent is there then or about to be, and is read again until its number is right.
        // The lists' lengths have no number.  That they are complete rests on the atomics: whoever adds has the answer before its block arrives, so the addition is done, in the one
        // place where it and the receiver's exchange can be done.  (A fence before the arrival, which would also say so to the memory model, takes 0.25 - 0.45 us a step, by a warp of
        // its own 0.13 - 1.0; an acquire in the poll empties the first-level cache, 0.4 us where there are traps: 15,598 on 441 x 234 3.45 -> 3.85.)  An addition that came late all
        // the same would be found by the next to use the list, who would wait for a record in vain, or by the sum at the end of the launch: either way the error word is set.
        Word* const counter = reinterpret_cast<Word*>(pp.barrier) + 32u;      // two, by the parity of the step; arrivals, from bit 24 on the episodes that ended, from bit 56 on blocks that stop
        auto arrive = [&](unsigned par, Word news) {
            if constexpr (GRID) { if (tid == THREADS - 1u) asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" :: "l"(counter + 32u * par), "l"(1ull + news) : "memory"); }
            else { __syncwarp(); space.arrive(); }
        };
        edges_out(0u);
        arrive(0u, 0ull);
        const unsigned tmax = p.max_steps > 0 ? (unsigned)p.max_steps : 0x7FFFFFFFu;
        const bool early = PLAIN || l.eps_mode != 2;               // the epsilon of a step is known before the others have arrived
        unsigned long long g = p.step;
        unsigned ended = 0u;                                       // episodes finished in this launch, by all (GRID: in the steps of the other parity)
        const unsigned i = THREADS - 1u - tid;                     // the arrival this thread takes: those that have least to do take the first
        auto leave = [&](unsigned j) { unsigned at = head + free_slots + atomicAdd(&s_holes, 1u); if (at >= pp.slots) at -= pp.slots; if (at >= pp.slots) at -= pp.slots; holes[at] = (unsigned short)j; };
        uint2 arr;                                                 // the arrival, as it came

        unsigned turn = 0u;                                        // the step modulo 3
        for (bool over = false; !over; ++step, ++g, ++tag, turn = turn == 2u ? 0u : turn + 1u) {
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
                if (o.dest & AWAY) {                               // (the answer is not waited for here)
                    if constexpr (GRID) o.at = atomicAdd(pp.listed + there * G + (o.dest >> 16 & 0xFFu), 1u);
                    else o.at = add_there(at_block(s_mailed + there, (o.dest >> 16) & 15u), 1u);
                }
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
                    const unsigned d = (o.dest >> 16) & 0xFFu;
                    if (o.at < THREADS) {
                        if constexpr (GRID) {
                            Word* const q = pp.list + (((size_t)there * G + d) * THREADS + o.at) * 2u;
                            asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" :: "l"(q), "l"((Word)now.x << 32 | (tag + 1u)), "l"((Word)now.y << 32 | (tag + 1u)) : "memory");
                        } else put_there(at_block(mail + there * THREADS + o.at, d), now);
                    } else {                                         // no room: everybody stops after this step, and this is where it stands then
                        unsigned x, y; cell_of((s_cut[d] << 3) + rec_loc(now), x, y);
                        p.st[o.id] = make_int4((int)x, (int)y, (int)o.t, (int)o.id);
                        s_full = 1u; ++kept;
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
            const Word* const post = pp.list + (((size_t)turn * G + b) * THREADS + i) * 2u;       // GRID: this thread's place in the list
            auto delivered = [&](uint2& q) -> bool {
                Word u, v;
                asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(u), "=l"(v) : "l"(post) : "memory");
                if ((unsigned)u != tag || (unsigned)v != tag) return false;
                q = make_uint2((unsigned)(u >> 32), (unsigned)(v >> 32));
                return true;
            };
            if (early && !last) {
                if (resident) r = rec[tid];
                else if constexpr (GRID) { if (i < PT_AT_ONCE && !delivered(r)) r.y = HOLE; }
                else { const unsigned long long v = *reinterpret_cast<volatile unsigned long long*>(here + i); r = make_uint2((unsigned)v, (unsigned)(v >> 32)); }
            }
            Look first;
            const bool act = r.y != HOLE;
            if (act) look(r, first);
            unsigned arrived;
            Word news = 0ull;
            if constexpr (GRID) {
                unsigned listed = 0u;
                bool ok = true, have = false;
                if (my_ghost) {                                    // perhaps it is here already
                    const Word w = look_word(my_ghost + (size_t)par * pp.keys);
                    have = (unsigned)w == tag;
                    if (have) ghost[par * pp.ghosts + tid] = __uint_as_float((unsigned)(w >> 32));
                }
                if (i == 0u) {
                    const unsigned target = (step / 2u + 1u) * G;
                    unsigned long long t0 = 0ull;
                    Word w;
                    for (unsigned it = 1u;; ++it) {
                        w = look_word(counter + 32u * par);
                        if (((unsigned)w & 0xFFFFFFu) >= target) break;
                        if ((it & 1023u) == 0u) {
                            unsigned long long now; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                            if (t0 == 0ull) t0 = now;
                            else if (now - t0 > GRID_WAIT_NS) { atomicOr(&p.ctl->error, ERR_COPY_TIMEOUT); w = ~0ull; break; }
                        }
                    }
                    s_word = w;
                }
                __syncthreads();
                news = s_word;
                if (news == ~0ull) return;
                if (i == PT_AT_ONCE) listed = atomicExch(pp.listed + turn * G + b, 0u);      // (nobody adds to it again before this block's next arrival)
                bool came = act && !resident;                      // this thread's arrival
                if (came) arr = r;
                else if (i < PT_AT_ONCE) came = delivered(arr);
                for (unsigned k = tid; k < nghost; k += THREADS) {
                    const Word* const q = k == tid ? my_ghost : ghost_word(k);
                    unsigned v = 0u;
                    if (!q || (k == tid && have)) continue;
                    const Word w = look_word(q + (size_t)par * pp.keys);
                    if ((unsigned)w == tag) v = (unsigned)(w >> 32); else ok = ok && wait_word(q + (size_t)par * pp.keys, tag, v);
                    ghost[par * pp.ghosts + k] = __uint_as_float(v);
                }
                if (i == PT_AT_ONCE) s_in = listed;
                if (tid == 0u) s_taken = s_holes = 0u;
                __syncthreads();
                arrived = min(s_in, THREADS);
                if (i >= arrived) arr = make_uint2(0u, HOLE);
                else if (!came) { unsigned u = 0u, v = HOLE; ok = ok && wait_word(post, tag, u) && wait_word(post + 1, tag, v); arr = make_uint2(u, v); }
                if (!ok) { atomicOr(&p.ctl->error, ERR_COPY_TIMEOUT); s_full = 1u; }       // (what was to come never came: the launch ends for all)
            } else {
                __syncwarp();
                space.wait();
                if (tid == 0u) s_taken = s_holes = 0u;             // (the last step's were read before the barrier; nobody adds before the next __syncthreads)
                arrived = min(s_mailed[turn], THREADS);
                arr = i < arrived ? here[i] : make_uint2(0u, HOLE);
            }
            over = last || (GRID ? (news >> 56) != 0ull : s_stop[par] != 0u);
            if (!PLAIN && l.eps_mode == 2 && step) {
                unsigned all;
                if constexpr (GRID) { const unsigned sum = (unsigned)(news >> 24); all = sum + ended; ended = sum; }      // the sums of the steps of both parities
                else { for (unsigned k = 0; k < G; ++k) ended += s_news[par][k]; all = ended; }
                eps_index.next(p, l, PLAIN, all, true);
                if (!over) { eps = __ldg(p.eps_tab + eps_index.at); thr = !(eps > 0.0f) ? 0u : eps >= 1.0f ? (1u << 24) : (unsigned)ceilf(eps * 16777216.0f); }
            }
            if (over) break;
            if constexpr (!GRID) __syncthreads();
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
            if (!GRID && tid < G) {
                if (s_full != 0u || new_hi > pp.limit) put_there(at_block(s_stop + next, tid), 1u);
                if (!PLAIN && l.eps_mode == 2) put_there(at_block(&s_news[next][b], tid), s_over);
            }
            __syncthreads();
            ++tag;
            edges_out(next);
            --tag;
            if constexpr (GRID) arrive(next, ((Word)s_over << 24) + (s_full != 0u || new_hi > pp.limit ? 1ull << 56 : 0ull));
            for (unsigned k = tid; k < cells / 2u; k += THREADS) reinterpret_cast<uint4*>(counts)[k] = make_uint4(0u, 0u, 0u, 0u);
            if constexpr (!GRID) {
                if (tid == 0u) { s_mailed[turn] = 0u; s_over = 0u; }       // (the next to add to this list do so after the barrier)
                if (i < arrived) here[i].y = HOLE;
            }
            const unsigned used = min(taken, free_slots);
            head += used; if (head >= pp.slots) head -= pp.slots;
            free_slots += s_holes - used;
            hi = new_hi;
            if constexpr (GRID) { __syncwarp(); if (i == 0u) s_over = 0u; } else arrive(0u, 0ull);
            if (l.eps_mode == 1) { ++eps_index.at; if (step + 1u < l.steps) eps = __ldg(p.eps_tab + eps_index.at); }
        }
        {                                                          // back to environment order
            auto put = [&](const uint2 r) { unsigned x, y; cell_of(k0 + rec_loc(r), x, y); p.st[rec_id(r)] = make_int4((int)x, (int)y, (int)rec_t(r), (int)rec_id(r)); ++kept; };
#pragma unroll 1
            for (unsigned j = tid; j < hi; j += THREADS) if (rec[j].y != HOLE) put(rec[j]);
            if (arr.y != HOLE) put(arr);
        }
        if constexpr (GRID) {
            kept = __reduce_add_sync(FULL, kept);
            if ((tid & 31u) == 0u && kept) atomicAdd(pp.barrier + 192u, kept);
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
    if constexpr (!GRID) { space.arrive(); space.wait(); }         // (nobody leaves while others may still write into its shared memory)
    if (step < l.steps) {                                          // the same for every block
        if (b == 0u && tid == 0u && 8u * step < l.steps) {
            if (*pp.broken == l.epoch) *pp.gave_up = p.step + 1ull;
            *pp.broken = l.epoch + l.steps + 2u;
        }
        int4* const work = fits ? p.st : pp.dealt;
        if constexpr (GRID) {
            space.arrive(); if (!space.wait()) return;
            if (tid < 3u) pp.listed[tid * G + b] = 0u;             // what was listed for the step that nobody took
            // One applies what a crowd has counted: a crowd is what ends up here.  (38,000 on 200 x 190, all drawn to one cell, lr 1e-5: everybody 29.5 us a step, the first 17.6, the gather
            // engine from the start 17.1; lr 0.1 12.7 / 10.4 / 10.3.)
            run_steps<Home::Registers, THREADS, PLAIN, true>(p, l, space, work, nullptr, step);
        } else run_steps<Home::Registers, THREADS, PLAIN, true>(p, l, space, work, nullptr, step);
        if (!fits) {
            __syncthreads();
            const unsigned first = b * l.chunk, n = first < p.N ? min(l.chunk, p.N - first) : 0u;
            for (unsigned k = tid; k < n; k += THREADS) { const int4 r = work[first + k]; p.st[r.w] = r; }
        }
    }
    if (GRID && last_to_finish<false>(p)) {
        if (fits && *reinterpret_cast<volatile unsigned*>(pp.barrier + 192u) != p.N) atomicOr(&p.ctl->error, ERR_BAD_STATE);      // not every environment has come back
        pp.barrier[0] = 0u; pp.barrier[64] = pp.barrier[65] = pp.barrier[128] = pp.barrier[129] = 0u; pp.barrier[192] = 0u;
    }
}

// ------------------------------------------------------------------------------------------------
constexpr size_t PT_SHARED = 218u * 1024u;       // dynamic shared memory of a block: 227 KB less the static words here and in step_loop.cuh
static size_t patch_shared(const PatchP& pp) {
    return 25 * (size_t)pp.cells + 18 * (size_t)pp.slots + (pp.grid ? 8u : 32u) * (size_t)pp.threads + 16 * (size_t)pp.ghosts + (size_t)(pp.bits + 31u) / 32u * 4u + 16;
}
// Whether the patches of a world fit the blocks' shared memory, and how it is shared out.
static bool plan(const Params& p, PatchP& pp, bool grid) {
    pp = PatchP{};
    const size_t S = p.S, N = p.N;
    const unsigned G = grid ? std::min(p.sms, PT_MOST_BLOCKS) : (unsigned)std::min<size_t>(PT_BLOCKS, std::max<size_t>(1, (std::max(S, N) + 63) / 64));
    pp.grid = grid;
    unsigned sh = 3u;
    while (sh < 7u && ((size_t)2 << (2u * sh)) <= S / G) ++sh;       // bands about as high as a patch is wide
    while (sh > 3u && (((size_t)p.H + (1u << sh) - 1u) >> sh << sh) * 8u > (size_t)p.H * 9u) --sh;      // (and no more than an eighth of the last one empty)
    pp.shift = sh;
    pp.w_rcp = p.W > 1 ? (unsigned)((1ull << 32) / (unsigned)p.W) : 0xFFFFFFFFu;
    const size_t keys = ((((size_t)p.H + (1u << sh) - 1u) >> sh) << sh) * (size_t)p.W;
    if (keys > (size_t)G * 16384u) return false;
    pp.keys = (unsigned)keys; pp.bins = pp.keys / 8u;
    const size_t avg_n = (N + G - 1) / G;
    pp.threads = avg_n <= 128u ? 256u : avg_n <= 256u ? 512u : 768u;        // residents and arrivals in different warps
    if (grid && pp.threads == 256u) pp.threads = 512u;
    if (avg_n > pp.threads) return false;            // (what a launch gives up goes on with one environment a thread)
    pp.limit = (unsigned)(avg_n * 2u + 256u);
    pp.slots = pp.limit + pp.threads;
    if (pp.slots > 32767u) return false;
    // an environment weighs as much as w_env / 16 cells: the more the better the blocks' work is balanced, and the larger the patches where nobody is
    for (unsigned w = 128u; w >= 8u; w -= (w + 3u) / 4u) {
        pp.w_env = w;
        pp.cells = (unsigned)((keys + (N * w + 15) / 16 + G - 1) / G + 23u) & ~7u;
        pp.ghosts = 2u * (1u << sh) + 2u * (pp.cells / (1u << sh) + 2u);
        pp.bits = (unsigned)S;                           // (without, a restart takes an access to L2 or two)
        if (patch_shared(pp) > PT_SHARED) pp.bits = 0u;
        pp.shared = (unsigned)patch_shared(pp);
        if (pp.cells <= 16384u && pp.ghosts <= 16384u && pp.shared <= PT_SHARED) { pp.blocks = G; return true; }
    }
    return false;
}
// Not where episodes start on one cell, and everybody passes through one patch: 12,000 on 200 x 190 cells 3.9 / 5.2 (us a step, gather engine / a cluster here).
// Not on crowded grids: a patch is eight cells or more, and the one beside the goal has most of the population; how well that goes depends on where it lies.  Us a step, gather engine /
// patches, 256 or 512 a call, one goal: in a cluster 1,100 on 17 x 17 3.1 / 2.4, on 12 x 12 2.8 / 3.5; 1,500 on 10 x 10 3.0 / 3.8; 4,096 on 32 x 32 3.8 / 2.8, on 16 x 16 4.0 / 4.6; 6,144 on 40 x 40
// 4.0 / 4.05 (16 a call 4.3 / 5.0); 8,192 on 64 x 64 4.4 / 3.5, on 45 x 45 4.3 / 5.2; on the whole GPU 10,240 on 72 x 72 5.0 / 3.7, 12,288 on 78 x 78 4.8 / 5.2, 10,000 on 50 x 50 4.9 / 5.2.
// In a cluster up to 512 a block: 10,240 on 101 x 101 5.0 / 5.1, and there on the whole GPU 3.7; 12,288 on 157 x 157 with five goals 5.2 / 5.3 / 3.7.
// On the whole GPU up to one environment a thread.
bool patch_plan(const Params& p, PatchP& pp) {
    const size_t S = p.S, N = p.N;
    const bool sparse = N <= (N <= 4096u ? 4u : 2u) * S;
    if (p.start_mode == 2 && sparse) {
        if (N <= PT_MOST_ENVS && plan(p, pp, false)) return true;
        if (N <= (size_t)PT_MOST_THREADS * p.sms && plan(p, pp, true)) return true;
    }
    pp = PatchP{};
    return false;
}
template <unsigned THREADS, bool PLAIN, bool GRID>
static cudaError_t launch(const Params& p, const StepLaunch& l, const PatchP& pp, cudaStream_t st) {
    auto* const fn = k_patch_steps<THREADS, PLAIN, GRID>;
    cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PT_SHARED);
    if (e == cudaSuccess && !GRID) e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(pp.blocks); cfg.blockDim = dim3(THREADS); cfg.stream = st;
    cfg.dynamicSmemBytes = pp.shared;
    cudaLaunchAttribute at[1];
    if (GRID) { at[0].id = cudaLaunchAttributeCooperative; at[0].val.cooperative = 1; }
    else {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = pp.blocks; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    }
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, p, l, pp);
}
template <bool PLAIN>
static cudaError_t launch(const Params& p, const StepLaunch& l, const PatchP& pp, cudaStream_t st) {
    if (pp.grid) return pp.threads == 512u ? launch<512u, PLAIN, true>(p, l, pp, st) : launch<768u, PLAIN, true>(p, l, pp, st);
    return pp.threads == 256u ? launch<256u, PLAIN, false>(p, l, pp, st) : pp.threads == 512u ? launch<512u, PLAIN, false>(p, l, pp, st) : launch<768u, PLAIN, false>(p, l, pp, st);
}
cudaError_t launch_patch_steps(const Params& p, const StepLaunch& l, const PatchP& pp, cudaStream_t st) { return plain(p, l) ? launch<true>(p, l, pp, st) : launch<false>(p, l, pp, st); }

}  // namespace cudarl
