// kernels.cuh -- device-side data layout and launch entry points shared by kernels.cu, tile_engine.cu (the
// sm_100a kernels) and context.cu (the C ABI).  Nothing here is visible outside the library.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cudarl {

// ---- per-cell word (16 bits per grid cell, array padded to 256 bytes): the cell's class ------------
enum : unsigned {
    CW_OBST = 1u,      // cell blocks movement                     (src/kernels.cu:29-36 of the reference)
    CW_GOAL = 2u,      // cell ends the episode, reward 1          (src/environment.cu:43-46)
    CW_TRAP = 4u,      // an obstacle whose penalty replaces the step cost of an agent that walks into it (src/kernels.cu:61-63)
};

// ---- control block in device memory ------------------------------------------------------------
struct Ctl {
    unsigned long long episodes, goals, timeouts, conflicts, long_chains;
    unsigned long long eval_reached, eval_steps;   // sums of a running rollout; zero between rollouts
    unsigned int done_blocks;       // blocks of a kernel that hands results to the host: those that have written theirs; zero between kernels
    unsigned long long general;     // environment-steps that went through the entry/chain path
    unsigned int eps_idx;           // index of the current step's epsilon in the table
    unsigned int eps_mode;          // 0 fixed index, 1 advance by one per step, 2 per-episode index
    unsigned int eps_len;           // table length (clamp)
    unsigned long long eps_base_k;  // per-episode mode: table[0] belongs to episodes/N == eps_base_k
    unsigned int active_count;      // update_batch: mailbox slots holding a chain,
    unsigned int long_count;        // chains left to k_fix_long: zero between calls
    unsigned int error;             // sticky internal error bits
    unsigned int never;             // zero for good: what a wait that a test makes run out looks at
    float eps_used;                 // epsilon of the most recent step (for the stats call)
};

enum : unsigned { ERR_SCRATCH_OVERFLOW = 1u, ERR_BAD_STATE = 2u, ERR_COPY_TIMEOUT = 32u };   // = CUDARL_DEVERR_* of cudarl.h

// ---- results handed to the host without a copy ---------------------------------------------------
// One per context, at the head of its pinned, mapped stage block.  A word carries 32 bits of a result and, above them, the number of
// the call it belongs to: the host waits for each word it needs by its number, so the words need no order among themselves and no
// fence (launch to seen result 7.3 us on a B200 machine, 9.3 with values, fence and flag, 9 - 10 for a copy or a synchronisation of
// the stream).  Word 0 carries Ctl::error and is also the flag behind arrays in the stage, which do take a fence.
struct HostBox { unsigned long long w[31], gave_up; };           // (gave_up: see PatchP)
struct Handover { HostBox* box; unsigned ticket; };              // box == nullptr: nothing to hand over

// ---- tile engine (tile_engine.cu): the layout the train step runs on ---------------------------
// The grid is cut into T x T tiles (T = 16 or 8); one WARP steps one tile at a time.  The table is a single
// dense array updated in place: a tile's cells are read and written by the tile's own warp only, and what
// a move across a tile edge needs from the neighbour -- max_a Q_t of the cell beyond the edge -- comes from a
// small double-buffered border array that every tile refreshes at the end of its step.
// Every tile owns a REGION of the record array that only the tile's own warp writes (environments that
// stay) and a fixed arrival buffer that other warps append to with an atomic cursor (environments that
// walk or restart into the tile).  Records, counters and border values alternate by step parity, so a step
// reads one set and writes the other.
constexpr unsigned ARR_CAP = 32u;  // arrival slots per tile and step; what does not fit goes to the spill list
struct TileP {
    unsigned tshift, T;        // tile edge = 1 << tshift cells
    unsigned tiles_x, tiles_y, ntiles;
    unsigned tiles_x_rcp;      // floor(2^32 / tiles_x): umulhi(n, tiles_x_rcp) is n / tiles_x or one less, for every n < 2^32
    unsigned grid;             // blocks of the persistent step kernel (SMs x resident blocks per SM)
    unsigned wait_polls;       // 0: copy waits are bounded by time (seconds); > 0 (tests only): a wait of this many polls before the copies are issued, which must run out
    uint2* rec[2];             // 8-byte records {id, t << 8 | row in tile << 4 | column in tile} of the environments that stayed; [step & 1] is current
    uint2* reg;                // ntiles + 1: {start of the tile's region, its capacity}
    uint2* cnt[2];             // ntiles: {records in the region, records in the arrival buffer}
    uint2* arr[2];             // ntiles x ARR_CAP arrival slots, same 8-byte records
    int4* ovf[2];              // records {x, y, t, id} that found their tile's arrival buffer full, any tile, N slots
    unsigned* tctl;            // [0..2] spill counts (read step%3, append (step+1)%3, clear (step+2)%3); [3..4] scratch cursors by parity
    unsigned char* tcls;       // ntiles x cls_stride: one move byte per cell, tile by tile (which of the four moves are blocked / end on a goal)
    unsigned cls_stride;
    float* bmax[2];            // ntiles x 4T: max_a Q of the cells just outside the tile's north / south / west / east edge; [step & 1] is current
    uint2* scratch;            // scratch_cap x 8 bytes: 32-bit (cell, action) counters of the tiles the general path counts in global memory
    unsigned scratch_cap;
    unsigned nq;               // tile queues of the step kernel: one per SM
    unsigned* tq;              // 3 x nq ticket counters: [step % 3] in use, [(step + 2) % 3] cleared
    CUtensorMap tmq;           // the table as a 2-D tensor of floats (4W x H), box 4T x T: one copy instruction per tile
};

// ---- gather engine (gather_engine.cu): many train steps per launch, for tables that stay in L2 -----
struct GatherP {
    unsigned* barrier;         // arrivals of all blocks of all launches so far (wraps)
    unsigned* cnt[2];          // 4 S counters: environments on a (cell, action) in this step, by step parity; zero between launches
    unsigned char* mv;         // S move bytes
    unsigned char* state;      // N x 24 bytes: the environments during a launch, where shared memory has no room for them
    unsigned *bins, *part, *rank;           // dealing by cell: 8 counters per 8 x 8 cells (zero between launches), one word per block, N ranks
    unsigned bins_x, nbins;
    unsigned chunk, grid, threads;          // environments per block; blocks; threads per block
    unsigned home;                          // where the environments are during a launch: 0 registers, 1 shared memory, 2 global memory
    unsigned deal_every;                    // steps between two dealings by cell; 0 = the environments stay in their order
    unsigned cluster, arena;                // all blocks in one cluster; the world in the shared memory of one block
};
// ---- patch engine (patch_engine.cu): the world in the shared memory of several blocks, for launches of many steps ----
constexpr unsigned PT_MOST_THREADS = 768u, PT_BLOCKS = 16u, PT_MOST_BLOCKS = 256u, PT_MOST_ENVS = 8192u, PT_CLUSTERS = 8u, PT_BIN_WEIGHT = 128u;      // 16 for each of a bin's cells
struct PatchP {
    unsigned blocks, threads;  // 0 blocks: the world does not fit
    bool grid;                 // on all multiprocessors instead of in a cluster
    unsigned shift, keys, bins;             // rows of a band = 1 << shift; cells of all bands; bins of eight cells
    unsigned cells, slots, limit, ghosts;   // most cells, slots, environments and edge values of a patch
    unsigned w_env, shared;    // weight of an environment; bytes of shared memory
    unsigned bits, w_rcp;      // cells in the map of start cells (all or none); floor(2^32 / W): umulhi(n, w_rcp) is n / W or one less, for every n < 2^32
    unsigned *count, *part, *rank, *cut;    // the counting sort: per bin (zero between launches), per block, per environment; first bin of every patch
    int4* dealt;               // the records sorted by bin
    unsigned* broken;          // the number (epoch) of the launch after the last that patches have not seen through its first eighth
    volatile unsigned long long* gave_up;   // a word of the box: one more than the first step of the last such launch that came behind another
    // grid: words under the number of their step
    unsigned* barrier;         // a barrier of the grid; from word 64 on, two counters 256 bytes apart; word 192, the environments that have come back; zero between launches
    unsigned* listed;          // 3 x blocks: records in a block's list, by step modulo 3; zero before they are for
    unsigned long long *list, *edge;        // 3 x blocks x threads records of two words; 2 x keys: max_a Q of the cells along the patches' edges
};
struct StepLaunch {
    unsigned steps, chunk, barrier_base, epoch;          // epoch: the number of the first step for the patch engine's words, used once
    int eps_mode, trace;
    unsigned eps_len; unsigned long long eps_base_k;     // eps_mode 2: entries of the table, and the episodes / environments of its first
    const int4* in; int4* out;                           // in != out: deal by cell first
};

// ---- everything a kernel needs, passed by value ------------------------------------------------
// The world as the small kernels need it: a launch costs 0.5 us less with these 170 bytes than with all of Params.
struct World {
    int W, H;
    unsigned S;            // cells
    unsigned N;            // local environments
    unsigned env_offset;   // global index of local env 0
    unsigned k0, k1;       // Philox key base = seed (k1 is xor-ed with the stream tag)
    int max_steps;
    int start_mode;
    unsigned start_cell;   // CENTRE / FIXED start
    unsigned fallback_start;
    float lr, gamma;
    int legacy_clamp;
    float4* Q;             // the table: S float4, row s = the 4 action values of cell s; every kernel updates it in place
    unsigned short* cw;    // S cell words (padded to 256 bytes: map_closed of step_loop.cuh reads 64 at a time)
    const uint2* traps;    // sparse trap table, ascending by cell: {cell, penalty as float bits}
    unsigned ntraps;
    // environment state outside train steps: one int4 {x, y, t, id} per environment (all int32, one
    // coalesced 16-byte vector per thread), record k = environment k
    int4* st;
    int4* st2;             // scratch of the same size (export of x[N] | y[N] | t[N])
    float* reward; unsigned char* done;        // per ENVIRONMENT (caller-driven stepping only)
    Ctl* ctl;
    unsigned long long step;   // set by the host per launch: global batched step index g (keys the policy stream, selects the counter plane)
};
constexpr unsigned SORT_MOST_BLOCKS = 256u;
struct SortP {
    unsigned* barrier;     // zero between calls
    uint2 *a, *b;          // {cell * 4 + action, target}: as many as transitions
    unsigned *part, *total, *hist;     // per block, per digit, per digit and block
    unsigned blocks;       // of the launch: all run at the same time
};
constexpr size_t SORT_WORDS = 1u + SORT_MOST_BLOCKS + 512u + 512u * (size_t)SORT_MOST_BLOCKS;      // barrier, part, total, hist
struct Params : World {
    unsigned policy_keys[20];   // the ten round keys of the policy stream, two words each: operands straight from the constant bank (on an 8-byte
                                // boundary: 4 bytes further a step on 8 x 8 tiles took 302 us instead of 297)
    unsigned policy_pre[4];     // k_tile_step: what its step and the keys alone make of the first two rounds
    uint4* ent;            // update_batch, by transition: cell * 4 + action, index, target, index + 1 of the next in its chain (0 = end)
    unsigned sms;          // multiprocessors of the device
    unsigned* mailbox;     // update_batch: chain heads (0 = empty), power-of-two size
    unsigned mb_slots;     // mailbox slots (power of two, multiple of BLOCK)
    unsigned* active;      // list of the mailbox slots that hold a chain in this step (mb_slots entries)
    unsigned* longq;       // slots of the chains left to k_fix_long (mb_slots entries)
    const float* eps_tab;
    int* tr_a; float* tr_r; unsigned char* tr_d;   // optional trace of the last step, per ENVIRONMENT
    SortP so;              // update_batch: the sort of k_fix_long
    // per-launch values set by the host
    unsigned eps_idx;          // index of this step's epsilon in eps_tab
    int eps_from_ctl;          // 1: take the index from ctl (per-episode schedule)
    TileP tp;
    GatherP gp;
};

constexpr int BLOCK = 256;
constexpr unsigned STEP_SAT = 0xFFFFFEu;    // an episode's step counter saturates here (the tile records keep 24 bits of it)

// launch wrappers (kernels.cu); all asynchronous on `st`
void launch_identity_ids(const Params& p, cudaStream_t st);
void launch_export_state(const Params& p, int* out, unsigned stride, Handover h, cudaStream_t st);   // out = x | y | t in environment order, rows of `stride` words (a multiple of 4)
struct CopySpan { const void* src; void* dst; unsigned bytes; };
void launch_copy_out(const Params& p, const CopySpan* spans, int n, Handover h, cudaStream_t st); // up to two spans of device memory into mapped host memory
void launch_post(const Params& p, Handover h, cudaStream_t st);                                   // words 1.. = the counters of the control block, in the order of cudarl_stats, low half first; then epsilon
void launch_import_state(const Params& p, const int* x, const int* y, const int* t, cudaStream_t st);
void launch_reset_all(const Params& p, cudaStream_t st);
void launch_step_actions(const Params& p, const int* d_actions, float* d_rewards, unsigned char* d_dones, Handover h, cudaStream_t st);
void launch_step_one(const Params& p, int action, bool reset, int x, int y, Handover h, cudaStream_t st);        // one environment: words 1-4 = x, y, reward bits, done
// update_batch: transitions checked and packed by the host, in device memory or in the mapped stage -- cell * 4 + action with bit 31 =
// the episode ended there; next cell; reward.  The box is posted when the table is updated.
struct Transitions { const unsigned* at; const unsigned* next; const float* r; };
constexpr unsigned UPDATE_SMALL = 1024u;
void launch_update_batch(const Params& p, unsigned n, const Transitions& tr, Handover h, cudaStream_t st);
void launch_q_init(const Params& p, int kind, float scale, cudaStream_t st);
// greedy rollout (rollout.cu); hop: one word per cell, scratch; words 1-4 = environments that reached a goal, steps taken, low halves first
cudaError_t launch_rollout(const Params& p, unsigned* hop, unsigned max_steps, unsigned long long nonce, Handover h, cudaStream_t st);
// tile engine (tile_engine.cu)
size_t tile_step_smem(const Params& p);
int  tile_engine_configure(Params& p, int device);                  // opt in to the dynamic shared memory the step needs; sets tp.grid
void launch_tile_bucket(const Params& p, cudaStream_t st);         // p.st (any slot order) -> tile regions of parity p.step & 1
void launch_tile_classes(const Params& p, cudaStream_t st);       // cell words -> per-tile class bytes (after any change of the grid)
void launch_tile_export(const Params& p, cudaStream_t st);         // tile regions -> p.st in environment order
void launch_tile_step(Params& p, bool trace, cudaStream_t st);
unsigned tile_cls_stride(unsigned tshift);                         // bytes of one tile's class block
void launch_tile_border(const Params& p, cudaStream_t st);         // border array of parity p.step & 1 from the table (after any change of the table outside train steps)
// gather engine (gather_engine.cu)
void gather_plan(Params& p);
unsigned gather_barriers(const StepLaunch& l);                      // arrivals per block of a launch
void launch_gather_export(const Params& p, const int4* work, cudaStream_t st);      // records in any order -> p.st
void launch_gather_moves(const Params& p, cudaStream_t st);         // cell words -> move bytes
cudaError_t launch_gather_steps(const Params& p, const StepLaunch& l, cudaStream_t st);
// patch engine (patch_engine.cu)
bool patch_plan(const Params& p, PatchP& pp);                       // false: the world does not fit
cudaError_t launch_patch_steps(const Params& p, const StepLaunch& l, const PatchP& pp, cudaStream_t st);      // p.st -> p.st (or from l.in)
// arena engine (arena_engine.cu)
bool arena_plan(Params& p);                                         // false: the world does not fit
cudaError_t launch_arena_steps(const Params& p, const StepLaunch& l, cudaStream_t st);
// Replica averaging, the slice this rank owns: table[cell0 + i] = (sum over ranks 0..R-1 in that order) / R, where rank `self`'s
// rows are the table's own and the other ranks' rows lie in `others` (R - 1 slices of n rows, ascending rank).
void launch_q_average_peers(float4* const* tables, unsigned R, unsigned self, size_t cell0, size_t n, float scale, cudaStream_t st);
void launch_q_average_slice(float4* table, const float4* others, unsigned R, unsigned self, size_t cell0, size_t n, float scale, cudaStream_t st);
void launch_cell_set(const Params& p, unsigned cell, unsigned cls, int clear_goals, cudaStream_t st);

}  // namespace cudarl
