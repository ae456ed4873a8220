// hostio.cpp -- see hostio.h.
#include "hostio.h"
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <sys/mman.h>
#include <thread>
#include <vector>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

namespace cudarl {
namespace {

// A slot is one huge page of the caller's array where that is made of huge pages: each is faulted in by one core.  Twenty slots keep
// twelve cores and the copy engine busy.  Measured on a B200 machine (16 cores, 268 MB into a fresh NumPy array): 56 ms through the
// driver, 9.6 ms with 8 copying threads, 7.5 with 12; into memory that has been written before 5.6 either way, the speed of the link.
constexpr size_t SLOT_BYTES = (size_t)2 << 20;
constexpr size_t CHUNK_MIN = (size_t)64 << 10, PIECE_MIN = (size_t)256 << 10, HOST_CHUNK_MOST = (size_t)128 << 10;
// From here on a result array is likely to be fresh memory.
constexpr size_t TOUCH_MIN = (size_t)4 << 20;
// Copies within the host between a stage and the caller: shared from a quarter of a megabyte on.
constexpr size_t HOST_MIN = (size_t)256 << 10, HOST_PIECE = (size_t)32 << 10;
constexpr int SLOTS = 20, MAX_WORKERS = 11, MAX_DEVICES = 64;
// Below this the driver copies, although a ring that is there is the faster from half a megabyte on (B200 machine, us, ring / driver: in 512 KB 34 / 40,
// 3 MB 124 / 178, 8 MB 223 / 434; out into memory written before 768 KB 48 / 65, 4 MB 178 / 226, into fresh memory 112 / 362 and 420 / 1,830): a
// process that only has such transfers is spared the ring's set-up, 3 ms whatever its size (registering takes 0.5 - 4 ms a call), and the stages of
// the contexts take most of them anyway.
constexpr size_t SHARED_MIN_OUT = (size_t)768 << 10, SHARED_MIN_IN = (size_t)3 << 20;

// What one core copies at a time; `at`: where it lies in the slot of its piece.
struct Chunk { unsigned char* host; unsigned char* dev; size_t bytes; Fill fill; const void* arg; size_t first; size_t piece, at; };
// What the copy engine moves at a time: chunks [chunk, chunk + count).  Enqueueing one takes the caller's thread about 8 us, so they are
// larger than what is best for the cores: 4 MB in 32 pieces took 290 us.
struct Piece { unsigned char* dev; size_t bytes, chunk, count; };
enum class Way { Out, In, Host, HostIn, Touch }; // device -> caller, caller -> device, stage -> caller, caller -> stage; pages of the caller faulted in

// One transfer.  The caller's thread alone talks to the driver (several threads asking for events and enqueueing copies hold each
// other up in it) and copies when it has nothing else to do; the workers only copy.
struct Job {
    std::vector<Chunk> chunks; std::vector<Piece> pieces;
    Way way = Way::Host;
    std::atomic<size_t> next{0};                 // first chunk nobody has taken
    std::atomic<size_t> landed{0};               // Out: chunks whose piece is complete
    std::atomic<size_t> turn[SLOTS];             // the piece the slot is free for
    std::atomic<size_t> copied[SLOTS];           // chunks of the slot's piece copied out of it, or into it
    std::atomic<size_t> done{0};                 // chunks copied by a thread
    std::atomic<bool> failed{false};
    std::atomic<int> busy{0};                    // workers inside the job
};

struct Pool {
    std::mutex mu;                               // members below
    int refs = 0;
    std::vector<Stage> spare;                    // blocks given back by contexts that went
    std::mutex use;                              // held by the one transfer that uses the ring
    unsigned char *ring = nullptr, *raw = nullptr;       // slots, and the mapping they lie in
    cudaEvent_t events[MAX_DEVICES][SLOTS] = {};
    // workers
    std::mutex wmu; std::condition_variable wake;
    std::vector<std::thread> workers;
    Job* job = nullptr; std::atomic<uint64_t> job_no{0}; std::atomic<bool> stop{false};
};
Pool& pool() { static Pool* p = new Pool; return *p; }     // never destroyed: workers may outlive static destructors at process exit

inline void cpu_relax() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
}

// Have the page of a byte faulted in for writing, the byte unchanged: the result that will lie there may never come.  One access that reads and
// writes: a read first would map the page of zeros, which takes a second fault, and huge pages apart.
inline void fault_in(unsigned char* b) {
#if defined(__x86_64__)
    asm volatile("lock orb $0, %0" : "+m"(*b) : : "memory", "cc");
#else
    __atomic_fetch_or(b, (unsigned char)0, __ATOMIC_RELAXED);
#endif
}

// Into memory that the device reads next: past the caches.  The device's reads of lines that lie modified in a core's cache run at
// about 5 GB/s on a B200 machine (16 MB took 1.3 ms, 0.45 ms this way).  line_end: the rest of the line that the last
// byte lies in is nobody's and may be written.
void copy_past_caches(unsigned char* d, const unsigned char* s, size_t n, bool line_end) {
#if defined(__x86_64__)
    size_t k = std::min(n, (size_t)(-(intptr_t)d & 15));
    std::memcpy(d, s, k);
    for (; k + 64 <= n; k += 64) {
        const __m128i a = _mm_loadu_si128((const __m128i*)(s + k)), b = _mm_loadu_si128((const __m128i*)(s + k + 16)),
                      c = _mm_loadu_si128((const __m128i*)(s + k + 32)), e = _mm_loadu_si128((const __m128i*)(s + k + 48));
        _mm_stream_si128((__m128i*)(d + k), a); _mm_stream_si128((__m128i*)(d + k + 16), b);
        _mm_stream_si128((__m128i*)(d + k + 32), c); _mm_stream_si128((__m128i*)(d + k + 48), e);
    }
    if (k < n && line_end && ((uintptr_t)(d + k) & 63u) == 0u) {      // a whole line again, so that it stays out of this core's cache
        alignas(16) unsigned char rest[64] = {};
        std::memcpy(rest, s + k, n - k);
        for (int b = 0; b < 64; b += 16) _mm_stream_si128((__m128i*)(d + k + b), _mm_load_si128((const __m128i*)(rest + b)));
    } else std::memcpy(d + k, s + k, n - k);
    _mm_sfence();
#else
    std::memcpy(d, s, n);
#endif
}

// A chunk on its way to the device: copied, or made in pieces that fit the first-level cache.
void send(unsigned char* dst, const unsigned char* src, const Chunk& c, bool line_end) {
    if (!c.fill) { copy_past_caches(dst, src, c.bytes, line_end); return; }
    alignas(64) unsigned char part[8192];
    for (size_t k = 0; k < c.bytes; k += sizeof(part)) {
        const size_t b = std::min(sizeof(part), c.bytes - k);
        c.fill(part, c.first + k, b, c.arg);
        copy_past_caches(dst + k, part, b, line_end);
    }
}

// Take and copy one chunk if one is ready.
bool copy_one(Job& j) {
    size_t k = j.next.load(std::memory_order_relaxed);
    if (k >= j.chunks.size()) return false;
    const Chunk& c = j.chunks[k];
    const size_t slot = c.piece % SLOTS;
    if (j.way == Way::Out && k >= j.landed.load(std::memory_order_acquire)) return false;
    if (j.way == Way::In && j.turn[slot].load(std::memory_order_acquire) != c.piece) return false;
    if (!j.next.compare_exchange_strong(k, k + 1)) return true;          // another thread was quicker: look again
    unsigned char* const buf = pool().ring + slot * SLOT_BYTES + c.at;
    switch (j.way) {
        case Way::Out:
            std::memcpy(c.host, buf, c.bytes);
            if (j.copied[slot].fetch_add(1, std::memory_order_acq_rel) + 1 == j.pieces[c.piece].count) { j.copied[slot] = 0; j.turn[slot].store(c.piece + SLOTS, std::memory_order_release); }
            break;
        case Way::In: send(buf, c.host, c, false); j.copied[slot].fetch_add(1, std::memory_order_release); break;
        case Way::Host: std::memcpy(c.host, c.dev, c.bytes); break;
        case Way::HostIn: send(c.host, c.dev, c, true); break;
        case Way::Touch: for (size_t b = 0; b < c.bytes; b += 4096) fault_in(c.host + b); break;
    }
    j.done.fetch_add(1, std::memory_order_release);
    return true;
}
void help(Job& j) {
    while (j.next.load(std::memory_order_relaxed) < j.chunks.size() && !j.failed) if (!copy_one(j)) cpu_relax();
}

constexpr int IDLE_LOOKS = 2000;                 // about 50-100 us

void worker_main() {
    Pool& p = pool();
    uint64_t seen = 0;
    for (;;) {
        Job* j;
        // transfers come in bursts (actions in, rewards out): look for the next one for a moment before going to sleep
        for (int k = 0; k < IDLE_LOOKS && !p.stop && p.job_no.load(std::memory_order_relaxed) == seen; ++k) cpu_relax();
        {
            std::unique_lock<std::mutex> lk(p.wmu);
            p.wake.wait(lk, [&] { return p.stop || (p.job && p.job_no != seen); });
            if (p.stop) return;
            seen = p.job_no; j = p.job;
            j->busy.fetch_add(1);                 // under the lock: the caller withdraws the job before it waits for busy == 0
        }
        help(*j);
        j->busy.fetch_sub(1);
    }
}

// Under `use`.
void ready_workers() {
    Pool& p = pool();
    if (!p.workers.empty()) return;
    const int n = std::min(MAX_WORKERS, (int)std::thread::hardware_concurrency() * 3 / 4 - 1);      // with the caller three quarters of the cores
    p.stop = false;
    try {
        for (int k = 0; k < n; ++k) p.workers.emplace_back(worker_main);
    } catch (const std::exception&) {}           // a limit on threads: those that exist do, or the caller's alone
}
// Cut into chunks of at most `most` bytes, or of less (but not below `least`) so that a short transfer still has two for every core; for the
// copy engine (`pieces`) into eight pieces or more, of up to a slot, each of whole chunks.
void cut(Job& j, const Segment* segs, int n, size_t most, size_t least, bool pieces) {
    size_t total = 0, chunk = most, piece = SLOT_BYTES;
    for (int s = 0; s < n; ++s) total += segs[s].bytes;
    while (chunk > least && total / chunk < 2u * (MAX_WORKERS + 1)) chunk >>= 1;
    while (piece > PIECE_MIN && total / piece < 8u) piece >>= 1;
    for (int s = 0; s < n; ++s) {
        unsigned char* h = (unsigned char*)segs[s].host; unsigned char* d = (unsigned char*)segs[s].dev;
        const bool made = segs[s].fill != nullptr;
        const uintptr_t base = made ? 0u : (uintptr_t)h;
        for (size_t first = 0; first < segs[s].bytes;) {
            if (pieces && (first == 0 || ((base + first) & (piece - 1)) == 0)) j.pieces.push_back(Piece{d + first, 0, j.chunks.size(), 0});
            const size_t edge = chunk - ((base + first) & (chunk - 1)), b = std::min(segs[s].bytes - first, edge);
            Chunk c{made && !h ? nullptr : h + first, made && !d ? nullptr : d + first, b, segs[s].fill, segs[s].arg, first, 0, 0};
            if (pieces) { Piece& p = j.pieces.back(); c.piece = j.pieces.size() - 1; c.at = p.bytes; p.bytes += b; ++p.count; }
            j.chunks.push_back(c);
            first += b;
        }
    }
}
void publish(Job& j) {
    Pool& p = pool();
    { std::lock_guard<std::mutex> lk(p.wmu); p.job = &j; ++p.job_no; }
    p.wake.notify_all();
}
void withdraw(Job& j) {
    Pool& p = pool();
    { std::lock_guard<std::mutex> lk(p.wmu); p.job = nullptr; }
    while (j.busy.load(std::memory_order_acquire)) cpu_relax();
}

// Ordinary memory, faulted in by all cores as huge pages and then registered: 3 ms for the 40 MB that cudaHostAlloc takes 20 for.
cudaError_t ready_ring(int device) {
    Pool& p = pool();
    if (!p.ring) {
        const size_t bytes = SLOT_BYTES * SLOTS;
        unsigned char* const raw = (unsigned char*)mmap(nullptr, bytes + SLOT_BYTES, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        if (raw == MAP_FAILED) return cudaErrorMemoryAllocation;
        unsigned char* const ring = (unsigned char*)(((uintptr_t)raw + SLOT_BYTES - 1) & ~(uintptr_t)(SLOT_BYTES - 1));
        madvise(ring, bytes, MADV_HUGEPAGE);
        const Segment all{ring, nullptr, bytes, [](void* d, size_t, size_t n, const void*) { std::memset(d, 0, n); }, nullptr};
        Job j;
        j.way = Way::HostIn;
        cut(j, &all, 1, SLOT_BYTES, SLOT_BYTES, false);
        publish(j);
        help(j);
        withdraw(j);
        const cudaError_t e = cudaHostRegister(ring, bytes, cudaHostRegisterPortable);
        if (e != cudaSuccess) { munmap(raw, bytes + SLOT_BYTES); return e; }
        p.raw = raw; p.ring = ring;
    }
    for (int k = 0; k < SLOTS; ++k)
        if (!p.events[device][k]) { const cudaError_t e = cudaEventCreateWithFlags(&p.events[device][k], cudaEventDisableTiming); if (e != cudaSuccess) return e; }
    return cudaSuccess;
}

cudaError_t run_job(Job& j, int device, cudaStream_t st) {
    Pool& p = pool();
    cudaEvent_t* const ev = p.events[device];
    const size_t n = j.pieces.size();
    for (size_t k = 0; k < SLOTS; ++k) { j.turn[k] = k; j.copied[k] = 0; }
    publish(j);
    size_t issued = 0, complete = 0;             // pieces enqueued, and known to be complete, in order
    cudaError_t e = cudaSuccess;
    while (e == cudaSuccess && (complete < n || j.done.load(std::memory_order_acquire) < j.chunks.size())) {
        // what has landed first: the other threads wait for it
        if (complete < issued) {
            const size_t slot = complete % SLOTS;
            const cudaError_t q = cudaEventQuery(ev[slot]);
            if (q == cudaSuccess) {
                if (j.way == Way::In) { j.copied[slot] = 0; j.turn[slot].store(complete + SLOTS, std::memory_order_release); }
                else j.landed.store(j.pieces[complete].chunk + j.pieces[complete].count, std::memory_order_release);
                ++complete;
                continue;
            }
            if (q != cudaErrorNotReady) { e = q; break; }
        }
        if (issued < n) {
            const size_t slot = issued % SLOTS;
            const Piece& c = j.pieces[issued];
            unsigned char* const buf = p.ring + slot * SLOT_BYTES;
            const bool ready = j.turn[slot].load(std::memory_order_acquire) == issued && (j.way == Way::Out || j.copied[slot].load(std::memory_order_acquire) == c.count);
            if (ready) {
                e = j.way == Way::Out ? cudaMemcpyAsync(buf, c.dev, c.bytes, cudaMemcpyDeviceToHost, st) : cudaMemcpyAsync(c.dev, buf, c.bytes, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaEventRecord(ev[slot], st);
                ++issued;
                continue;
            }
        }
        // In: a thread that copies does not send off what the others have filled, and the link idles meanwhile
        if (j.way == Way::Out || p.workers.empty()) copy_one(j); else cpu_relax();
    }
    if (e != cudaSuccess) { j.failed = true; withdraw(j); cudaStreamSynchronize(st); return e; }
    withdraw(j);
    return cudaSuccess;
}

cudaError_t copy_all(const Segment* segs, int n, bool out, int device, cudaStream_t st) {
    size_t total = 0;
    bool made = false;
    for (int s = 0; s < n; ++s) { total += segs[s].bytes; made |= segs[s].fill != nullptr; }
    Pool& p = pool();
    if ((made || total >= (out ? SHARED_MIN_OUT : SHARED_MIN_IN)) && device >= 0 && device < MAX_DEVICES) {
        if (out && total >= TOUCH_MIN && cudaStreamQuery(st) == cudaErrorNotReady) {
            // the device is still at work enqueued earlier: the pages the results go to are faulted in meanwhile
            std::unique_lock<std::mutex> lk(p.use, std::try_to_lock);
            if (lk.owns_lock()) {
                ready_workers();
                Job t;
                t.way = Way::Touch;
                cut(t, segs, n, SLOT_BYTES, SLOT_BYTES, false);
                publish(t);
                help(t);
                withdraw(t);
            }
        }
        const cudaError_t e = cudaStreamSynchronize(st);               // without the ring: the wait may be as long as a training run
        if (e != cudaSuccess) return e;
        std::unique_lock<std::mutex> lk(p.use, std::try_to_lock);      // another thread's transfer has the ring: let the driver do this one
        if (lk.owns_lock()) {
            ready_workers();
            if (ready_ring(device) == cudaSuccess) {
                Job j;
                j.way = out ? Way::Out : Way::In;
                cut(j, segs, n, SLOT_BYTES, CHUNK_MIN, true);
                return run_job(j, device, st);
            }
            cudaGetLastError();                  // no pinned memory to be had: the driver's copies do without
        }
    }
    for (int s = 0; s < n; ++s) {
        if (segs[s].fill) {                      // through pageable memory of our own
            const size_t room = std::min(segs[s].bytes, SLOT_BYTES);
            const std::unique_ptr<unsigned char[]> made(new (std::nothrow) unsigned char[room]);
            if (!made) return cudaErrorMemoryAllocation;
            for (size_t first = 0; first < segs[s].bytes; first += room) {
                const size_t b = std::min(room, segs[s].bytes - first);
                segs[s].fill(made.get(), first, b, segs[s].arg);
                cudaError_t e = cudaMemcpyAsync((unsigned char*)segs[s].dev + first, made.get(), b, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                if (e != cudaSuccess) return e;
            }
            continue;
        }
        const cudaError_t e = out ? cudaMemcpyAsync(segs[s].host, segs[s].dev, segs[s].bytes, cudaMemcpyDeviceToHost, st)
                                  : cudaMemcpyAsync(segs[s].dev, segs[s].host, segs[s].bytes, cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(st);
}

}  // namespace

// Plain loops over plain arrays, which the compiler turns into vector code; with AVX2 where the processor has it.
#if defined(__x86_64__) && defined(__GNUC__) && !defined(__clang__)
#define VECTORISED __attribute__((target_clones("avx2", "default"), optimize("O3")))
#else
#define VECTORISED
#endif
VECTORISED static uint32_t cells_actions(uint32_t* __restrict o, const int32_t* __restrict x, const int32_t* __restrict y, const int32_t* __restrict a,
                                         const uint8_t* __restrict dn, size_t n, uint32_t W, uint32_t H) {
    uint32_t bad = 0;
    for (size_t k = 0; k < n; ++k) {
        const uint32_t ux = (uint32_t)x[k], uy = (uint32_t)y[k], ua = (uint32_t)a[k];
        bad |= (uint32_t)(ux >= W) | (uint32_t)(uy >= H) | (uint32_t)(ua >= 4u);
        o[k] = ((uy * W + ux) << 2) | (ua & 3u) | ((uint32_t)(dn[k] != 0) << 31);
    }
    return bad;
}
VECTORISED static uint32_t cells(uint32_t* __restrict o, const int32_t* __restrict x, const int32_t* __restrict y, size_t n, uint32_t W, uint32_t H) {
    uint32_t bad = 0;
    for (size_t k = 0; k < n; ++k) {
        const uint32_t ux = (uint32_t)x[k], uy = (uint32_t)y[k];
        bad |= (uint32_t)(ux >= W) | (uint32_t)(uy >= H);
        o[k] = uy * W + ux;
    }
    return bad;
}
VECTORISED static uint32_t bounded(uint32_t* __restrict o, const int32_t* __restrict v, size_t n, uint32_t most) {
    uint32_t bad = 0;
    for (size_t k = 0; k < n; ++k) { const uint32_t u = (uint32_t)v[k]; bad |= (uint32_t)(u > most); o[k] = u; }
    return bad;
}
void copy_bounded(void* dst, size_t first, size_t bytes, const void* source) {
    BoundedSource& s = *(BoundedSource*)source;
    if (bounded((uint32_t*)dst, s.from + first / 4, bytes / 4, s.most)) s.bad = true;
}
void pack_cell_action(void* dst, size_t first, size_t bytes, const void* source) {
    TransitionSource& s = *(TransitionSource*)source;
    const size_t i = first / 4;
    if (cells_actions((uint32_t*)dst, s.sx + i, s.sy + i, s.a + i, s.dn + i, bytes / 4, s.W, s.H)) s.bad = true;
}
void pack_next_cell(void* dst, size_t first, size_t bytes, const void* source) {
    TransitionSource& s = *(TransitionSource*)source;
    const size_t i = first / 4;
    if (cells((uint32_t*)dst, s.nx + i, s.ny + i, bytes / 4, s.W, s.H)) s.bad = true;
}

void hostio_retain() { Pool& p = pool(); std::lock_guard<std::mutex> lk(p.mu); ++p.refs; }

void hostio_release() {
    Pool& p = pool();
    std::lock_guard<std::mutex> lk(p.mu);
    if (--p.refs > 0) return;
    std::lock_guard<std::mutex> use(p.use);
    { std::lock_guard<std::mutex> w(p.wmu); p.stop = true; }
    p.wake.notify_all();
    for (auto& t : p.workers) t.join();
    p.workers.clear();
    if (p.ring) { cudaHostUnregister(p.ring); munmap(p.raw, SLOT_BYTES * (SLOTS + 1)); p.ring = p.raw = nullptr; }
    for (auto& dev : p.events) for (auto& e : dev) if (e) { cudaEventDestroy(e); e = nullptr; }
    for (auto& s : p.spare) cudaFreeHost(s.host);
    p.spare.clear();
}

cudaError_t stage_take(Stage* s, size_t bytes) {
    Pool& p = pool();
    {
        std::lock_guard<std::mutex> lk(p.mu);
        for (size_t k = 0; k < p.spare.size(); ++k)
            if (p.spare[k].bytes == bytes) { *s = p.spare[k]; p.spare.erase(p.spare.begin() + (long)k); std::memset(s->host, 0, 256); return cudaSuccess; }
    }
    Stage t;
    t.bytes = bytes;
    cudaError_t e = cudaHostAlloc((void**)&t.host, bytes, cudaHostAllocPortable | cudaHostAllocMapped);
    if (e != cudaSuccess) return e;
    e = cudaHostGetDevicePointer((void**)&t.dev, t.host, 0);
    if (e != cudaSuccess) { cudaFreeHost(t.host); return e; }
    std::memset(t.host, 0, 256);
    *s = t;
    return cudaSuccess;
}
void stage_give(Stage* s) {
    if (!s->host) return;
    Pool& p = pool();
    std::lock_guard<std::mutex> lk(p.mu);
    if (p.spare.size() < 4) p.spare.push_back(*s); else cudaFreeHost(s->host);
    *s = Stage{};
}

void copy_host(const Segment* segs, int n, bool into_stage) {
    size_t total = 0;
    for (int s = 0; s < n; ++s) total += segs[s].bytes;
    if (total >= HOST_MIN) {
        std::unique_lock<std::mutex> lk(pool().use, std::try_to_lock);
        if (lk.owns_lock()) {
            ready_workers();
            Job j;
            j.way = into_stage ? Way::HostIn : Way::Host;
            cut(j, segs, n, HOST_CHUNK_MOST, HOST_PIECE, false);
            publish(j);
            help(j);
            withdraw(j);                         // every worker has left: every chunk is copied
            return;
        }
    }
    for (int s = 0; s < n; ++s)
        if (into_stage) send((unsigned char*)segs[s].host, (const unsigned char*)segs[s].dev, Chunk{nullptr, nullptr, segs[s].bytes, segs[s].fill, segs[s].arg, 0}, true);
        else std::memcpy(segs[s].host, segs[s].dev, segs[s].bytes);
}
cudaError_t copy_out(const Segment* segs, int n, int device, cudaStream_t st) { return copy_all(segs, n, true, device, st); }
cudaError_t copy_in(const Segment* segs, int n, int device, cudaStream_t st) { return copy_all(segs, n, false, device, st); }

}  // namespace cudarl
