// hostio_check.cpp -- the copies between caller memory and the device (hostio.cpp) on a machine without one: the runtime calls they make are
// answered by the stand-ins below, "device" memory is host memory, and what cannot be had in earnest (a thread that does not start, memory that
// cannot be pinned, a stream that fails) is had by a switch.  One scenario per run, named on the command line; 0 = as it should be.
#include "../../cudarl-arena_b200/csrc/hostio.cpp"
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <dlfcn.h>
#include <map>
#include <random>
#include <string>

namespace fake {
std::mutex mu;
std::map<unsigned char*, size_t> pinned;                     // registered and allocated ranges
std::atomic<int> threads_left{1 << 30};
std::atomic<bool> no_device_pointer{false}, no_register{false}, fails{false};
std::atomic<bool> busy[2];                                  // streams 0 and 1 still at work
std::atomic<long> direct{0}, through_ring{0};                // copies from or to memory that is not pinned, and that is
std::atomic<cudaError_t> last{cudaSuccess};
cudaError_t set(cudaError_t e) { if (e != cudaSuccess && e != cudaErrorNotReady) last = e; return e; }
bool is_pinned(const void* p) {
    std::lock_guard<std::mutex> lk(mu);
    auto it = pinned.upper_bound((unsigned char*)p);
    return it != pinned.begin() && (--it, (unsigned char*)p < it->first + it->second);
}
size_t pinned_bytes() { std::lock_guard<std::mutex> lk(mu); size_t b = 0; for (auto& r : pinned) b += r.second; return b; }
}  // namespace fake

extern "C" {
cudaError_t cudaGetLastError(void) { return fake::last.exchange(cudaSuccess); }
cudaError_t cudaHostRegister(void* p, size_t n, unsigned) { if (fake::no_register) return fake::set(cudaErrorMemoryAllocation); std::lock_guard<std::mutex> lk(fake::mu); fake::pinned[(unsigned char*)p] = n; return cudaSuccess; }
cudaError_t cudaHostUnregister(void* p) { std::lock_guard<std::mutex> lk(fake::mu); return fake::pinned.erase((unsigned char*)p) ? cudaSuccess : cudaErrorHostMemoryNotRegistered; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::aligned_alloc(4096, (n + 4095) / 4096 * 4096); return cudaHostRegister(*p, n, 0); }
cudaError_t cudaFreeHost(void* p) { cudaHostUnregister(p); std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { if (fake::no_device_pointer) return fake::set(cudaErrorInvalidValue); *d = h; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t s) { return fake::busy[(size_t)s] ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { if (fake::fails) return fake::set(cudaErrorLaunchFailure); while (fake::busy[(size_t)s]) std::this_thread::yield(); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    (fake::is_pinned(kind == cudaMemcpyDeviceToHost ? d : s) ? fake::through_ring : fake::direct)++;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
    static auto real = (int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create");
    return fake::threads_left-- > 0 ? real(t, a, f, arg) : EAGAIN;
}
}

using namespace cudarl;
#define EXPECT(c) do { if (!(c)) { std::fprintf(stderr, "line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)
typedef std::vector<unsigned char> Bytes;

static Bytes noise(size_t n, unsigned seed) { Bytes b(n); std::minstd_rand r(seed + 1); for (auto& v : b) v = (unsigned char)(r() >> 7); return b; }
// Three arrays of odd lengths and places out, in, and between a stage and the caller; transitions packed on the way in.
static void round_trip(size_t total, unsigned seed) {
    const size_t n[3] = {total / 2 + seed % 7, total / 3, total - total / 2 - total / 3};
    Bytes dev[3], host[3], back[3]; Segment s[3];
    for (int k = 0; k < 3; ++k) { dev[k] = noise(n[k], seed + (unsigned)k); host[k] = Bytes(n[k] + 5, 0); s[k] = Segment{host[k].data() + k, dev[k].data(), n[k]}; }
    EXPECT(copy_out(s, 3, 0, nullptr) == cudaSuccess);
    for (int k = 0; k < 3; ++k) { EXPECT(std::memcmp(host[k].data() + k, dev[k].data(), n[k]) == 0); EXPECT(host[k][n[k] + k] == 0); back[k] = Bytes(n[k], 0); s[k].dev = back[k].data(); }
    EXPECT(copy_in(s, 3, 0, nullptr) == cudaSuccess);
    for (int k = 0; k < 3; ++k) EXPECT(back[k] == dev[k]);
    // a stage owns whole cache lines
    Bytes stage(3 * ((total + 127) / 64 * 64) + 64, 9); unsigned char* at = (unsigned char*)(((uintptr_t)stage.data() + 63) / 64 * 64);
    Segment in[3], out[3];
    for (int k = 0; k < 3; ++k) { in[k] = Segment{at, dev[k].data(), n[k]}; std::fill(host[k].begin(), host[k].end(), 0); out[k] = Segment{host[k].data() + k, at, n[k]}; at += (n[k] + 63) / 64 * 64; }
    copy_host(in, 3, true); copy_host(out, 3, false);
    for (int k = 0; k < 3; ++k) { EXPECT(std::memcmp(host[k].data() + k, dev[k].data(), n[k]) == 0); EXPECT(host[k][n[k] + k] == 0); }

    const uint32_t m = (uint32_t)(total / 12), W = 1000, H = 777;
    std::vector<int32_t> x(m), y(m), a(m), nx(m), ny(m); Bytes dn(m);
    std::minstd_rand r(seed + 1);
    for (uint32_t i = 0; i < m; ++i) { x[i] = r() % W; y[i] = r() % H; a[i] = r() % 4; nx[i] = r() % W; ny[i] = r() % H; dn[i] = r() % 3; }
    std::vector<uint32_t> p(m), q(m);
    TransitionSource src(x.data(), y.data(), a.data(), nx.data(), ny.data(), dn.data(), W, H);
    const Segment made[2] = {Segment{nullptr, p.data(), m * 4u, pack_cell_action, &src}, Segment{nullptr, q.data(), m * 4u, pack_next_cell, &src}};
    EXPECT(copy_in(made, 2, 0, nullptr) == cudaSuccess);
    EXPECT(!src.bad);
    for (uint32_t i = 0; i < m; ++i) EXPECT(p[i] == ((uint32_t)(y[i] * (int)W + x[i]) * 4u + (uint32_t)a[i] | (dn[i] ? 1u << 31 : 0u)) && q[i] == (uint32_t)ny[i] * W + (uint32_t)nx[i]);
    if (m) { ny[m - 1] = (int32_t)H; EXPECT(copy_in(made, 2, 0, nullptr) == cudaSuccess); EXPECT(src.bad); }
}
static const size_t SIZES[] = {0, 1, 1000, 70001, (256u << 10) + 3, (768u << 10) + 1, (3u << 20) + 5, (10u << 20) + 77, (90u << 20) + 1};
static void round_trips() { unsigned k = 0; for (size_t n : SIZES) round_trip(n, ++k); }

static void plain() { round_trips(); EXPECT(fake::through_ring > 0); }
// Four callers at once: one of them has the ring, the others do without.
static void callers() {
    std::vector<std::thread> t;
    for (unsigned k = 0; k < 4; ++k) t.emplace_back([k] { for (unsigned j = 0; j < 40; ++j) round_trip((j * 7919u * 4099u + k * 65537u) % (6u << 20), 1000 * k + j); });
    for (auto& u : t) u.join();
}
// No thread can be started, or only some.
static void no_threads() { fake::threads_left = 0; round_trips(); }
static void few_threads() { fake::threads_left = 3; round_trips(); fake::threads_left = 0; round_trips(); }
// A block whose device address cannot be had is not handed out, now or later.
static void stage() {
    Stage a, b;
    fake::no_device_pointer = true;
    EXPECT(stage_take(&a, 1 << 20) == cudaErrorInvalidValue);
    stage_give(&a);
    fake::no_device_pointer = false;
    EXPECT(stage_take(&b, 1 << 20) == cudaSuccess && b.host && b.dev == b.host && b.bytes == (1u << 20));
    stage_give(&b);
    EXPECT(stage_take(&a, 1 << 20) == cudaSuccess && a.host && a.dev == a.host);
    stage_give(&a);
}
// No memory can be pinned: the driver's own copies, and no error left behind for the next check.
static void no_ring() {
    fake::no_register = true;
    round_trips();
    EXPECT(fake::through_ring == 0 && cudaGetLastError() == cudaSuccess);
    fake::no_register = false;
    round_trips();
    EXPECT(fake::through_ring > 0);
}
// What the device does before a result fails: the caller's array is as it was.
static void failed_work() {
    fake::busy[0] = true; fake::fails = true;
    const Bytes before = noise((9u << 20) + 5, 3); Bytes host = before, dev(before.size(), 1);
    const Segment s{host.data(), dev.data(), host.size()};
    EXPECT(copy_out(&s, 1, 0, nullptr) == cudaErrorLaunchFailure);
    EXPECT(host == before);
    fake::busy[0] = false; fake::fails = false;
}
// While one caller waits for its stream, another has the ring.
static void long_wait() {
    const Bytes dev = noise(9u << 20, 5); Bytes a(dev.size(), 0), b(dev.size(), 0), d = dev;
    const Segment sa{a.data(), d.data(), d.size()}, sb{b.data(), d.data(), d.size()};
    fake::busy[0] = true;
    std::thread waits([&] { EXPECT(copy_out(&sa, 1, 0, (cudaStream_t)0) == cudaSuccess); });
    std::this_thread::sleep_for(std::chrono::milliseconds(200));
    EXPECT(copy_out(&sb, 1, 0, (cudaStream_t)1) == cudaSuccess);
    EXPECT(fake::through_ring > 0 && fake::direct == 0 && b == dev);
    fake::busy[0] = false;
    waits.join();
    EXPECT(fake::direct == 0 && a == dev);
}
// Values checked on their way, into a stage and through the ring: the only one out of bounds is found wherever it is.
static void bounded() {
    for (size_t n : {(size_t)1, (size_t)77, (size_t)70001, (size_t)1500003}) {
        std::vector<int32_t> v(n); std::vector<uint32_t> to((n + 31) / 16 * 16);
        std::minstd_rand r((unsigned)n);
        for (auto& u : v) u = (int32_t)(r() % 1000);
        for (int way = 0; way < 2; ++way)
            for (int32_t wrong : {0, 999, 1000, -1, INT32_MIN, INT32_MAX}) {
                const size_t at = r() % n; const int32_t was = v[at];
                v[at] = wrong;
                BoundedSource src(v.data(), 999u);
                Segment s; s.bytes = n * 4; s.fill = copy_bounded; s.arg = &src;
                if (way) { s.host = to.data(); copy_host(&s, 1, true); } else { s.dev = to.data(); EXPECT(copy_in(&s, 1, 0, nullptr) == cudaSuccess); }
                EXPECT(src.bad == (wrong < 0 || wrong > 999) && std::memcmp(to.data(), v.data(), n * 4) == 0);
                v[at] = was;
            }
    }
}

int main(int argc, char** argv) {
    const std::map<std::string, void (*)()> all = {{"plain", plain}, {"callers", callers}, {"no_threads", no_threads}, {"few_threads", few_threads}, {"stage", stage}, {"no_ring", no_ring}, {"failed_work", failed_work}, {"long_wait", long_wait}, {"bounded", bounded}};
    const auto it = argc > 1 ? all.find(argv[1]) : all.end();
    if (it == all.end()) { for (auto& s : all) std::puts(s.first.c_str()); return 2; }
    hostio_retain();
    it->second();
    hostio_release();
    EXPECT(fake::pinned_bytes() == 0);                       // all of it is given back
    return 0;
}
