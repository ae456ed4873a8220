// hostio.h -- moving caller memory to and from the device.
//
// Caller buffers are pageable, and a copy the driver makes from or to pageable memory runs at the speed of ONE core copying (and, into
// a freshly allocated array, faulting its pages in): 268 MB came back at 4.8 GB/s, with the link at 56 GB/s.  Here large copies go
// through a ring of pinned slots: the copy engine fills a slot while several cores empty others.
//
// The ring, its worker threads and the pinned blocks below belong to the process, are shared by its contexts, bounded in size, and
// given back when the last context goes.  Every function may be called from several threads at once.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <cstddef>
#include <cstdint>

namespace cudarl {

// One array of a copy.  With `fill`, the bytes on their way to the device do not lie in the caller's memory: fill(dst, first, bytes, arg)
// makes `bytes` of them from offset `first` on (both multiples of 4), called from several threads for different parts.
typedef void (*Fill)(void* dst, size_t first, size_t bytes, const void* arg);
struct Segment { void* host; void* dev; size_t bytes; Fill fill = nullptr; const void* arg = nullptr; };

// One pinned block mapped into the device, for the small results and inputs of a context.
struct Stage { unsigned char* host = nullptr; unsigned char* dev = nullptr; size_t bytes = 0; };

// Fills for the transitions of an update_batch: one word each, checked (`bad`: one was outside the grid or the action set).
struct TransitionSource {
    const int32_t *sx, *sy, *a, *nx, *ny; const uint8_t* dn; uint32_t W, H;
    std::atomic<bool> bad{false};
    TransitionSource(const int32_t* sx_, const int32_t* sy_, const int32_t* a_, const int32_t* nx_, const int32_t* ny_, const uint8_t* dn_, uint32_t W_, uint32_t H_)
        : sx(sx_), sy(sy_), a(a_), nx(nx_), ny(ny_), dn(dn_), W(W_), H(H_) {}
};
void pack_cell_action(void* dst, size_t first, size_t bytes, const void* source);      // cell * 4 + action, bit 31 = the episode ended there
void pack_next_cell(void* dst, size_t first, size_t bytes, const void* source);

// Values of 0 .. most, checked on the way (`bad`: one was not).
struct BoundedSource {
    const int32_t* from; uint32_t most;
    std::atomic<bool> bad{false};
    BoundedSource(const int32_t* from_, uint32_t most_) : from(from_), most(most_) {}
};
void copy_bounded(void* dst, size_t first, size_t bytes, const void* source);

void hostio_retain();                         // one per context: keeps the process-wide parts alive
void hostio_release();
cudaError_t stage_take(Stage* s, size_t bytes);      // zeroed first 256 bytes
void stage_give(Stage* s);

// Device -> host: everything enqueued on `st` before has been waited for and the data is in the caller's arrays on return.
cudaError_t copy_out(const Segment* segs, int n, int device, cudaStream_t st);
// Host -> device, ordered on `st`: the caller's arrays may be reused on return.
cudaError_t copy_in(const Segment* segs, int n, int device, cudaStream_t st);

// Between a stage and the caller: `dev` is the source, `host` the destination, both host memory; into_stage: the device reads it next, and the destination owns its
// cache lines to the end of the last one.
void copy_host(const Segment* segs, int n, bool into_stage);

}  // namespace cudarl
