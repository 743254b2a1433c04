// Host-side resources that outlive one call: streams, events and pinned memory, and the copies between pageable host
// memory and the device that use them.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <vector>

#include "common.cuh"
#include "pages.h"

namespace b200 {

// Which context of the current device this is: another one after cudaDeviceReset, which takes streams, events, pinned
// memory, executables and function attributes with it (a stale handle is not refused but crashes).  0: cannot be told.
unsigned long long context_id();

// What a session or a stage call needs from the driver besides device memory.  Creating and destroying it costs one to
// three milliseconds a time, and on a busy host single calls (pinned memory above all) stall for 0.1 to 1.2 s, so the
// sets are kept per device and handed to the next caller: at most kMaxIdleSets idle ones,
// b200tsne_release_cached_memory() gives them back.  Safe from several threads: a set has one user at a time.
struct StreamSet {
    int device = -1;
    unsigned long long context = 0;   // its handles are of this context
    cudaStream_t stream = nullptr, stream2 = nullptr, stream3 = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_spectrum = nullptr, ev_spread = nullptr, ev_order = nullptr, ev_t0 = nullptr, ev_t1 = nullptr;
    IterState *h_state = nullptr;   // pinned
    // Pinned memory that kernels read and write across the bus: the state of a small map in one piece (Session::small_state).
    // The size bounds what is held pinned; it is no crossover (21,845 points, the most that it holds: state in, one iteration,
    // state out 278 -> 168 us).  Made at first use: 20 us, but 1.2 ms where the driver has to pin a new block for it.
    static constexpr size_t kIoBytes = (size_t)512 << 10;
    float *io = nullptr;
    // Executable graphs that finished sessions left behind.  Instantiating one of 16 iterations takes 1.3 ms (now and
    // then 100 on a busy host) and destroying it another; updating one of the same shape takes 0.1 ms.  They hold stale
    // addresses and are only launched after an update.
    struct KeptExec {
        cudaGraphExec_t exec;
        unsigned long long shape;
    };
    std::vector<KeptExec> execs;
};
int stream_set_acquire(StreamSet **out, int device);   // makes `device` current
void stream_set_release(StreamSet *s);                 // waits for its streams; null is fine
float *stream_set_io(StreamSet *s);                    // `io`; null when it cannot be had
bool stream_set_alive(const StreamSet *s);             // its context still is the device's; makes the device current

// An executable for `graph`: a kept one of the same shape, updated, else a new one; null if neither can be had.
cudaGraphExec_t graph_exec_acquire(StreamSet *s, cudaGraph_t graph, unsigned long long shape);
bool graph_exec_kept(const StreamSet *s, unsigned long long shape);   // one of that shape waits to be updated
void graph_exec_release(StreamSet *s, cudaGraphExec_t exec, unsigned long long shape);

// Copies between pageable host memory and the device on `st`.  Large ones go through pinned chunks filled (or emptied)
// by several host threads; small ones, pinned memory and callers that cannot have staging memory use one
// cudaMemcpyAsync.  copy_in returns once a pageable source may be changed (pinned memory is read until the stream has
// passed the copy); copy_out returns with the data in place.
int copy_in(void *dst_device, const void *src_host, size_t bytes, cudaStream_t st);
int copy_out(void *dst_host, const void *src_device, size_t bytes, cudaStream_t st);

bool pageable(const void *p);     // host memory that CUDA knows nothing of
bool plain_host(const void *p);   // host memory, pinned or not: neither device nor managed memory, which a copy takes as well

void host_pools_release(int device);   // idle sets and staging memory of one device

}  // namespace b200
