// Kept streams and pinned memory, and the host <-> device copies (see hostio.h).
#include "hostio.h"

#include <cuda.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <thread>
#include <vector>

namespace b200 {
namespace {

constexpr int kMaxIdleSets = 4;        // idle stream sets kept per device
constexpr size_t kMaxKeptExecs = 16;   // executable graphs kept per set

// Staging memory: kLanes host threads, each with two pinned chunks of its own, so that a thread fills one chunk while
// the copy engine reads the other.  One thread moves pageable memory at about 10 GB/s (what a plain cudaMemcpyAsync
// reaches), the link at about 55: eight lanes fill it where the host has the cores.
constexpr int kLanes = 8;
constexpr size_t kChunk = (size_t)1 << 20;
// Measured: 188 MB of points 19 ms by a plain copy, 7 ms in lanes; at 8 MB starting the threads costs what they save.
constexpr size_t kStagedMin = kPopulateEnd;
constexpr int kMaxIdleStages = 2;                // 16 MiB of pinned memory each, kept per device

struct Stage {
    int device = -1;
    unsigned long long context = 0;
    char *mem = nullptr;               // [kLanes][2][kChunk], pinned
    cudaEvent_t ev[kLanes][2] = {};
    cudaEvent_t begin = nullptr;
    cudaStream_t io[kLanes] = {};      // copy_out: a lane waits for its own chunks only
};

std::mutex g_lock;
std::vector<StreamSet *> g_sets;       // idle
std::vector<Stage *> g_stages;         // idle

void set_destroy(StreamSet *s)
{
    for (StreamSet::KeptExec &k : s->execs) cudaGraphExecDestroy(k.exec);
    if (s->ev_fork) cudaEventDestroy(s->ev_fork);
    if (s->ev_join) cudaEventDestroy(s->ev_join);
    if (s->ev_spectrum) cudaEventDestroy(s->ev_spectrum);
    if (s->ev_spread) cudaEventDestroy(s->ev_spread);
    if (s->ev_order) cudaEventDestroy(s->ev_order);
    if (s->ev_t0) cudaEventDestroy(s->ev_t0);
    if (s->ev_t1) cudaEventDestroy(s->ev_t1);
    if (s->stream) cudaStreamDestroy(s->stream);
    if (s->stream2) cudaStreamDestroy(s->stream2);
    if (s->stream3) cudaStreamDestroy(s->stream3);
    if (s->h_state) cudaFreeHost(s->h_state);
    if (s->io) cudaFreeHost(s->io);
    delete s;
}

int set_create(StreamSet *s)
{
    B200_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    B200_CUDA(cudaStreamCreateWithFlags(&s->stream2, cudaStreamNonBlocking));
    B200_CUDA(cudaStreamCreateWithFlags(&s->stream3, cudaStreamNonBlocking));
    B200_CUDA(cudaEventCreateWithFlags(&s->ev_fork, cudaEventDisableTiming));
    B200_CUDA(cudaEventCreateWithFlags(&s->ev_join, cudaEventDisableTiming));
    B200_CUDA(cudaEventCreateWithFlags(&s->ev_spectrum, cudaEventDisableTiming));
    B200_CUDA(cudaEventCreateWithFlags(&s->ev_spread, cudaEventDisableTiming));
    B200_CUDA(cudaEventCreateWithFlags(&s->ev_order, cudaEventDisableTiming));
    B200_CUDA(cudaEventCreate(&s->ev_t0));
    B200_CUDA(cudaEventCreate(&s->ev_t1));
    B200_CUDA(cudaMallocHost((void **)&s->h_state, sizeof(IterState)));
    return 0;
}

void stage_destroy(Stage *g)
{
    for (int l = 0; l < kLanes; l++) {
        for (int k = 0; k < 2; k++)
            if (g->ev[l][k]) cudaEventDestroy(g->ev[l][k]);
        if (g->io[l]) cudaStreamDestroy(g->io[l]);
    }
    if (g->begin) cudaEventDestroy(g->begin);
    if (g->mem) cudaFreeHost(g->mem);
    delete g;
}

int stage_create(Stage *g)
{
    B200_CUDA(cudaMallocHost((void **)&g->mem, (size_t)kLanes * 2 * kChunk));
    B200_CUDA(cudaEventCreateWithFlags(&g->begin, cudaEventDisableTiming));
    for (int l = 0; l < kLanes; l++) {
        for (int k = 0; k < 2; k++) B200_CUDA(cudaEventCreateWithFlags(&g->ev[l][k], cudaEventDisableTiming));
        B200_CUDA(cudaStreamCreateWithFlags(&g->io[l], cudaStreamNonBlocking));
    }
    return 0;
}

// An idle one of this device and context, or null.  Those of a context that is gone are forgotten: their handles went
// with it.
template <class T> T *take_idle(std::vector<T *> &idle, int device, unsigned long long context)
{
    std::lock_guard<std::mutex> hold(g_lock);
    T *found = nullptr;
    for (size_t i = idle.size(); i-- > 0;) {
        T *t = idle[i];
        if (t->device != device || (found && t->context == context)) continue;
        idle.erase(idle.begin() + i);
        if (t->context == context) found = t;
        else delete t;
    }
    return found;
}

// null when it cannot be had (not an error: the caller copies without it)
Stage *stage_acquire(int device)
{
    const unsigned long long context = context_id();
    if (Stage *kept = take_idle(g_stages, device, context)) return kept;
    Stage *g = new Stage();
    g->device = device;
    g->context = context;
    if (stage_create(g) != 0) {
        stage_destroy(g);
        (void)cudaGetLastError();
        return nullptr;
    }
    return g;
}

// nothing may be in flight on it
void stage_release(Stage *g)
{
    {
        std::lock_guard<std::mutex> hold(g_lock);
        int idle = 0;
        for (Stage *o : g_stages) idle += o->device == g->device;
        if (idle < kMaxIdleStages) {
            g_stages.push_back(g);
            return;
        }
    }
    stage_destroy(g);
}

cudaMemoryType memory_type(const void *p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return cudaMemoryTypeUnregistered;
    }
    return a.type;
}

int lanes_for(size_t bytes)
{
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    return (int)std::min<size_t>(std::min<size_t>(kLanes, std::max(1u, cores / 2)), (bytes + kChunk - 1) / kChunk);
}

// runs body(lane) on `lanes` threads, this one among them; the first CUDA error wins
template <class F> cudaError_t on_lanes(int lanes, int device, F body)
{
    std::atomic<int> err{(int)cudaSuccess};
    auto run = [&](int lane) {
        cudaError_t e = lane == 0 ? cudaSuccess : cudaSetDevice(device);
        if (e == cudaSuccess) e = body(lane);
        if (e != cudaSuccess) {
            int none = (int)cudaSuccess;
            err.compare_exchange_strong(none, (int)e);
        }
    };
    std::vector<std::thread> others;
    int started = 1;
    try {
        for (; started < lanes; started++) others.emplace_back(run, started);
    } catch (const std::exception &) {
        // no more threads to be had: the lanes that did not start run here
    }
    run(0);
    for (int l = started; l < lanes; l++) run(l);
    for (std::thread &t : others) t.join();
    return (cudaError_t)err.load();
}

}  // namespace

bool pageable(const void *p) { return memory_type(p) == cudaMemoryTypeUnregistered; }

bool plain_host(const void *p)
{
    const cudaMemoryType t = memory_type(p);
    return t == cudaMemoryTypeUnregistered || t == cudaMemoryTypeHost;
}

unsigned long long context_id()
{
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static const GetId get = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &found) != cudaSuccess) {
            (void)cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<GetId>(f);
    }();
    unsigned long long id = 0;
    return get && get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

int stream_set_acquire(StreamSet **out, int device)
{
    *out = nullptr;
    B200_CUDA(cudaSetDevice(device));
    const unsigned long long context = context_id();
    *out = take_idle(g_sets, device, context);
    if (*out) return 0;
    StreamSet *s = new StreamSet();
    s->device = device;
    s->context = context;
    const int rc = set_create(s);
    if (rc != 0) {
        set_destroy(s);
        return rc;
    }
    *out = s;
    return 0;
}

bool stream_set_alive(const StreamSet *s)
{
    if (cudaSetDevice(s->device) != cudaSuccess) (void)cudaGetLastError();   // an error that stays: the handles are still valid
    return s->context == context_id();
}

float *stream_set_io(StreamSet *s)
{
    if (!s->io && cudaMallocHost((void **)&s->io, StreamSet::kIoBytes) != cudaSuccess) {
        (void)cudaGetLastError();
        s->io = nullptr;
    }
    return s->io;
}

void stream_set_release(StreamSet *s)
{
    if (!s) return;
    if (!stream_set_alive(s)) {
        delete s;
        return;
    }
    const bool fine = cudaStreamSynchronize(s->stream) == cudaSuccess && cudaStreamSynchronize(s->stream2) == cudaSuccess &&
                      cudaStreamSynchronize(s->stream3) == cudaSuccess;
    if (fine) {
        std::lock_guard<std::mutex> hold(g_lock);
        int idle = 0;
        for (StreamSet *o : g_sets) idle += o->device == s->device;
        if (idle < kMaxIdleSets) {
            g_sets.push_back(s);
            return;
        }
    }
    set_destroy(s);
}

cudaGraphExec_t graph_exec_acquire(StreamSet *s, cudaGraph_t graph, unsigned long long shape)
{
    for (size_t i = s->execs.size(); i-- > 0;) {
        if (s->execs[i].shape != shape) continue;
        cudaGraphExec_t exec = s->execs[i].exec;
        s->execs.erase(s->execs.begin() + i);
        cudaGraphExecUpdateResultInfo info;
        if (cudaGraphExecUpdate(exec, graph, &info) == cudaSuccess) return exec;
        (void)cudaGetLastError();
        cudaGraphExecDestroy(exec);   // other nodes after all (another attractive kernel, say)
    }
    cudaGraphExec_t exec = nullptr;
    if (cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return exec;
}

bool graph_exec_kept(const StreamSet *s, unsigned long long shape)
{
    for (const auto &e : s->execs)
        if (e.shape == shape) return true;
    return false;
}

void graph_exec_release(StreamSet *s, cudaGraphExec_t exec, unsigned long long shape)
{
    if (!s) {
        cudaGraphExecDestroy(exec);
        return;
    }
    // The one that was used longest ago makes room: a new one takes 2 to 3 ms (16 iterations), and a program that goes on with
    // what it does now would pay that in each of its sessions.
    if (s->execs.size() >= kMaxKeptExecs) {
        cudaGraphExecDestroy(s->execs.front().exec);
        s->execs.erase(s->execs.begin());
    }
    s->execs.push_back({exec, shape});
}

int copy_in(void *dst, const void *src, size_t bytes, cudaStream_t st)
{
    if (bytes == 0) return 0;
    Stage *g = nullptr;
    int device = 0;
    B200_CUDA(cudaGetDevice(&device));
    if (bytes >= kStagedMin && lanes_for(bytes) > 1 && pageable(src)) g = stage_acquire(device);
    if (!g) {
        B200_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        return 0;
    }
    const int lanes = lanes_for(bytes);
    const size_t chunks = (bytes + kChunk - 1) / kChunk;
    cudaError_t e = on_lanes(lanes, device, [&](int lane) -> cudaError_t {
        int k = 0;
        size_t done = 0;
        for (size_t c = lane; c < chunks; c += lanes, k ^= 1, done++) {
            char *slot = g->mem + ((size_t)lane * 2 + k) * kChunk;
            if (done >= 2) {   // the copy engine is done with this slot
                const cudaError_t w = cudaEventSynchronize(g->ev[lane][k]);
                if (w != cudaSuccess) return w;
            }
            const size_t n = std::min(kChunk, bytes - c * kChunk);
            memcpy(slot, static_cast<const char *>(src) + c * kChunk, n);
            cudaError_t r = cudaMemcpyAsync(static_cast<char *>(dst) + c * kChunk, slot, n, cudaMemcpyHostToDevice, st);
            if (r == cudaSuccess) r = cudaEventRecord(g->ev[lane][k], st);
            if (r != cudaSuccess) return r;
        }
        return cudaSuccess;
    });
    // the last chunks are still on their way: the staging memory must not be reused before they have left
    const cudaError_t w = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = w;
    stage_release(g);
    B200_CUDA(e);
    return 0;
}

int copy_out(void *dst, const void *src, size_t bytes, cudaStream_t st)
{
    if (bytes == 0) return 0;
    Stage *g = nullptr;
    int device = 0;
    B200_CUDA(cudaGetDevice(&device));
    if (bytes >= kStagedMin && lanes_for(bytes) > 1 && pageable(dst)) g = stage_acquire(device);
    if (!g) {
        B200_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        B200_CUDA(cudaStreamSynchronize(st));
        return 0;
    }
    const int lanes = lanes_for(bytes);
    const size_t chunks = (bytes + kChunk - 1) / kChunk;
    cudaError_t e = cudaEventRecord(g->begin, st);   // the data is complete once the stream reaches this
    if (e == cudaSuccess)
        e = on_lanes(lanes, device, [&](int lane) -> cudaError_t {
            cudaStream_t io = g->io[lane];
            cudaError_t r = cudaStreamWaitEvent(io, g->begin, 0);
            auto fetch = [&](size_t c, int k) {
                const size_t n = std::min(kChunk, bytes - c * kChunk);
                cudaError_t f = cudaMemcpyAsync(g->mem + ((size_t)lane * 2 + k) * kChunk, static_cast<const char *>(src) + c * kChunk, n,
                                                cudaMemcpyDeviceToHost, io);
                return f == cudaSuccess ? cudaEventRecord(g->ev[lane][k], io) : f;
            };
            if (r == cudaSuccess) r = fetch(lane, 0);
            int k = 0;
            for (size_t c = lane; r == cudaSuccess && c < chunks; c += lanes, k ^= 1) {
                if (c + lanes < chunks) r = fetch(c + lanes, k ^ 1);
                if (r == cudaSuccess) r = cudaEventSynchronize(g->ev[lane][k]);
                if (r == cudaSuccess)
                    memcpy(static_cast<char *>(dst) + c * kChunk, g->mem + ((size_t)lane * 2 + k) * kChunk, std::min(kChunk, bytes - c * kChunk));
            }
            const cudaError_t w = cudaStreamSynchronize(io);
            return r == cudaSuccess ? w : r;
        });
    const cudaError_t w = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = w;
    stage_release(g);
    B200_CUDA(e);
    return 0;
}

void host_pools_release(int device)
{
    const unsigned long long context = context_id();
    while (StreamSet *s = take_idle(g_sets, device, context)) set_destroy(s);
    while (Stage *g = take_idle(g_stages, device, context)) stage_destroy(g);
}

}  // namespace b200
