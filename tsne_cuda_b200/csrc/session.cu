// Host orchestration of the device-resident FIt-SNE state: allocation, the set-up pipeline from
// points to affinities, and the gradient loop (reference: the body of tsnecuda::RunTsne,
// src/fit_tsne.cu:84-166 for the set-up and :402-580 for the loop).
//
// One iteration on one GPU is seven kernels (one more in a large map, three more where the spread order is refreshed) and no
// host synchronisation:
//   stream  : [order x3] -> spread -> FFT rows -> FFT columns -> FFT rows^-1 --> update (interpolates the repulsive force)
//   stream2 : clear forces -> attractive ---------------------------------------^
//   stream3 : kernel spectrum of a large map -> (FFT rows); the spread's launch has a small map's
// A sharded run, and one whose stages are timed, gathers the repulsive force in a kernel of its own before the update.
// The embedding's min/max and the normalisation sum travel between kernels in device memory
// (IterState), so the two per-iteration host round trips of the reference do not exist.
// A sharded run adds two meetings of the ranks per iteration and exchanges over peer memory
// (peer.h): spread -> meet -> sum of the partial grids -> FFT ... update into every rank -> meet.
#include "session.h"

#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <string>

#include "comm.h"
#include "hostio.h"
#include "peer.h"

namespace b200 {

// ---- error plumbing -------------------------------------------------------------------------
static thread_local std::string g_last_error;
void set_error(const std::string &msg) { g_last_error = msg; }
const std::string &last_error() { return g_last_error; }
int cuda_fail(cudaError_t e, const char *what, const char *file, int line)
{
    g_last_error = std::string("CUDA error '") + cudaGetErrorString(e) + "' in " + what + " at " + file + ":" +
                   std::to_string(line);
    return -2;
}

// ---- arena ------------------------------------------------------------------------------------
// Device memory comes from the device's default stream-ordered pool with the release threshold lifted, so
// what one call frees the next call gets back without a trip to the driver (a fit allocates and frees
// about 5 GB at N = 10^6; cudaMalloc/cudaFree of that cost tens of milliseconds per call).  Every arena
// is released only after the streams that used its memory have been synchronised, so the memory may be
// handed to any stream afterwards.  b200tsne_release_cached_memory() returns the pool to the driver.
static int configure_pool()
{
    static std::atomic<unsigned long long> done[64];   // the context (plus one) that it was done in
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    const unsigned long long context = context_id() + 1;
    if (dev < 0 || dev >= 64 || done[dev].load(std::memory_order_relaxed) == context) return 0;
    cudaMemPool_t pool;
    B200_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
    unsigned long long keep = ~0ull;
    B200_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    done[dev].store(context, std::memory_order_relaxed);
    return 0;
}

int release_cached_memory()
{
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    cudaMemPool_t pool;
    B200_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
    B200_CUDA(cudaDeviceSynchronize());
    host_pools_release(dev);
    B200_CUDA(cudaMemPoolTrimTo(pool, 0));
    return 0;
}

DeviceArena::~DeviceArena() { release(); }
int DeviceArena::alloc(void **p, size_t bytes)
{
    *p = nullptr;
    if (bytes == 0) bytes = 16;
    B200_TRY(configure_pool());
    B200_CUDA(cudaMallocAsync(p, bytes, cudaStreamPerThread));
    ptrs.push_back(*p);
    // B200TSNE_POISON=1 fills every new allocation with 0xFF bytes (NaN floats, -1 ints): pooled memory is not
    // zero like fresh device memory often is, and this makes any read of memory the library has not written
    // show up at once (the GPU suite passes with it)
    static const bool poison = getenv("B200TSNE_POISON") && atoi(getenv("B200TSNE_POISON")) != 0;
    if (poison) {
        B200_CUDA(cudaMemsetAsync(*p, 0xff, bytes, cudaStreamPerThread));
        B200_CUDA(cudaStreamSynchronize(cudaStreamPerThread));
    }
    return 0;
}
void DeviceArena::forget()
{
    consumers.clear();
    ptrs.clear();
}
void DeviceArena::release()
{
    // also on error paths, where kernels queued on a consumer stream may still be running
    if (!ptrs.empty())
        for (cudaStream_t st : consumers) cudaStreamSynchronize(st);
    consumers.clear();
    for (void *p : ptrs) cudaFreeAsync(p, cudaStreamPerThread);
    if (!ptrs.empty()) cudaStreamSynchronize(cudaStreamPerThread);
    ptrs.clear();
}

// ---- session ------------------------------------------------------------------------------------
int Session::init(int64_t N_, int K_, int64_t lo, int64_t hi, int device_)
{
    if (N_ <= 0 || K_ <= 0 || lo < 0 || hi > N_ || lo > hi) { set_error("session: invalid sizes"); return -1; }
    if (N_ >= (int64_t)1 << 31) { set_error("session: more than 2^31-1 points are not supported (int32 ids)"); return -4; }
    N = N_; K = K_; row_lo = lo; row_hi = hi; device = device_;
    B200_CUDA(cudaSetDevice(device));
    // (Stream priorities were measured both ways and change nothing: the attractive kernel and the grid
    // pipeline compete for the same load/store units rather than for block slots.)
    B200_TRY(stream_set_acquire(&host, device));
    stream = host->stream; stream2 = host->stream2; stream3 = host->stream3;
    ev_fork = host->ev_fork; ev_join = host->ev_join; ev_spectrum = host->ev_spectrum; ev_spread = host->ev_spread; ev_order = host->ev_order; ev_t0 = host->ev_t0; ev_t1 = host->ev_t1;
    h_state = host->h_state;
    arena.serve(stream);
    arena.serve(stream2);
    arena.serve(stream3);
    blocked_arena.serve(stream);
    blocked_arena.serve(stream2);
    // Y2 and the force arrays are padded so that an in-place all-gather over up to 16 ranks fits
    const int64_t npad = N + 16;
    const int64_t r = std::max<int64_t>(rows(), 1);
    B200_TRY(arena.alloc((void **)&P, sizeof(float) * r * K));
    B200_TRY(arena.alloc((void **)&ids, sizeof(int32_t) * r * K));
    B200_TRY(arena.alloc((void **)&order, sizeof(int32_t) * r));
    B200_TRY(arena.alloc((void **)&order_alt, sizeof(int32_t) * r));
    B200_TRY(arena.alloc((void **)&order_keys, sizeof(int32_t) * r));
    B200_TRY(arena.alloc((void **)&box_hist, sizeof(int32_t) * kBoxes * kBoxes));
    B200_TRY(launch_order_identity(order, rows(), stream));
    B200_CUDA(cudaMemsetAsync(box_hist, 0, sizeof(int32_t) * kBoxes * kBoxes, stream));
    if (rows() < kSortMin) order_refresh = 0;
    order_refresh_early = rows() >= kSortEachFrom ? 1 : rows() >= kSortMin ? 4 : rows() >= kSortEarlyMin ? 8 : 0;
    bool never = false;
    if (const char *e = getenv("B200TSNE_ORDER_REFRESH")) {
        order_refresh = std::max(0, atoi(e));
        never = order_refresh == 0;
        order_refresh_early = std::max(1, order_refresh_early);
    }
    if (const char *e = getenv("B200TSNE_ORDER_REFRESH_EARLY")) order_refresh_early = order_refresh_early_sharded = std::max(1, atoi(e));
    if (never) order_refresh_early = 0;
    if (order_refresh == 0) order_refresh_early_sharded = 0;   // ranks sort in both phases or in neither
    if (const char *e = getenv("B200TSNE_GRAPHS")) use_graphs = atoi(e) != 0;
    B200_TRY(arena.alloc((void **)&Y2, sizeof(float2) * npad));
    B200_TRY(arena.alloc((void **)&Fattr, sizeof(float2) * npad));
    B200_TRY(arena.alloc((void **)&Frep, sizeof(float2) * npad));
    B200_TRY(arena.alloc((void **)&gains, sizeof(float2) * r));
    B200_TRY(arena.alloc((void **)&u, sizeof(float2) * r));
    B200_TRY(arena.alloc((void **)&soa_tmp, sizeof(float) * 2 * N));
    B200_TRY(arena.alloc((void **)&w, sizeof(float4) * kG * kG));
    B200_TRY(arena.alloc((void **)&ytilde, sizeof(float4) * kG * kG));
    B200_TRY(arena.alloc(&fft_mem, fft_workspace_bytes()));
    B200_TRY(arena.alloc((void **)&state, sizeof(IterState)));
    B200_TRY(fft_workspace_init(&fft, fft_mem, stream));
    Y2_own = Y2;
    w_own = w;
    ic = make_interp_consts();
    B200_CUDA(cudaMemsetAsync(w, 0, sizeof(float4) * kG * kG, stream));
    B200_CUDA(cudaMemsetAsync(Y2, 0, sizeof(float2) * npad, stream));
    B200_CUDA(cudaMemsetAsync(Fattr, 0, sizeof(float2) * npad, stream));
    B200_CUDA(cudaMemsetAsync(Frep, 0, sizeof(float2) * npad, stream));
    B200_TRY(launch_state_reset(state, stream));
    B200_TRY(launch_fill(reinterpret_cast<float *>(gains), 1.0f, 2 * r, stream));
    B200_CUDA(cudaMemsetAsync(u, 0, sizeof(float2) * r, stream));
    B200_CUDA(cudaStreamSynchronize(stream));
    return 0;
}

void Session::destroy()
{
    cudaSetDevice(device);
    if (host && !stream_set_alive(host)) {   // the device was reset: memory, streams and executables are gone already
        graphs.clear();
        blocked_arena.forget();
        arena.forget();
        stream = stream2 = stream3 = nullptr;
    }
    if (stream) cudaStreamSynchronize(stream);
    if (stream2) cudaStreamSynchronize(stream2);
    if (stream3) cudaStreamSynchronize(stream3);
    drop_graphs();
    if (px) { peer_exchange_release(px, comm); px = nullptr; }
    comm = nullptr;  // owned by the communicator cache (comm.h)
    blocked.clear();
    blocked_arena.release();
    arena.release();
    stream_set_release(host);
    host = nullptr;
    h_state = nullptr; stream = stream2 = stream3 = nullptr; ev_fork = ev_join = ev_spectrum = ev_spread = ev_order = ev_t0 = ev_t1 = nullptr;
}

int Session::set_embedding_soa(const float *Y_host, bool reset)
{
    B200_CUDA(cudaSetDevice(device));
    B200_TRY(copy_in(soa_tmp, Y_host, sizeof(float) * 2 * N, stream));
    B200_TRY(launch_soa_to_aos(soa_tmp, Y2, N, stream, state_order()));
    if (reset) {
        const int64_t r = std::max<int64_t>(rows(), 1);
        B200_TRY(launch_fill(reinterpret_cast<float *>(gains), 1.0f, 2 * r, stream));
        B200_CUDA(cudaMemsetAsync(u, 0, sizeof(float2) * r, stream));
        step = 0;
    }
    B200_TRY(launch_state_reset(state, stream));
    done_seen = 0;
    B200_TRY(launch_minmax_init(Y2, N, state, step & 1, stream));
    B200_CUDA(cudaMemsetAsync(w, 0, sizeof(float4) * kG * kG, stream));
    B200_CUDA(cudaStreamSynchronize(stream));
    launches += 4;
    return 0;
}

int Session::get_embedding_soa(float *Y_host)
{
    B200_CUDA(cudaSetDevice(device));
    B200_TRY(launch_aos_to_soa(Y2, soa_tmp, N, stream, state_order()));
    B200_TRY(copy_out(Y_host, soa_tmp, sizeof(float) * 2 * N, stream));
    launches += 1;
    return 0;
}

int Session::get_optimizer_soa(float *momentum_host, float *gains_host)
{
    B200_CUDA(cudaSetDevice(device));
    const int64_t r = rows();
    if (r == 0) return 0;
    if (momentum_host) {
        B200_TRY(launch_aos_to_soa(u, soa_tmp, r, stream, state_order()));
        B200_TRY(copy_out(momentum_host, soa_tmp, sizeof(float) * 2 * r, stream));
    }
    if (gains_host) {
        B200_TRY(launch_aos_to_soa(gains, soa_tmp, r, stream, state_order()));
        B200_TRY(copy_out(gains_host, soa_tmp, sizeof(float) * 2 * r, stream));
    }
    return 0;
}

int Session::set_optimizer_soa(const float *momentum_host, const float *gains_host)
{
    B200_CUDA(cudaSetDevice(device));
    const int64_t r = rows();
    if (r == 0) return 0;
    if (momentum_host) {
        B200_TRY(copy_in(soa_tmp, momentum_host, sizeof(float) * 2 * r, stream));
        B200_TRY(launch_soa_to_aos(soa_tmp, u, r, stream, state_order()));
        B200_CUDA(cudaStreamSynchronize(stream));
    }
    if (gains_host) {
        B200_TRY(copy_in(soa_tmp, gains_host, sizeof(float) * 2 * r, stream));
        B200_TRY(launch_soa_to_aos(soa_tmp, gains, r, stream, state_order()));
        B200_CUDA(cudaStreamSynchronize(stream));
    }
    return 0;
}

// (the order of the points does not matter at these sizes, so the state is in the caller's)
static_assert(StreamSet::kIoBytes / (6 * sizeof(float)) <= (size_t)kAttractiveTile, "a state in one piece is in natural order");

bool Session::small_state(const void *Y, const void *momentum, const void *gains) const
{
    if (rows() != N || (comm && comm->world > 1) || sizeof(float) * 6 * (size_t)N > StreamSet::kIoBytes) return false;
    for (const void *p : {Y, momentum, gains})
        if (p && !plain_host(p)) return false;
    return stream_set_io(host) != nullptr;
}

int Session::set_small_state(const float *Y_host, const float *momentum_host, const float *gains_host, int at_step)
{
    B200_CUDA(cudaSetDevice(device));
    const size_t block = 2 * (size_t)N;
    memcpy(host->io, Y_host, sizeof(float) * block);
    memcpy(host->io + block, momentum_host, sizeof(float) * block);
    memcpy(host->io + 2 * block, gains_host, sizeof(float) * block);
    step = at_step;
    done_seen = 0;
    B200_TRY(launch_state_reset(state, stream));
    B200_TRY(launch_load_state(host->io, Y2, u, gains, N, state, step & 1, stream));
    B200_CUDA(cudaMemsetAsync(w, 0, sizeof(float4) * kG * kG, stream));
    // like the copying path: the call's work and its errors are its own (left queued, 8 us of a set_state, run(1), get_state
    // of 110 moved into the next call), and the pinned memory is free for the next state
    B200_CUDA(cudaStreamSynchronize(stream));
    launches += 2;
    return 0;
}

// null arrays are not asked for
int Session::get_small_state(float *Y_host, float *momentum_host, float *gains_host)
{
    B200_CUDA(cudaSetDevice(device));
    B200_TRY(launch_store_state(Y_host ? Y2 : nullptr, momentum_host ? u : nullptr, gains_host ? gains : nullptr, host->io, N, stream));
    B200_CUDA(cudaStreamSynchronize(stream));
    const size_t block = 2 * (size_t)N;
    float *to[3] = {Y_host, momentum_host, gains_host};
    for (int k = 0; k < 3; k++)
        if (to[k]) memcpy(to[k], host->io + k * block, sizeof(float) * block);
    launches += 1;
    return 0;
}

namespace {
// Times the stages of one iteration when stage timers are on (serialised on one stream).
struct StageClock {
    Session *s;
    cudaEvent_t a = nullptr, b = nullptr;
    explicit StageClock(Session *s_) : s(s_)
    {
        if (s->stage_timers) { cudaEventCreate(&a); cudaEventCreate(&b); }
    }
    ~StageClock()
    {
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    }
    void begin(cudaStream_t st) { if (a) cudaEventRecord(a, st); }
    void end(cudaStream_t st, int stage, int n_launches)
    {
        s->launches += n_launches;
        if (!a) return;
        s->stage_launches[stage] += n_launches;
        cudaEventRecord(b, st);
        cudaEventSynchronize(b);
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, a, b);
        s->stage_ms[stage] += ms;
    }
};
}  // namespace

// norm_mode, stop_norm: see launch_update
int Session::one_iteration(int norm_mode, float stop_norm, bool sorts)
{
    const int slot = step & 1;
    const bool late = step >= force_magnify_iters;
    const float momentum = late ? post_momentum : pre_momentum;
    const float exag = late ? 1.0f : exaggeration;
    const bool multi = comm && comm->world > 1;
    const bool p2p = multi && px != nullptr;   // exchanges over peer memory instead of collectives
    StageClock clk(this);
    cudaStream_t sa = stage_timers ? stream : stream2;  // attractive stream
    const bool spectrum_in_spread = !stage_timers && spread_takes_spectrum(rows());
    if (p2p) {
        // the grid buffer of the next iteration: the peers finished reading it before they signalled the
        // update this rank waited for at the end of the previous iteration
        B200_CUDA(cudaMemsetAsync(px->w_local(px->parity ^ 1), 0, sizeof(float4) * kG * kG, stream));
    }

    // The attractive kernel and the grid pipeline run side by side and divide the SMs between them (blocks_beside_grid), so a
    // large iteration is bound by the SM time of its kernels: at N = 10^6, settled, the update 32 us and the spread 20 on all
    // SMs, then 170 us of the attractive kernel beside the rest of the pipeline.  A higher stream priority for the attractive
    // kernel changed nothing.
    // An L2 evict-first policy on the attractive kernel's stream loads: +0.8 %, not kept.
    if (!stage_timers) {
        B200_CUDA(cudaEventRecord(ev_fork, stream));
        B200_CUDA(cudaStreamWaitEvent(stream2, ev_fork, 0));
        B200_TRY(attractive(sa));
        B200_CUDA(cudaEventRecord(ev_join, stream2));
        launches += attractive_launches();
        // The kernel's spectrum needs the bounding box only, like the attractive force, so the two start together: in front of
        // that force it delays it by 13 us (10^6 points, exaggerated / settled: 249 / 249 us an iteration, beside it 235 / 240).
        // Small maps have it in the spread's launch.
        if (!spectrum_in_spread) {
            B200_CUDA(cudaStreamWaitEvent(stream3, ev_fork, 0));
            B200_TRY(launch_kernel_spectrum(state, slot, fft, stream3));
            B200_CUDA(cudaEventRecord(ev_spectrum, stream3));
            launches += 1;
        }
    }

    // The embedding reshuffles quickly while it is being exaggerated and slowly afterwards, and a large one pays more for boxes
    // that are mixed up than for a sort: more than kSortEachFrom points are sorted in every iteration early, fewer every
    // fourth or eighth, and every eighth later (below kSortMin points not at all).  An iteration while exaggerated, from a
    // blob / from a blob with a learning rate of n / 12 / from a layout:
    //     points      natural order        every 8th            every 4th            every one (on the chain)
    //     3,000       26.4 / 26.8 / 27.4   26.2 / 26.2 / 26.1
    //     5,000       29.0 / 28.5 / 30.0   26.9 / 26.6 / 26.7
    //     20,011      39.6 / 40.0 / 43.0   30.2 / 32.1 / 29.2   30.3 / 32.3 / 29.3
    //     60,000      38.8 / 38.8 / 33.8   37.2 / 40.5 / 35.1   36.6 / 39.8 / 34.4   44.4 / 44.6 / 44.2
    //     90,000                                                48.9 / 57.2 / 41.3   47.7 / 48.9 / 48.7
    //     130,000                                               59.4 / 73.3 / 50.6   53.3 / 56.0 / 55.7
    //     200,000     102 / 93 / 67        73.7 / 92.7 / 63.2   71.9 / 93.0 / 62.8   63.3 / 63.5 / 63.6
    // (Sorting the rows for iteration t + 1
    // at the end of iteration t, while waiting for the other ranks, was measured on two GPUs: the next bounding box is only
    // known after that meeting, and boxes taken from the previous one - the embedding grows by more than a box
    // width per exaggerated iteration - break the runs of equal boxes: spread 61 us instead of 15.)
    const int refresh = refresh_period(step);
    // An order that is to serve several iterations may as well be one older: its sort is then off the chain, beside it.
    const bool sorts_beside = sorts && refresh > 1 && !multi && !stage_timers;
    if (sorts && !sorts_beside) {
        clk.begin(stream);
        B200_TRY(launch_order_count(Y2, row_lo, row_hi, order, order_alt, order_keys, box_hist, state, slot, stream));
        B200_TRY(launch_order_scatter(rows(), order, order_alt, order_keys, box_hist, stream));
        clk.end(stream, kStOrder, 3);
    }
    clk.begin(stream);
    B200_TRY(launch_spread(Y2, row_lo, row_hi, refresh > 0 ? order : nullptr, sorts && !sorts_beside ? box_hist : nullptr, state, slot, ic, w,
                           spectrum_in_spread ? &fft : nullptr, stream));
    clk.end(stream, kStSpread, 1);
    if (sorts_beside) {
        B200_CUDA(cudaEventRecord(ev_spread, stream));
        B200_CUDA(cudaStreamWaitEvent(stream3, ev_fork, 0));
        B200_TRY(launch_order_count(Y2, row_lo, row_hi, order, order_alt, order_keys, box_hist, state, slot, stream3));
        B200_CUDA(cudaStreamWaitEvent(stream3, ev_spread, 0));   // it reads the order
        B200_TRY(launch_order_scatter(rows(), order, order_alt, order_keys, box_hist, stream3));
        B200_CUDA(cudaMemsetAsync(box_hist, 0, sizeof(int32_t) * kBoxes * kBoxes, stream3));
        B200_CUDA(cudaEventRecord(ev_order, stream3));
        launches += 3;
    }
    if (p2p) {
        clk.begin(stream);
        if (grid_two_shot) {
            B200_TRY(launch_peer_grid_allreduce(px, px->parity, stream));
            clk.end(stream, kStExchange, 1);
        } else {
            B200_TRY(launch_peer_barrier(px, kFlagSpread, nullptr, 0, stream));
            B200_TRY(launch_peer_grid_reduce(px, px->parity, w_sum, stream));
            clk.end(stream, kStExchange, 2);
        }
    } else if (multi) {
        clk.begin(stream);
        B200_TRY(comm->all_reduce_sum_f32(reinterpret_cast<float *>(w), (size_t)kG * kG * 4, stream));
        clk.end(stream, kStExchange, 0);
    }
    clk.begin(stream);
    float4 *charges = p2p ? w_sum : w;
    if (stage_timers) B200_TRY(launch_kernel_spectrum(state, slot, fft, stream));
    else if (!spectrum_in_spread) B200_CUDA(cudaStreamWaitEvent(stream, ev_spectrum, 0));
    B200_TRY(launch_convolve_rows(charges, state, slot, fft, stream));
    int free_sms = 0;
    if (!multi) B200_TRY(free_beside_attractive(blocked, beside_attractive(), &free_sms));
    B200_TRY(launch_convolve(charges, ytilde, state, slot, fft, !p2p, free_sms, stream));   // sums Z over ALL points on the grid: no exchange
    clk.end(stream, kStConvolve, stage_timers ? 4 : 3);
    const bool fused = !multi && !stage_timers;   // the update interpolates the repulsive force itself
    if (!fused) {
        clk.begin(stream);
        B200_TRY(launch_gather(Y2, row_lo, row_hi, state, slot, ic, ytilde, Frep, stream));
        clk.end(stream, kStGather, 1);
    }
    if (stage_timers) {
        clk.begin(stream);
        B200_TRY(attractive(stream));
        clk.end(stream, kStAttractive, attractive_launches());
    } else {
        B200_CUDA(cudaStreamWaitEvent(stream, ev_join, 0));
        if (sorts_beside) B200_CUDA(cudaStreamWaitEvent(stream, ev_order, 0));
    }
    clk.begin(stream);
    UpdateTargets dst;
    dst.n = 1;
    dst.p[0] = Y2;
    if (p2p) {   // the new rows go straight into the next embedding buffer of every rank
        dst.n = comm->world;
        for (int r = 0; r < comm->world; r++) dst.p[r] = px->tab.y[px->parity ^ 1][r];
    }
    B200_TRY(launch_update(Y2, dst, Fattr, Frep, fused ? ytilde : nullptr, ic, gains, u, N, row_lo, row_hi, state, slot, eta, momentum, exag,
                           norm_mode, stop_norm, stream));
    clk.end(stream, kStUpdate, 1);
    if (p2p) {
        clk.begin(stream);
        // the update kernel left this rank's min/max in slot^1; the meeting makes them global
        B200_TRY(launch_peer_barrier(px, kFlagUpdate, state, slot ^ 1, stream));
        px->parity ^= 1;
        Y2 = px->y_local(px->parity);
        w = px->w_local(px->parity);
        clk.end(stream, kStExchange, 1);
    } else if (multi) {
        clk.begin(stream);
        const int64_t chunk = (N + comm->world - 1) / comm->world;
        B200_TRY(comm->all_gather_inplace(Y2, sizeof(float2) * (size_t)chunk, stream));
        B200_TRY(launch_minmax_init(Y2, N, state, slot ^ 1, stream));
        clk.end(stream, kStExchange, 2);
    }
    step++;
    return 0;
}

BesideGrid Session::beside_attractive() const
{
    // (an iteration that sorts once in a while leaves as many SMs as the others)
    return stage_timers ? BesideGrid::nothing : refresh_period(step) == 1 ? BesideGrid::sorting : BesideGrid::settled;
}

int Session::attractive(cudaStream_t st)
{
    if (blocked.ready) return launch_attractive_blocked(blocked, Y2, Fattr, st, resident, beside_attractive());
    B200_TRY(launch_attractive(P, ids, Y2, N, K, row_lo, row_hi, Fattr, st));
    if (extra.count > 0) B200_TRY(launch_attractive_extra(extra.ptr, extra.ids, extra.val, Y2, N, row_lo, row_hi, Fattr, st));
    return 0;
}

int Session::set_resident(bool on)
{
    if (on == resident) return 0;
    if (!blocked.ready || rows() != N) { set_error("session: no point order to keep the state in"); return -1; }
    // Frep is scratch between iterations
    float2 *arrays[3] = {Y2, u, gains};
    for (float2 *a : arrays) {
        B200_TRY(launch_reorder_pairs(a, Frep, N, blocked.perm, /*scatter=*/!on, stream));
        B200_CUDA(cudaMemcpyAsync(a, Frep, sizeof(float2) * (size_t)N, cudaMemcpyDeviceToDevice, stream));
    }
    B200_CUDA(cudaStreamSynchronize(stream));
    resident = on;
    return 0;
}

int Session::build_blocked()
{
    B200_CUDA(cudaStreamSynchronize(stream));
    B200_CUDA(cudaStreamSynchronize(stream2));
    drop_graphs();   // captured iterations hold the pointers of the previous copy
    B200_TRY(set_resident(false));   // back to the natural order while the old copy's order still exists
    blocked.clear();
    blocked_arena.release();
    blocked_arena.serve(stream);
    blocked_arena.serve(stream2);
    B200_TRY(blocked_attractive_build(&blocked, blocked_arena, P, ids, N, K, row_lo, row_hi, cell_order, extra.count > 0 ? &extra : nullptr,
                                      stream));
    const char *e = getenv("B200TSNE_ATTRACTIVE_RESIDENT");
    const bool multi = comm && comm->world > 1;
    if (blocked.ready && !multi && rows() == N && !(e && atoi(e) == 0)) B200_TRY(set_resident(true));
    return 0;
}

void Session::drop_graphs()
{
    for (IterGraph &g : graphs)
        if (g.exec) graph_exec_release(host, g.exec, g.shape());
    graphs.clear();
}

bool Session::sorts_at(int b, int block) const
{
    const int period = refresh_period(step);   // (a block is of one phase)
    if (period <= 1) return period == 1;
    const bool fixed = kGraphIters % period == 0;
    if (fixed && block >= kGraphIters) return b % period == 0;
    if (fixed) return b == 0 && since_sort >= (block > 1 ? 2 * period : period);
    const int first = std::max(0, period - since_sort);
    return b >= first && (b - first) % period == 0;
}

int Session::refresh_period(int at) const
{
    const bool early = at < force_magnify_iters + 50;
    if (!early) return order_refresh;
    return comm && comm->world > 1 ? order_refresh_early_sharded : order_refresh_early;
}

// How many of the next iterations one graph covers; 0 when the next one has to be launched directly.  A graph holds
// iterations of one phase of the schedule: an even number (the state slots and the exchange buffers alternate), or a
// single one where a caller steps one by one.
int Session::graph_block(int remaining) const
{
    // (a sharded run qualifies when it exchanges over peer memory: its meetings are kernels of this library)
    if (!use_graphs || stage_timers || (comm && comm->world > 1 && !px)) return 0;
    long long left = remaining;
    for (const int end : {force_magnify_iters, force_magnify_iters + 50})
        if (step < end) left = std::min<long long>(left, (long long)end - step);
    if (left >= kGraphIters && !(step & 1)) return kGraphIters;
    if (left >= 2 && !(step & 1)) return 2;
    return px ? 0 : 1;
}

// Capturing a block and having an executable for it costs 100 us (updated) to 400 (a new pair; sixteen iterations 2 to 3 ms) more
// than the launches it saves cost once, so it has to serve again: blocks that this call repeats or that an earlier one asked for, single iterations (50 us
// saved) that were asked for kSingleFrom times.  A caller that steps one by one and changes the schedule every time
// never gets there (2,000 / 60,000 points, us per step: 286 / 436 with a capture each, 119 / 118 launched directly); the odd
// iteration at the end of a short call does not pay for an executable of its own.
bool Session::worth_capturing(const IterGraph &key, int remaining)
{
    if (key.iters > 2 || (key.iters == 2 && remaining >= 4)) return true;
    if (key.iters == 1 && remaining > 1) return false;   // the odd one before a block
    for (IterGraph &m : missed)
        if (m.same(key)) return ++m.asked >= (key.iters > 1 ? 2 : kSingleFrom);
    if (missed.size() >= kMaxGraphs) missed.erase(missed.begin());
    missed.push_back(key);
    missed.back().asked = 1;
    return false;
}

// 0: done, `iters` iterations of at most the number asked for.  1: not captured, the caller launches directly.  Negative:
// error.  remaining: iterations left in the call.
int Session::run_graph_block(int &iters, int remaining, int norm_mode, float stop_norm)
{
    const bool late = step >= force_magnify_iters;
    IterGraph key;
    key.iters = iters;
    key.parity = px ? px->parity : step & 1;
    key.late = late;
    key.eta = eta;
    key.exaggeration = late ? 1.0f : exaggeration;
    key.momentum = late ? post_momentum : pre_momentum;
    key.norm_mode = norm_mode;
    key.stop_norm = stop_norm;
    int last_sort = -1;
    for (int b = 0; b < iters; b++)
        if (sorts_at(b, iters)) { key.sorts |= 1u << b; last_sort = b; }
    const int period = refresh_period(step);
    key.nodes = (period == 0 ? kNatural : period == 1 ? kSortsEach : 0) | (spread_takes_spectrum(rows()) ? kSpectrumInSpread : 0);
    IterGraph *g = nullptr;
    for (IterGraph &have : graphs)
        if (have.same(key)) g = &have;
    if (!g) {
        if (iters == kGraphIters && remaining < kLargeFrom && !graph_exec_kept(host, key.shape())) {
            iters = 2;
            return run_graph_block(iters, remaining, norm_mode, stop_norm);
        }
        if (!worth_capturing(key, remaining)) return 1;
    }
    if (!g) {
        if (graphs.size() >= kMaxGraphs) drop_graphs();
        // capture: the launches are recorded, not run, so the host-side counters are put back afterwards
        const int step0 = step;
        const int64_t launches0 = launches;
        cudaGraph_t graph = nullptr;
        B200_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        int rc = 0;
        for (int b = 0; b < iters && rc == 0; b++) rc = one_iteration(norm_mode, stop_norm, key.sorts >> b & 1);
        const cudaError_t end = cudaStreamEndCapture(stream, &graph);
        key.launches = launches - launches0;
        step = step0;
        launches = launches0;
        const bool same_buffers = !px || px->parity == key.parity;
        if (px && px->parity != key.parity) { px->parity = key.parity; Y2 = px->y_local(key.parity); w = px->w_local(key.parity); }
        if (rc == 0 && end == cudaSuccess && graph && same_buffers) key.exec = graph_exec_acquire(host, graph, key.shape());
        if (graph) cudaGraphDestroy(graph);
        if (rc != 0 || end != cudaSuccess || !key.exec) {
            (void)cudaGetLastError();
            use_graphs = false;   // the caller falls back to direct launches
            return 1;
        }
        graphs.push_back(key);
        g = &graphs.back();
    }
    B200_CUDA(cudaGraphLaunch(g->exec, stream));
    step += iters;
    since_sort = last_sort < 0 ? since_sort + iters : iters - last_sort;
    launches += g->launches;
    return 0;
}

int Session::iterate(int n_iters, float min_gradient_norm, float *elapsed_ms, int *iters_done)
{
    B200_CUDA(cudaSetDevice(device));
    const bool multi = comm && comm->world > 1;
    const bool early_stop = min_gradient_norm > 0.0f;
    // One GPU checks the norm on the device: the host queues a block of iterations and learns afterwards how many of
    // them took place (the ones after the stop change nothing).  Ranks have to take the decision together, on the host.
    const bool device_stop = early_stop && !multi;
    const int norm_mode = device_stop ? 2 : (early_stop || force_norm ? 1 : 0);
    int done = 0;
    bool stopped = false;
    B200_CUDA(cudaEventRecord(ev_t0, stream));
    if (device_stop) {   // no iteration of this call has a norm yet: a huge one in the slot that the first looks at
        B200_CUDA(cudaMemsetAsync(&state->unorm2[(step & 1) ^ 1], 0x7f, sizeof(double), stream));
    }
    for (int it = 0; it < n_iters && !stopped;) {
        // a meeting of the ranks gave up (the kernel says so in mapped host memory): queue nothing more
        if (px && *px->err_host) break;
        int block = (early_stop && multi) || (norm_mode == 1) ? 0 : graph_block(n_iters - it);
        const int step0 = step;
        if (block > 0) {
            const int rc = run_graph_block(block, n_iters - it, norm_mode, min_gradient_norm);
            if (rc < 0) return rc;
            if (rc != 0) block = 0;
        }
        if (block == 0) {
            const bool sorts = sorts_at(0, 1);
            since_sort = sorts ? 1 : since_sort + 1;
            B200_TRY(one_iteration(norm_mode, min_gradient_norm, sorts));
            block = 1;
        }
        it += block;
        done += block;
        if (!early_stop) continue;
        const int last = (step - 1) & 1;
        B200_CUDA(cudaMemcpyAsync(h_state, state, sizeof(IterState), cudaMemcpyDeviceToHost, stream));
        B200_CUDA(cudaStreamSynchronize(stream));
        if (device_stop) {
            const int took = h_state->done - done_seen;
            done_seen = h_state->done;
            done -= block - took;
            step = step0 + took;
            last_unorm = (float)sqrt(h_state->unorm2[last]);   // of the last one that took place: later ones repeat it
            stopped = took < block || last_unorm < min_gradient_norm;
            // the queued rest has gone through the state slots without changing anything but their turn
            if ((block - took) & 1) B200_TRY(launch_state_swap(state, stream));
            continue;
        }
        // every rank must take the same decision: sum the squared norms
        B200_TRY(comm->all_reduce_sum_f64(&state->unorm2[last], 1, stream));
        B200_CUDA(cudaMemcpyAsync(h_state, state, sizeof(IterState), cudaMemcpyDeviceToHost, stream));
        B200_CUDA(cudaStreamSynchronize(stream));
        last_unorm = (float)sqrt(h_state->unorm2[last]);
        if (last_unorm < min_gradient_norm) stopped = true;
    }
    B200_CUDA(cudaEventRecord(ev_t1, stream));
    B200_CUDA(cudaMemcpyAsync(h_state, state, sizeof(IterState), cudaMemcpyDeviceToHost, stream));
    B200_CUDA(cudaStreamSynchronize(stream));
    B200_CUDA(cudaStreamSynchronize(stream2));
    if (elapsed_ms) B200_CUDA(cudaEventElapsedTime(elapsed_ms, ev_t0, ev_t1));
    if (iters_done) *iters_done = done;
    done_seen = h_state->done;
    if (done > 0) last_Z = (float)h_state->z_last - (float)N;
    if (norm_mode == 1 && !early_stop && done > 0) last_unorm = (float)sqrt(h_state->unorm2[(step - 1) & 1]);
    if (h_state->bad) { set_error("non-finite coordinates in the embedding"); return -3; }
    if (px) {
        int expired = 0;
        B200_CUDA(cudaMemcpy(&expired, px->err, sizeof(int), cudaMemcpyDeviceToHost));
        if (expired || *px->err_host) {
            px->failed = true;
            set_error("peer exchange: a rank did not arrive within " + std::to_string(px->timeout_ns / 1000000ull) + " ms");
            return -5;
        }
    }
    return 0;
}

int Session::attach_peer_exchange()
{
    if (!comm || comm->world < 2 || px) return 0;
    const char *e = getenv("B200TSNE_EXCHANGE");   // "nccl": collectives only (must be set alike on all ranks)
    if (e && strcmp(e, "nccl") == 0) return 0;
    B200_CUDA(cudaSetDevice(device));
    B200_TRY(peer_exchange_acquire(&px, comm, N + 16, stream));
    if (!px) return 0;
    // The grid sum: every rank reads all partial grids ((W - 1) x 2.4 MB over NVLink per rank), or the slice owners
    // form (2 x 2.4 MB x (W - 1) / W and one more flag round trip).  B200TSNE_GRID_SUM = "all" / "slices"; default:
    // slices from eight ranks on.  Measured at N = 10^6: four ranks, slices 3 % slower (6 078 against 6 290
    // iterations/s: the extra round trip costs more than 3.6 MB less traffic saves); eight ranks, slices 12 % faster
    // (7 807 against 6 939: 4.2 MB instead of 16.8 MB per rank and iteration).
    {
        const char *g = getenv("B200TSNE_GRID_SUM");
        grid_two_shot = g ? strcmp(g, "slices") == 0 : comm->world >= 8;
    }
    if (grid_two_shot) w_sum = px->ws_local();
    else B200_TRY(arena.alloc((void **)&w_sum, sizeof(float4) * kG * kG));
    B200_CUDA(cudaMemcpyAsync(px->y_local(px->parity), Y2_own, sizeof(float2) * (size_t)N, cudaMemcpyDeviceToDevice, stream));
    B200_CUDA(cudaStreamSynchronize(stream));
    Y2 = px->y_local(px->parity);
    w = px->w_local(px->parity);
    return 0;
}

// ---- set-up: points -> kNN -> perplexity -> symmetrised fixed-width P ------------------------------
int Session::affinities_from_points(const float *X_host, int D, float perplexity, float eps)
{
    B200_CUDA(cudaSetDevice(device));
    if (D <= 0 || !X_host) { set_error("affinities: invalid points"); return -1; }
    if (K > N) { set_error("affinities: num_neighbors exceeds num_points"); return -1; }
    const bool multi = comm && comm->world > 1;
    DeviceArena tmp;
    tmp.serve(stream);
    float *X = nullptr, *d2 = nullptr, *p_all = nullptr;
    int32_t *ids_all = nullptr;
    unsigned int *max_enc = nullptr;
    const int64_t r = rows();
    const int64_t chunk = multi ? (N + comm->world - 1) / comm->world : N;
    const int64_t npad = multi ? chunk * comm->world : N;

    StageClock clk(this);
    B200_TRY(tmp.alloc((void **)&X, sizeof(float) * N * D));
    B200_TRY(copy_in(X, X_host, sizeof(float) * N * D, stream));
    clk.begin(stream);   // the search itself: the points are on their way
    B200_TRY(tmp.alloc((void **)&d2, sizeof(float) * std::max<int64_t>(chunk, 1) * K));
    B200_TRY(tmp.alloc((void **)&max_enc, sizeof(unsigned int)));
    // Every rank holds all the points.  By default the QUERIES are sharded: a rank searches its own
    // rows against the whole database and needs no exchange, and its cost falls as 1/world (the
    // search costs about the same per query whatever the database size).  B200TSNE_KNN_SHARD=database
    // shards the DATABASE instead, as a deployment whose points do not fit one GPU would: every rank
    // searches all queries against its own rows, and the owners of the query rows receive the
    // partial lists (all-to-all) and merge them.  Both give the same lists bit for bit.
    const char *shard_env = getenv("B200TSNE_KNN_SHARD");
    bool db_sharded = multi && shard_env && strcmp(shard_env, "database") == 0;
    if (multi && !shard_env && knn_tc_supported(N, D, K)) {
        // no wish stated: shard the database when the operand images of ALL points and the buffers of this rank's
        // queries would not fit in half of what is free (every rank decides alike: same sizes, and the ranks of a
        // node have the same memory)
        size_t free_b = 0, total_b = 0;
        B200_CUDA(cudaMemGetInfo(&free_b, &total_b));
        const int64_t batch = std::min<int64_t>(std::max<int64_t>(r, 1), 1 << 20);
        if (knn_tc_workspace_bytes(D, K, batch, N, N <= kCellRowsMax) > total_b / 2) db_sharded = true;
    }
    // the cells of the points: the search visits by them, and the blocked copy of P numbers the points by them
    const char *attr_mode = getenv("B200TSNE_ATTRACTIVE");
    const bool want_order = N > kAttractiveTile && !(attr_mode && strcmp(attr_mode, "rows") == 0);
    PointCells cells;
    const bool cells_search = !db_sharded && knn_tc_supported(N, D, K);
    if (want_order || cells_search) B200_TRY(point_cells_build(&cells, X, D, 0, N, cells_search, tmp, stream));
    if (!db_sharded) {
        B200_TRY(knn_search(X, N, D, K, row_lo, row_hi, 0, N, ids, d2, &knn_stats, stream, cells.cells ? &cells : nullptr));
    } else {
        int32_t *part_i = nullptr, *recv_i = nullptr;
        float *part_d = nullptr, *recv_d = nullptr;
        B200_TRY(tmp.alloc((void **)&part_i, sizeof(int32_t) * npad * K));
        B200_TRY(tmp.alloc((void **)&part_d, sizeof(float) * npad * K));
        B200_TRY(tmp.alloc((void **)&recv_i, sizeof(int32_t) * npad * K));
        B200_TRY(tmp.alloc((void **)&recv_d, sizeof(float) * npad * K));
        B200_CUDA(cudaMemsetAsync(part_i, 0x7f, sizeof(int32_t) * npad * K, stream));
        B200_CUDA(cudaMemsetAsync(part_d, 0x7f, sizeof(float) * npad * K, stream));
        B200_TRY(knn_search(X, N, D, K, 0, N, row_lo, row_hi, part_i, part_d, &knn_stats, stream));
        B200_TRY(comm->all_to_all(part_i, recv_i, sizeof(int32_t) * (size_t)chunk * K, stream));
        B200_TRY(comm->all_to_all(part_d, recv_d, sizeof(float) * (size_t)chunk * K, stream));
        B200_TRY(launch_knn_merge(recv_i, recv_d, comm->world, chunk * K, r, K, ids, d2, stream));
    }
    B200_TRY(launch_knn_finalize(ids, d2, r * K, stream));
    clk.end(stream, kStKnn, 4);

    clk.begin(stream);
    // the order in which the attractive force's blocked copy of P numbers the points (every rank computes the same)
    if (want_order) {
        if (!cell_order) B200_TRY(arena.alloc((void **)&cell_order, sizeof(int32_t) * N));
        B200_TRY(order_points_by_cell(cells, X, D, cell_order, stream));
    }

    clk.begin(stream);
    const unsigned int zero_enc = enc_float(0.0f);
    B200_CUDA(cudaMemcpyAsync(max_enc, &zero_enc, sizeof(unsigned int), cudaMemcpyHostToDevice, stream));
    B200_TRY(launch_absmax(d2, r * K, max_enc, stream));
    if (multi) B200_TRY(comm->all_reduce_max_u32(max_enc, 1, stream));
    B200_TRY(tmp.alloc((void **)&p_all, sizeof(float) * npad * K));
    float *p_rows = p_all + (multi ? (size_t)comm->rank * chunk * K : 0);
    B200_TRY(launch_perplexity(d2, r, K, perplexity, eps, max_enc, p_rows, nullptr, stream));
    const int32_t *ids_for_sym = ids;
    if (multi) {
        B200_TRY(tmp.alloc((void **)&ids_all, sizeof(int32_t) * npad * K));
        B200_CUDA(cudaMemcpyAsync(ids_all + (size_t)comm->rank * chunk * K, ids, sizeof(int32_t) * r * K,
                                  cudaMemcpyDeviceToDevice, stream));
        B200_TRY(comm->all_gather_inplace(ids_all, sizeof(int32_t) * (size_t)chunk * K, stream));
        B200_TRY(comm->all_gather_inplace(p_all, sizeof(float) * (size_t)chunk * K, stream));
        ids_for_sym = ids_all;
    }
    // one GPU: the rows are taken in the cell order, cluster by cluster (the rows a row looks up are then in L2)
    const bool all_rows = !multi && row_lo == 0 && row_hi == N;
    float *furthest = nullptr;
    if (all_rows) B200_TRY(tmp.alloc((void **)&furthest, sizeof(float) * N));
    B200_TRY(launch_symmetrize(p_all, ids_for_sym, N, K, row_lo, row_hi, P, stream, all_rows && cell_order ? cell_order : nullptr, all_rows ? d2 : nullptr,
                               furthest));
    extra = ExtraEntries();
    if (symmetric_p || (getenv("B200TSNE_SYMMETRIC_P") && atoi(getenv("B200TSNE_SYMMETRIC_P")) != 0)) {
        // the mirror images of the one-directional edges whose target is an owned row (affinities.cu)
        int64_t n_extra = 0;
        int *cursor = nullptr;
        if (!extra_ptr) B200_TRY(arena.alloc((void **)&extra_ptr, sizeof(int) * (r + 1)));
        B200_TRY(launch_reverse_only_count(p_all, ids_for_sym, N, K, row_lo, row_hi, extra_ptr, &n_extra, stream));
        B200_TRY(tmp.alloc((void **)&cursor, sizeof(int) * std::max<int64_t>(r, 1)));
        B200_TRY(arena.alloc((void **)&extra_ids, sizeof(int32_t) * std::max<int64_t>(n_extra, 1)));   // (a second call leaves the first lists to the arena)
        B200_TRY(arena.alloc((void **)&extra_val, sizeof(float) * std::max<int64_t>(n_extra, 1)));
        B200_TRY(launch_reverse_only_fill(p_all, ids_for_sym, N, K, row_lo, row_hi, extra_ptr, cursor, extra_ids, extra_val, stream));
        extra.ptr = extra_ptr; extra.ids = extra_ids; extra.val = extra_val; extra.count = n_extra;
    }
    B200_TRY(build_blocked());
    clk.end(stream, kStAffinities, 3);
    B200_CUDA(cudaStreamSynchronize(stream));
    return 0;
}

}  // namespace b200
