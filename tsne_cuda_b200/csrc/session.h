// Device-resident state of one FIt-SNE run on one GPU (one rank of a multi-GPU run).
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "common.cuh"

namespace b200 {

struct Comm;          // comm.h
struct PeerExchange;  // peer.h
struct StreamSet;     // hostio.h

enum Stage { kStSpread = 0, kStConvolve, kStGather, kStAttractive, kStUpdate, kStExchange, kStKnn, kStAffinities, kStOrder };

// RAII holder for device allocations of a session
struct DeviceArena {
    std::vector<void *> ptrs;
    std::vector<cudaStream_t> consumers;   // streams whose work uses this memory: synchronised before anything is freed
    ~DeviceArena();
    void serve(cudaStream_t st) { consumers.push_back(st); }
    int alloc(void **p, size_t bytes);
    void release();
    void forget();   // the memory went with its context
};

struct Session {
    int device = 0;
    int64_t N = 0;           // all points
    int K = 0;
    int64_t row_lo = 0, row_hi = 0;  // owned rows
    StreamSet *host = nullptr;       // the streams, events and pinned memory below come from here
    cudaStream_t stream = nullptr;
    cudaStream_t stream2 = nullptr;  // attractive force overlaps the grid pipeline
    cudaStream_t stream3 = nullptr;  // and so does the kernel's spectrum
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_spectrum = nullptr, ev_spread = nullptr, ev_order = nullptr, ev_t0 = nullptr, ev_t1 = nullptr;
    DeviceArena arena;

    // affinities (owned rows)
    float *P = nullptr;       // [rows][K]
    int32_t *ids = nullptr;   // [rows][K]
    // Column-blocked copy of P for the attractive force (attractive_blocked.cu), built with the affinities when the
    // neighbours of a row fall into few tiles of the cell order; otherwise the row-major kernel reads P / ids.
    BlockedAttractive blocked;
    DeviceArena blocked_arena;
    int32_t *cell_order = nullptr;   // [N] point order by cell (from the points; null = natural order)
    int build_blocked();             // (re)builds `blocked` from P / ids; drops captured iterations
    // One GPU with the blocked copy: the embedding, momentum and gains live in the copy's point order (`resident`),
    // so the attractive stage needs no conversion; the accessors convert where values enter and leave.
    bool resident = false;
    int set_resident(bool on);       // converts the three arrays when the state changes
    const int32_t *state_order() const { return resident ? blocked.perm : nullptr; }
    // Opt-in: P truly symmetric, (p + p^T) / 2N, instead of the reference's fixed-width form that drops the mirror
    // image of one-directional edges.  The extra entries of the owned rows live beside P / ids.
    bool symmetric_p = false;
    ExtraEntries extra;
    int *extra_ptr = nullptr;
    int32_t *extra_ids = nullptr;
    float *extra_val = nullptr;
    // embedding and optimiser state
    float2 *Y2 = nullptr;     // [N] AoS, replicated on every rank
    float2 *Fattr = nullptr;  // [N] (owned rows valid)
    float2 *Frep = nullptr;   // [N] (owned rows valid)
    float2 *gains = nullptr;  // [rows]
    float2 *u = nullptr;      // [rows]
    float *soa_tmp = nullptr; // [2N] staging for SoA <-> AoS conversion
    int32_t *order = nullptr, *order_alt = nullptr, *order_keys = nullptr, *box_hist = nullptr;  // spread order (owned rows)
    // iterations between two counting sorts of the spread order once the embedding has settled, and while it is still being
    // exaggerated and 50 iterations after, on one GPU and on one of several (0 = natural order)
    int order_refresh = 8, order_refresh_early = 1, order_refresh_early_sharded = 1;
    // grid
    float4 *w = nullptr;      // [G][G]
    float4 *ytilde = nullptr; // [G][G]
    void *fft_mem = nullptr;
    FftWorkspace fft;
    IterState *state = nullptr;
    IterState *h_state = nullptr;  // pinned mirror
    InterpConsts ic;

    // schedule
    float eta = 200.0f, exaggeration = 12.0f, pre_momentum = 0.5f, post_momentum = 0.8f;
    int force_magnify_iters = 250;
    int step = 0;
    float last_Z = 0.0f, last_unorm = 0.0f;

    // instrumentation
    bool stage_timers = false;
    bool force_norm = false;   // maintain the update norm even without an early-stop threshold
    float stage_ms[kStages] = {0};
    int64_t stage_launches[kStages] = {0};
    int64_t launches = 0;

    KnnStats knn_stats;    // of the last affinities_from_points
    Comm *comm = nullptr;  // null on a single GPU
    // Sharded runs exchange over peer memory when every rank could map the others (peer.h); Y2 and w then
    // point into the exchange block and alternate between its two buffers, w_sum holds the reduced grid.
    PeerExchange *px = nullptr;
    float2 *Y2_own = nullptr;   // the session's own allocations, used whenever px is null
    float4 *w_own = nullptr;
    float4 *w_sum = nullptr;
    bool grid_two_shot = false;   // peer-memory exchange: the grid sum as slice owners (peer.h), chosen at attach
    int attach_peer_exchange();   // collective, after comm is set

    // Captured iterations (single GPU or peer-memory exchange, no stage timers): at small N the loop is bound by the
    // launch and dependency latency of its kernels, so blocks of iterations are replayed as CUDA graphs.  What a block
    // froze into its launches is its key.
    struct IterGraph {
        cudaGraphExec_t exec = nullptr;
        int iters = 0, parity = 0, norm_mode = 0;
        bool late = false;
        int nodes = 0;             // which kernels an iteration has beside the sorts' (kNatural, ...)
        unsigned sorts = 0;        // bit b: the b-th iteration sorts the spread order
        float eta = 0, exaggeration = 0, momentum = 0, stop_norm = 0;
        int64_t launches = 0;
        int asked = 0;             // of one without an executable: how many calls asked for it
        // what decides which nodes it has: an executable of the same shape can be updated instead of made anew
        unsigned long long shape() const { return (unsigned long long)sorts << 32 | (unsigned)iters << 4 | (unsigned)nodes; }
        bool same(const IterGraph &o) const
        {
            return iters == o.iters && parity == o.parity && norm_mode == o.norm_mode && late == o.late && nodes == o.nodes &&
                   sorts == o.sorts && eta == o.eta && exaggeration == o.exaggeration && momentum == o.momentum && stop_norm == o.stop_norm;
        }
    };
    static constexpr int kGraphIters = 16;   // iterations of a large block; what is left of a phase goes in pairs
    // A large block's first executable of a process costs 3 to 20 ms: calls of fewer iterations go in pairs until one exists
    // (20 iterations at 10^6 points after a warm-up of 3: 23.3 ms with it, 5.6 in pairs).
    static constexpr int kLargeFrom = 64;
    static constexpr int kSingleFrom = 6;
    static constexpr size_t kMaxGraphs = 24;
    std::vector<IterGraph> graphs, missed;   // with an executable; asked for lately, without one
    bool use_graphs = true;   // B200TSNE_GRAPHS=0 turns them off
    static constexpr int kNatural = 1, kSortsEach = 2, kSpectrumInSpread = 4;
    int refresh_period(int at) const;   // iterations between two sorts of the spread order at step `at` (0: natural order)
    // Does the b-th of `block` iterations launched together sort?  since_sort: iterations since the last that did.  Where the
    // period divides a large block (unless a variable says otherwise it does), these sort at fixed places, so that one executable
    // serves a phase, and pairs, of which one that sorts is another executable, half as often.
    // (since_sort stays when a state is set: the order is that of the points before, which costs a spread time but no result, and
    // a caller that sets a state for each step would pay for a sort in each.  32 iterations after another layout, one by one / in
    // pairs / in sixteens: 40,000 points 1,204 / 1,078 / 1,030 us, 10^6 7,887 / 7,788 / 7,715.)
    bool sorts_at(int b, int block) const;
    int since_sort = 1 << 20;
    int graph_block(int remaining) const;
    bool worth_capturing(const IterGraph &key, int remaining);
    int run_graph_block(int &iters, int remaining, int norm_mode, float stop_norm);
    int done_seen = 0;        // IterState::done as the host last saw it
    void drop_graphs();

    int64_t rows() const { return row_hi - row_lo; }
    int init(int64_t N, int K, int64_t row_lo, int64_t row_hi, int device);
    void destroy();
    int set_embedding_soa(const float *Y_host, bool reset);
    int get_embedding_soa(float *Y_host);
    // optimiser state of the owned rows (momentum = the reference's old_forces, gains), SoA [2][rows] on the host
    int get_optimizer_soa(float *momentum_host, float *gains_host);
    int set_optimizer_soa(const float *momentum_host, const float *gains_host);
    // Small maps of one GPU: the whole state crosses in one piece that a kernel reads or writes in pinned memory.  Copies of
    // the three arrays from and to pageable memory, each with a kernel and a wait, are most of a call that runs an iteration
    // or two: state in, one iteration, state out 182 -> 113 us at 2,000 points, 278 -> 168 at 21,845.
    // The host reads and writes the caller's arrays itself, so those in device or managed memory (null: not given) go by copies.
    bool small_state(const void *Y, const void *momentum, const void *gains) const;
    int set_small_state(const float *Y_host, const float *momentum_host, const float *gains_host, int at_step);
    int get_small_state(float *Y_host, float *momentum_host, float *gains_host);
    int iterate(int n_iters, float min_gradient_norm, float *elapsed_ms, int *iters_done);
    int one_iteration(int norm_mode, float stop_norm, bool sorts);
    BesideGrid beside_attractive() const;   // what runs beside the attractive kernel at this step
    int attractive(cudaStream_t st);   // Fattr of the owned rows from the current embedding
    int attractive_launches() const { return blocked.ready ? (resident ? 2 : 3) + (blocked.extra_C > 0) : 1 + (extra.count > 0); }
    int affinities_from_points(const float *X_host, int D, float perplexity, float eps);
};

}  // namespace b200
