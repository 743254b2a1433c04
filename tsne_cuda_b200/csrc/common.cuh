// Internal declarations shared by the kernels and the host orchestration of libtsnecuda.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

namespace b200 {

// ---- FIt-SNE grid constants (reference: src/fit_tsne.cu:246-272) ----
constexpr int kBoxes = 130;            // boxes per dimension (125 rounded up through the allowed list)
constexpr int kInterp = 3;             // Lagrange nodes per box and dimension
constexpr int kG = kBoxes * kInterp;   // 390 nodes per dimension
constexpr int kTerms = 4;              // charges (1, x, y, x^2+y^2)
constexpr int kM = 784;                // transform length of the zero-padded convolution (>= 2*kG-1)
constexpr int kStages = 9;             // instrumented stages (== B200TSNE_N_STAGES)

// ---- error plumbing ----
void set_error(const std::string &msg);
const std::string &last_error();
int release_cached_memory();   // session.cu: hand the device memory pool of the current device back to the driver
int cuda_fail(cudaError_t e, const char *what, const char *file, int line);

#define B200_CUDA(expr)                                                        \
    do {                                                                       \
        cudaError_t _e = (expr);                                               \
        if (_e != cudaSuccess) return ::b200::cuda_fail(_e, #expr, __FILE__, __LINE__); \
    } while (0)

#define B200_TRY(expr)            \
    do {                          \
        int _s = (expr);          \
        if (_s != 0) return _s;   \
    } while (0)

// Per-iteration scalars that live in device memory so that an iteration needs no host round trip.
// Slots are double-buffered by iteration parity: iteration `it` reads slot it&1 and prepares slot
// (it+1)&1 for its successor.
struct IterState {
    unsigned int min_enc[2];   // order-preserving encodings of min / max over all coordinates
    unsigned int max_enc[2];
    double zsum[2];            // sum_i Z_i, accumulated on the grid by the convolution's last pass
    double unorm2[2];          // sum of squared updates (only maintained on request)
    double z_last;             // zsum of the last iteration that changed the embedding
    int bad;                   // set when a non-finite coordinate is produced
    int done;                  // iterations that changed the embedding (counts on; the host looks at differences)
};

// Lagrange constants evaluated on the host exactly as the reference does (src/fit_tsne.cu:303-320).
struct InterpConsts {
    float sp[kInterp];
    float den[kInterp], den_inv[kInterp];
};
InterpConsts make_interp_consts();

__host__ __device__ inline unsigned int enc_float(float f)
{
#ifdef __CUDA_ARCH__
    unsigned int b = __float_as_uint(f);
#else
    union { float f; unsigned int u; } c; c.f = f; unsigned int b = c.u;
#endif
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__host__ __device__ inline float dec_float(unsigned int e)
{
    unsigned int b = (e & 0x80000000u) ? (e & 0x7fffffffu) : ~e;
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    union { float f; unsigned int u; } c; c.u = b; return c.f;
#endif
}

// ---- chained launches ----
// A kernel of the iteration's chain may be placed on the SMs while the one before it in its stream still runs.
// after_previous() returns when that one has ended and its stores are visible, so completion stays as transitive as with
// plain launches: every thread that touches more than constants makes the call, and a block that leaves early makes it too.
// let_next_start() allows the next one to be placed once all blocks have made it; without it, when all have ended.
// Before after_previous() a kernel touches constants, and nothing else unless the launch in front of it is an ORDINARY one
// and leaves alone what is read: that launch began after everything before it had ended, so what earlier kernels wrote is
// there.  Two kernels rest on that, and neither launch in front of them may become a chained one:
//   attractive_blocked_kernel   reads positions and its stream, behind clear_forces_kernel (writes the forces);
//   dense_distance_kernel       reads points and the list of queries, behind a selection (writes lists) whose own predecessors,
//                               back to the ordinary launch that a search begins with, write distances and lists only.
// Pointers to what an earlier kernel wrote are not __restrict__ but there: the compiler would be free to read through them
// before that call.
#ifdef __CUDACC__
// two floats in one register pair, as the packed instructions take them
__device__ __forceinline__ unsigned long long pack(float2 a)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 unpack(unsigned long long r)
{
    float2 a;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
    return a;
}
// Two zeros to add to a packed square, so that it is rounded for itself: of a packed product and a packed sum the compiler
// makes one rounding, and it does so too where it can see that the sum is with zero, so kernels have this as an argument.
constexpr unsigned long long kMinusZero2 = 0x8000000080000000ull;

__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 blocks, unsigned threads, size_t smem, cudaStream_t st, Args... args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = blocks;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
#endif

// ---- kernel launchers (all asynchronous on `st`; pointers are device memory) ----

// knn.cu
int launch_transpose(const float *X, int64_t N, int D, float *XT, cudaStream_t st);   // [N][D] -> [D][N]
int launch_knn_exact(const float *XT, int64_t N, int D, int K, int64_t q_lo, int64_t q_hi, int64_t db_lo,
                     int64_t db_hi, int32_t *ids, float *d2, cudaStream_t st);   // ids/d2 keep (INT_MAX,+inf) in unfilled slots
// cells.cu: nearest of at most kMaxCells sample points, for every row of a range, with the distance to it
struct DeviceArena;
constexpr int kMaxCells = 64;
struct CellTable {
    long long centre_row[kMaxCells];
    unsigned int radius_bits[kMaxCells];   // the rest belongs to one neighbour search, see knn_tc.cu
    int db_count[kMaxCells], q_count[kMaxCells];
    int db_start[kMaxCells + 1], q_start[kMaxCells + 1];
    int db_cursor[kMaxCells], q_cursor[kMaxCells];
};
struct PointCells {
    int cells = 0;
    int64_t lo = 0, n = 0;          // rows [lo, lo + n)
    CellTable *tab = nullptr;
    float *own = nullptr;           // [n] distance to the own cell's sample point
    unsigned char *cell = nullptr;  // [n]
    float *dist = nullptr;          // [n][kMaxCells] the distances to all of them, where they are kept
};
constexpr int64_t kCellRowsMax = (int64_t)1 << 20;   // rows whose distances to all sample points are kept (256 MB)
inline int point_cells_count(int64_t n) { return (int)(n < 4096 ? 1 : (n / 2048 < kMaxCells ? n / 2048 : kMaxCells)); }   // see point_cells_build
int point_cells_build(PointCells *pc, const float *X, int D, int64_t lo, int64_t n, bool distances, DeviceArena &arena, cudaStream_t st);
int point_cells_assign(const PointCells &pc, const float *X, int D, int64_t lo, int64_t n, float *dist, float *own, unsigned char *cell, cudaStream_t st);
int point_cells_chain(const PointCells &pc, const float *X, int D, int *rank, DeviceArena &arena, cudaStream_t st);

// knn_tc.cu: tensor-core filter + exact re-rank + proof (nd = database rows to scan); pc: the cells of the database rows
bool knn_tc_supported(int64_t nd, int D, int K);
// cells_kept: the queries' distances to the cells are at hand (PointCells::dist)
size_t knn_tc_workspace_bytes(int D, int K, int64_t nq, int64_t nd, bool cells_kept);
int launch_knn_tc(const float *X, int64_t N, int D, int K, int64_t q_lo, int64_t q_hi, int64_t db_lo, int64_t db_hi, const PointCells &pc,
                  int32_t *ids, float *d2, void *workspace, int **failed_list, int *n_failed_host, float *err_ratio_host,
                  cudaStream_t st);
int mbar_wait_selftest(int timeout_ms, float *waited_ms, cudaStream_t st);   // see b200tsne_selftest_bounded_waits
struct KnnStats {
    int tensor_core = 0;            // 1 when the tensor-core path ran
    int rows_recomputed = 0;        // rows the proof could not certify, recomputed by another search
    float filter_error_ratio = 0;   // largest observed filter error on the candidates / assumed bound
};
// X: [N][D] row-major on the device; picks the path, handles the fallback rows, synchronises `st`.
// pc (optional): the cells of rows [db_lo, db_hi), where the caller has them
int knn_search(const float *X, int64_t N, int D, int K, int64_t q_lo, int64_t q_hi, int64_t db_lo, int64_t db_hi,
               int32_t *ids, float *d2, KnnStats *stats, cudaStream_t st, const PointCells *pc = nullptr);
// knn_dense.cu: whole rows of distances and a selection (see that file); distances of NaN never rank
bool knn_dense_supported(int K);
int knn_dense(const float *X, int D, int K, int64_t q_lo, int64_t nq, const int *q_index, int64_t out_base, int64_t db_lo, int64_t db_hi,
              int32_t *ids, float *d2, DeviceArena &tmp, cudaStream_t st);
int knn_dense_load();
int knn_dense_in_scratch(const float *X, int64_t N, int D, int K, float *scratch, long long floats, int32_t *ids, float *d2, cudaStream_t st);
// knn.cu: search with the scratch in a fixed device array of the library (no allocation)
long long knn_noalloc_max_elems();
int knn_noalloc(const float *X, int64_t N, int D, int K, int32_t *ids, float *d2, cudaStream_t st);
int launch_knn_merge(const int32_t *ids_parts, const float *d2_parts, int parts, int64_t part_stride, int64_t n_rows,
                     int K, int32_t *ids, float *d2, cudaStream_t st);
int launch_knn_finalize(int32_t *ids, float *d2, int64_t n, cudaStream_t st);

// affinities.cu
int launch_absmax(const float *v, int64_t n, unsigned int *max_enc, cudaStream_t st);  // max_enc: enc_float accumulator, pre-set to enc(0)
int launch_perplexity(const float *d2, int64_t n_rows, int K, float perplexity, float eps, const unsigned int *max_enc,
                      float *p, float *betas, cudaStream_t st);
int launch_reverse_only_count(const float *p_all, const int32_t *ids_all, int64_t N, int K, int64_t row_lo, int64_t row_hi, int *ptr,
                              int64_t *count_host, cudaStream_t st);
int launch_reverse_only_fill(const float *p_all, const int32_t *ids_all, int64_t N, int K, int64_t row_lo, int64_t row_hi, const int *ptr,
                             int *cursor, int32_t *ext_ids, float *ext_val, cudaStream_t st);
// visit (optional): row_hi - row_lo row numbers inside [row_lo, row_hi), the order in which the rows are taken
// d2, furthest (optional, all rows): the exact distances of the lists, ascending in a row; N floats of scratch
int launch_symmetrize(const float *p_all, const int32_t *ids_all, int64_t N, int K, int64_t row_lo, int64_t row_hi,
                      float *P_rows, cudaStream_t st, const int32_t *visit = nullptr, const float *d2 = nullptr, float *furthest = nullptr);

// attractive.cu   (Y2: AoS float2 [N]; F2: AoS float2, rows [row_lo,row_hi) written at their global index)
int launch_attractive(const float *P_rows, const int32_t *ids_rows, const float2 *Y2, int64_t N, int K, int64_t row_lo,
                      int64_t row_hi, float2 *F2, cudaStream_t st);
// F2[row] += force of the rows' extra entries (variable-width list, see ExtraEntries below)
int launch_attractive_extra(const int *ptr, const int32_t *ext_ids, const float *ext_val, const float2 *Y2, int64_t N, int64_t row_lo,
                            int64_t row_hi, float2 *F2, cudaStream_t st);

// attractive_blocked.cu: column-blocked copy of P whose gathers come from shared memory (see that file)
// Further stored entries of the owned rows in variable-width form: row r (0-based among the owned rows) has the
// entries ptr[r] .. ptr[r + 1].  Used for the reverse-only edges that make P truly symmetric (affinities.cu).
struct ExtraEntries {
    const int *ptr = nullptr;        // [rows + 1]
    const int32_t *ids = nullptr;    // columns (point numbers)
    const float *val = nullptr;
    int64_t count = 0;
};
constexpr int kAttractiveTile = 28672;   // points per tile of the blocked copy; up to here the order of the points does not matter
struct BlockedAttractive {
    const float *ev = nullptr;
    const uint16_t *ec = nullptr;
    const int *chunk_row0 = nullptr, *tile_chunk0 = nullptr;
    const float *extra_ev = nullptr;       // second stream: the extra entries (none: extra_C = 0)
    const uint16_t *extra_ec = nullptr;
    const int *extra_chunk_row0 = nullptr, *extra_tile_chunk0 = nullptr;
    int extra_C = 0;
    int64_t extra_E = 0;
    const int32_t *perm = nullptr, *own_perm = nullptr, *own_pos = nullptr;
    float2 *Yp = nullptr, *Yown = nullptr, *Fp = nullptr;
    int ntiles = 0, T = 0, C = 0;
    int64_t E = 0, groups = 0, N = 0, row_lo = 0, rows = 0;
    float entries_per_group = 0.0f;   // of the sampled rows, under the chosen order
    bool ready = false;
    void clear();
};
// perm[q] = the point at position q of the cell order; pc: the cells of all N points
int order_points_by_cell(const PointCells &pc, const float *X, int D, int32_t *perm, cudaStream_t st);
int blocked_attractive_build(BlockedAttractive *b, DeviceArena &arena, const float *P_rows, const int32_t *ids_rows, int64_t N, int K,
                             int64_t row_lo, int64_t row_hi, const int32_t *perm, const ExtraEntries *extra, cudaStream_t st);
int launch_exclusive_scan_i32(int *data, int64_t n, cudaStream_t st);   // in place; small arrays (one block)
// in_cell_order: Y2 and F2 are in the copy's own point order (one GPU): no conversion before or after the kernel
// beside: what runs at the same time (the grid pipeline of an iteration that sorts its points, or one that does not)
enum class BesideGrid { nothing, sorting, settled };
int launch_attractive_blocked(const BlockedAttractive &b, const float2 *Y2, float2 *F2, cudaStream_t st, bool in_cell_order = false,
                              BesideGrid beside = BesideGrid::nothing);
int free_beside_attractive(const BlockedAttractive &b, BesideGrid beside, int *sms);   // SMs that it leaves alone then

// repulsive.cu
struct FftWorkspace {
    float4 *A;      // [columns 0 .. kM/2][four rows][8] row-transformed charges (see convolve.cu)
    float4 *B;      // the same after the column pass
    float2 *tw;     // [28][28] twiddles e^{-2 pi i k l / kM}
    float *Rk, *Kh; // row-transformed kernel; its spectrum by column
};
size_t fft_workspace_bytes();
int fft_workspace_init(FftWorkspace *ws, void *mem, cudaStream_t st);
int launch_state_reset(IterState *state, cudaStream_t st);   // both slots, sums and flags
int launch_state_swap(IterState *state, cudaStream_t st);    // exchanges the two slots (a stop between iterations of other parity)
int launch_minmax_init(const float2 *Y2, int64_t N, IterState *state, int slot, cudaStream_t st);
constexpr long long kSpreadDirectMax = 8192;      // up to here points are spread one by one
constexpr long long kSortMin = 32768;             // from here on the spread order is sorted (both: repulsive.cu),
constexpr long long kSortEarlyMin = 3000;         // from here on while the embedding is being exaggerated,
constexpr long long kSortEachFrom = 65536;        // from here on then in every iteration (session.cu)
constexpr long long kSpreadSingleMax = 131072;   // up to here a lane takes one point of the order
// order: local row indices sorted by box (null = natural order); see launch_order_count
// hist (optional): the sort's counters, cleared on the way for the next sort
int launch_spread(const float2 *Y2, int64_t row_lo, int64_t row_hi, const int32_t *order, int32_t *hist, const IterState *state,
                  int slot, InterpConsts ic, float4 *w, const FftWorkspace *spectrum, cudaStream_t st);
// spectrum (optional): the same launch does what launch_kernel_spectrum does; possible where a lane takes one point
inline bool spread_takes_spectrum(int64_t n) { return n > 0 && n <= kSpreadSingleMax; }
int launch_order_identity(int32_t *order, int64_t n, cudaStream_t st);
int launch_order_count(const float2 *Y2, int64_t row_lo, int64_t row_hi, const int32_t *order, int32_t *previous, int32_t *keys, int32_t *hist,
                       const IterState *state, int slot, cudaStream_t st);
int launch_order_scatter(int64_t n, int32_t *order, const int32_t *previous, const int32_t *keys, int32_t *hist, cudaStream_t st);
// convolve.cu: the kernel's spectrum along its first axis (needs the slot's min/max only), the first pass over the charges and
// the spectrum's second axis, and the rest; the last pass adds sum_i Z_i over all charges to state->zsum[slot] and clears w when asked to
int launch_kernel_spectrum(const IterState *state, int slot, const FftWorkspace &ws, cudaStream_t st);
int launch_convolve_rows(const float4 *w, const IterState *state, int slot, const FftWorkspace &ws, cudaStream_t st);
// free_sms: SMs that no other kernel fills meanwhile, as far as known
int launch_convolve(float4 *w, float4 *ytilde, IterState *state, int slot, const FftWorkspace &ws, bool zero_w, int free_sms, cudaStream_t st);
int launch_gather(const float2 *Y2, int64_t row_lo, int64_t row_hi, const IterState *state, int slot, InterpConsts ic,
                  const float4 *ytilde, float2 *Frep2, cudaStream_t st);

// update.cu
// where the updated rows go: one array (in place) or the embedding copy of every rank (peer memory)
constexpr int kMaxUpdateTargets = 16;
struct UpdateTargets {
    float2 *p[kMaxUpdateTargets];
    int n;
};
// ytilde given: the repulsive force is interpolated in the same kernel and Frep2 is not read; norm_mode: see update.cu
int launch_update(const float2 *Y2, const UpdateTargets &dst, const float2 *Fattr2, const float2 *Frep2, const float4 *ytilde, InterpConsts ic,
                  float2 *gains2, float2 *u2, int64_t N, int64_t row_lo, int64_t row_hi, IterState *state, int slot, float eta,
                  float momentum, float exaggeration, int norm_mode, float stop_norm, cudaStream_t st);
int launch_apply_forces_soa(float *Y, float *attr, float *rep, float *gains, float *old_forces, float eta, float Z,
                            float momentum, float exaggeration, int64_t N, cudaStream_t st);
// perm (optional): position q of the pair array holds point perm[q] of the block-wise (x block, y block) array
int launch_soa_to_aos(const float *soa, float2 *aos, int64_t N, cudaStream_t st, const int32_t *perm = nullptr);
int launch_aos_to_soa(const float2 *aos, float *soa, int64_t N, cudaStream_t st, const int32_t *perm = nullptr);
// A small map's state between the device and memory that the host shares with it, block-wise [2][N] each: embedding, momentum,
// gains one after the other (load: and the embedding's min/max into a slot that has been reset; store: null arrays left out)
int launch_load_state(const float *io, float2 *Y2, float2 *u2, float2 *gains2, int64_t N, IterState *state, int slot, cudaStream_t st);
int launch_store_state(const float2 *Y2, const float2 *u2, const float2 *gains2, float *io, int64_t N, cudaStream_t st);
// dst[q] = src[perm[q]], or with scatter dst[perm[q]] = src[q]
int launch_reorder_pairs(const float2 *src, float2 *dst, int64_t N, const int32_t *perm, bool scatter, cudaStream_t st);
int launch_fill(float *p, float v, int64_t n, cudaStream_t st);

}  // namespace b200
