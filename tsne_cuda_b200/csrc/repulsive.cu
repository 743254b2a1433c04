// FIt-SNE repulsive force: spread of the point charges onto the 390x390 Lagrange grid and interpolation
// of the potentials back to the points.
//
// Reference: src/kernels/nbodyfft.cu (binning :43-73, Lagrange weights :75-105, spread :107-139,
// kernel evaluation :175-203, FFT convolution :3-41 + :395-424, gather :141-173) and
// src/kernels/rep_forces.cu (charges :57-76, forces and Z_i :3-31), sequenced as in
// src/fit_tsne.cu:411-469.
//
// Design (nothing here is a translation of the reference's kernels):
//  * One kernel per point pass.  Box index, in-box coordinate, Lagrange weights and charges are
//    recomputed in registers by spread and gather; the reference's nine N-sized intermediate
//    arrays do not exist.  The grid is AoS float4 per node, stored as (x-charge, y-charge, count,
//    r^2-charge) = two packed complex numbers, so a point issues 9 vector reductions instead of 36
//    scalar atomics.
//  * The convolution is in convolve.cu.
#include "fft784.cuh"

#include <algorithm>

namespace b200 {

InterpConsts make_interp_consts()
{
    InterpConsts c;
    float h = 1 / (float)kInterp;
    c.sp[0] = h / 2;
    for (int i = 1; i < kInterp; i++) c.sp[i] = c.sp[i - 1] + h;
    for (int i = 0; i < kInterp; i++) {
        c.den[i] = 1;
        for (int j = 0; j < kInterp; j++)
            if (i != j) c.den[i] *= c.sp[i] - c.sp[j];
        c.den_inv[i] = 1 / c.den[i];
    }
    return c;
}

namespace {

// ------------------------------------------------------------------------------------------
// min / max of the embedding into a state slot (start-up and after an exchange of Y)
// ------------------------------------------------------------------------------------------
__global__ void state_reset_kernel(IterState *state, int slot, int all)
{
    state->min_enc[slot] = 0xffffffffu;
    state->max_enc[slot] = 0u;
    if (all) {
        state->min_enc[slot ^ 1] = 0xffffffffu;
        state->max_enc[slot ^ 1] = 0u;
        state->zsum[0] = 0.0;
        state->zsum[1] = 0.0;
        state->unorm2[0] = 0.0;
        state->unorm2[1] = 0.0;
        state->bad = 0;
        state->done = 0;
    }
}

__global__ void state_swap_kernel(IterState *state)
{
    const unsigned int mn = state->min_enc[0], mx = state->max_enc[0];
    const double z = state->zsum[0];
    state->min_enc[0] = state->min_enc[1]; state->max_enc[0] = state->max_enc[1]; state->zsum[0] = state->zsum[1];
    state->min_enc[1] = mn; state->max_enc[1] = mx; state->zsum[1] = z;
}

__global__ void __launch_bounds__(256) minmax_kernel(const float2 *__restrict__ Y2, long long N, IterState *state, int slot)
{
    float mn = INFINITY, mx = -INFINITY;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
        const float2 y = Y2[i];
        mn = fminf(mn, fminf(y.x, y.y));
        mx = fmaxf(mx, fmaxf(y.x, y.y));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0 && mn <= mx) {
        atomicMin(&state->min_enc[slot], enc_float(mn));
        atomicMax(&state->max_enc[slot], enc_float(mx));
    }
}

// ------------------------------------------------------------------------------------------
// spread
// ------------------------------------------------------------------------------------------
// Same-address floating-point reductions serialise in L2, and an embedding is anything but uniform
// over its bounding square (during early exaggeration half the points sit in a few hundred boxes).
// So the spread walks the points in an order that is sorted by box (refreshed every few iterations
// by a counting sort; a stale order only costs efficiency, never correctness, because the box of
// every point is recomputed here): lanes that fall into the same box are neighbours in the warp,
// their 36 contributions are combined with a segmented shuffle reduction, and only the first lane of
// each run issues the nine vector reductions.
__device__ __forceinline__ int axis_box(float c, const GridGeom &g)
{
    int idx = (int)in_boxes(c - g.cmin, g);
    idx = max(0, idx);
    return min(kBoxes - 1, idx);
}

// A lane takes kSpreadPerLane consecutive points of the order.  While they stay in one box it sums their 36
// contributions in registers; a box change inside the lane sends the finished sum to the grid directly.  The
// lane's last (open) run is then combined with those of its neighbours as described above, so the 180
// shuffles of the segmented reduction are paid once per 32 * kSpreadPerLane points.
//
// Fewer points leave most SMs idle with four points a lane: up to kSpreadSingleMax a lane takes one.  Points without an
// order, up to kSpreadDirectMax, are spread one by one, since in natural order the shuffles cost more than they save; the
// sort (three kernels, 15 us) is on the chain from kSortEachFrom points on only, see the session.  Whole iteration,
// exaggerated / settled, with the sort on the chain of every iteration: 5 000 points sorted 47 / 41 us, one by one 37 / 37;
// 20 011 points sorted 44 / 42, merged in natural order 41 / 41, one by one 57 / 42; 60 000 points sorted 54 / 49, natural
// order 61 / 49.  (Both kinds of small spread take blocks of two warps, which leave no SM idle, and the merge ends with the
// longest run.)
constexpr int kSpreadPerLane = 4;

__device__ __forceinline__ void spread_flush(float4 *__restrict__ w, int bx, int by, const float (&v)[kInterp][kInterp][4])
{
#pragma unroll
    for (int a = 0; a < kInterp; a++)
#pragma unroll
        for (int b = 0; b < kInterp; b++) {
            float4 *dst = w + (size_t)(bx * kInterp + a) * kG + (by * kInterp + b);
            atomicAdd(dst, make_float4(v[a][b][0], v[a][b][1], v[a][b][2], v[a][b][3]));
        }
}

// the counters of the next sort (a clear of its own would be one more node of the chain)
__device__ __forceinline__ void clear_histogram(int32_t *hist, int block, int blocks)
{
    for (int k = block * blockDim.x + threadIdx.x; k < kBoxes * kBoxes; k += blocks * blockDim.x) hist[k] = 0;
}

// What the first blocks of a small map's spread do: the first axis of the kernel's spectrum, which needs the bounding box like
// the spread and is needed by the kernel after it.  A stream of its own starts when the update has ended; this launch is on
// its way by then.
struct SpectrumRows {
    float *Rk;
    const float2 *tw;
    int blocks;   // 0: not here
};
constexpr int kSpreadSmallThreads = kSpecWarps * 32;

// hist (optional): the sort's counters, cleared here for the next one
// SPECTRUM: the first blocks have the spectrum's rows, with their twiddles in registers or read late.  The former leaves room
// for half as many blocks of points on an SM: an iteration at 20,011 / 30,011 / 60,000 / 100,000 points, exaggerated,
// 26.3 / 27.2 / 34.7 / 49.0 us, read late 26.8 / 27.7 / 34.2 / 47.9.
enum class SpreadSpectrum { none, late, registers };
template <int PER_LANE, SpreadSpectrum SPECTRUM>
__global__ void __launch_bounds__(PER_LANE == 1 ? kSpreadSmallThreads : 256)
spread_kernel(const float2 *Y2, long long row_lo, long long n_rows, const int32_t *order, const IterState *state, int slot, InterpConsts ic,
              float4 *w, int32_t *hist, SpectrumRows spec)
{
    int block = blockIdx.x, blocks = gridDim.x;
    if constexpr (SPECTRUM != SpreadSpectrum::none) {
        if (block < spec.blocks) {
            spectrum_rows<SPECTRUM == SpreadSpectrum::late>(spec.Rk, state, slot, spec.tw, block);
            return;
        }
        block -= spec.blocks;
        blocks -= spec.blocks;
    }
    after_previous();
    if (hist) clear_histogram(hist, block, blocks);
    const long long t0 = ((long long)block * blockDim.x + threadIdx.x) * PER_LANE;
    const int lane = threadIdx.x & 31;
    const GridGeom g = load_geom(state, slot);
    int key = -1, bx = 0, by = 0;
    float v[kInterp][kInterp][4];
#pragma unroll
    for (int a = 0; a < kInterp; a++)
#pragma unroll
        for (int b = 0; b < kInterp; b++)
#pragma unroll
            for (int c = 0; c < 4; c++) v[a][b][c] = 0.0f;
    // all loads of the lane first: they are independent of each other
    float2 ys[PER_LANE];
#pragma unroll
    for (int p = 0; p < PER_LANE; p++) {
        const long long t = t0 + p;
        if (t < n_rows) {
            const long long r = order ? (long long)order[t] : t;
            ys[p] = Y2[row_lo + r];
        }
    }
#pragma unroll
    for (int p = 0; p < PER_LANE; p++) {
        if (t0 + p >= n_rows) break;
        const float2 y = ys[p];
        int kx, ky;
        float Lx[kInterp], Ly[kInterp];
        axis_weights(y.x, g, ic, kx, Lx);
        axis_weights(y.y, g, ic, ky, Ly);
        const int k = ky * kBoxes + kx;
        if (k != key && key >= 0) {
            spread_flush(w, bx, by, v);
#pragma unroll
            for (int a = 0; a < kInterp; a++)
#pragma unroll
                for (int b = 0; b < kInterp; b++)
#pragma unroll
                    for (int c = 0; c < 4; c++) v[a][b][c] = 0.0f;
        }
        key = k; bx = kx; by = ky;
        const float c3 = y.x * y.x + y.y * y.y;
#pragma unroll
        for (int a = 0; a < kInterp; a++)
#pragma unroll
            for (int b = 0; b < kInterp; b++) {
                const float l = Lx[a] * Ly[b];
                v[a][b][0] += l * y.x; v[a][b][1] += l * y.y; v[a][b][2] += l; v[a][b][3] += l * c3;  // (x, y, count, r^2)
            }
    }
    // runs of equal keys among neighbouring lanes (their open runs)
    const int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const bool head = (lane == 0) || (key != prev);
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const unsigned above = (lane == 31) ? 0u : (heads & (0xffffffffu << (lane + 1)));
    const int run_end = above ? (__ffs(above) - 2) : 31;   // last lane of this lane's run
    if (heads != 0xffffffffu) {                             // at least one run longer than one lane
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const bool take = lane + d <= run_end;
            if (!__any_sync(0xffffffffu, take)) break;   // no run is that long
#pragma unroll
            for (int a = 0; a < kInterp; a++)
#pragma unroll
                for (int b = 0; b < kInterp; b++)
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const float o = __shfl_down_sync(0xffffffffu, v[a][b][c], d);
                        if (take) v[a][b][c] += o;
                    }
        }
    }
    if (head && key >= 0) spread_flush(w, bx, by, v);
}

// No order, no merging: a point per thread (few points, see kSpreadPerLane).
__global__ void __launch_bounds__(kSpreadSmallThreads)
spread_direct_kernel(const float2 *Y2, long long row_lo, long long n_rows, const IterState *state, int slot, InterpConsts ic, float4 *w, SpectrumRows spec)
{
    if (blockIdx.x < spec.blocks) {
        spectrum_rows<false>(spec.Rk, state, slot, spec.tw, blockIdx.x);
        return;
    }
    const long long t = (long long)(blockIdx.x - spec.blocks) * blockDim.x + threadIdx.x;
    after_previous();
    if (t >= n_rows) return;
    const float2 y = Y2[row_lo + t];
    const GridGeom g = load_geom(state, slot);
    int bx, by;
    float Lx[kInterp], Ly[kInterp];
    axis_weights(y.x, g, ic, bx, Lx);
    axis_weights(y.y, g, ic, by, Ly);
    const float c3 = y.x * y.x + y.y * y.y;
#pragma unroll
    for (int a = 0; a < kInterp; a++)
#pragma unroll
        for (int b = 0; b < kInterp; b++) {
            const float l = Lx[a] * Ly[b];
            atomicAdd(w + (size_t)(bx * kInterp + a) * kG + (by * kInterp + b), make_float4(l * y.x, l * y.y, l, l * c3));
        }
}

// ---- counting sort of the owned points by box (order[t] = local row index) ----
__global__ void order_identity_kernel(int32_t *order, long long n)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) order[t] = (int32_t)t;
}

// Both passes of the counting sort give a thread kOrderPerThread consecutive entries of the previous order,
// so that it has that many independent loads and atomics in flight (a pass is a chain of dependent L2
// round trips).  Atomics are combined across the warp: for each of its entries in turn, the lanes that
// hold the same key elect a leader that adds their number.  The points of a box are (nearly) contiguous in
// the previous order, so a warp sees few distinct keys.
constexpr int kOrderPerThread = 4;

__device__ __forceinline__ int point_key(const float2 *__restrict__ Y2, long long row, const GridGeom &g)
{
    const float2 y = Y2[row];
    return axis_box(y.y, g) * kBoxes + axis_box(y.x, g);
}

// keys[t] = box of point order[t]; hist[box] += 1; previous[t] = order[t] (the scatter writes `order` anew)
__global__ void __launch_bounds__(256)
order_histogram_kernel(const float2 *__restrict__ Y2, long long row_lo, long long n_rows, const int32_t *__restrict__ order,
                       const IterState *state, int slot, int32_t *__restrict__ keys, int32_t *__restrict__ hist, int32_t *__restrict__ previous)
{
    const long long t0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * kOrderPerThread;
    const int lane = threadIdx.x & 31;
    const GridGeom g = load_geom(state, slot);
    int k[kOrderPerThread] = {-1, -1, -1, -1};
    if (t0 + kOrderPerThread <= n_rows) {
        const int4 o = *reinterpret_cast<const int4 *>(order + t0);
        k[0] = point_key(Y2, row_lo + o.x, g);
        k[1] = point_key(Y2, row_lo + o.y, g);
        k[2] = point_key(Y2, row_lo + o.z, g);
        k[3] = point_key(Y2, row_lo + o.w, g);
        *reinterpret_cast<int4 *>(keys + t0) = make_int4(k[0], k[1], k[2], k[3]);
        *reinterpret_cast<int4 *>(previous + t0) = o;
    } else {
#pragma unroll
        for (int p = 0; p < kOrderPerThread; p++)
            if (t0 + p < n_rows) {
                const int32_t o = order[t0 + p];
                k[p] = point_key(Y2, row_lo + o, g);
                keys[t0 + p] = k[p];
                previous[t0 + p] = o;
            }
    }
#pragma unroll
    for (int p = 0; p < kOrderPerThread; p++) {
        const unsigned same = __match_any_sync(0xffffffffu, k[p]);
        if (k[p] >= 0 && lane == __ffs(same) - 1) atomicAdd(hist + k[p], __popc(same));
    }
}

// exclusive scan of the kBoxes^2 counters in place: one block, warp w owns the contiguous bins
// [w * kPerWarp, (w + 1) * kPerWarp) and walks them 32 at a time (coalesced), carrying its running total;
// one pass over the 32 warp totals gives every warp its offset
__global__ void __launch_bounds__(1024) order_scan_kernel(int32_t *hist)
{
    constexpr int kBins = kBoxes * kBoxes;
    constexpr int kPerWarp = (kBins + 31) / 32;
    constexpr int kRounds = (kPerWarp + 31) / 32;
    __shared__ int warp_tot[32];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    int v[kRounds], excl[kRounds];
#pragma unroll
    for (int j = 0; j < kRounds; j++) {
        const int off = j * 32 + lane, idx = wi * kPerWarp + off;
        v[j] = (off < kPerWarp && idx < kBins) ? hist[idx] : 0;
    }
    int carry = 0;
#pragma unroll
    for (int j = 0; j < kRounds; j++) {
        int incl = v[j];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        excl[j] = carry + incl - v[j];
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) warp_tot[wi] = carry;
    __syncthreads();
    if (wi == 0) {
        int t = warp_tot[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, t, d);
            if (lane >= d) t += o;
        }
        warp_tot[lane] = t;   // inclusive totals of the warps
    }
    __syncthreads();
    const int offset = wi > 0 ? warp_tot[wi - 1] : 0;
#pragma unroll
    for (int j = 0; j < kRounds; j++) {
        const int off = j * 32 + lane, idx = wi * kPerWarp + off;
        if (off < kPerWarp && idx < kBins) hist[idx] = excl[j] + offset;
    }
}

__global__ void __launch_bounds__(256)
order_scatter_kernel(const int32_t *__restrict__ order_in, const int32_t *__restrict__ keys, long long n_rows,
                     int32_t *__restrict__ cursor, int32_t *__restrict__ order_out)
{
    const long long t0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * kOrderPerThread;
    const int lane = threadIdx.x & 31;
    int k[kOrderPerThread] = {-1, -1, -1, -1}, o[kOrderPerThread] = {0, 0, 0, 0};
    if (t0 + kOrderPerThread <= n_rows) {
        const int4 kk = *reinterpret_cast<const int4 *>(keys + t0);
        const int4 oo = *reinterpret_cast<const int4 *>(order_in + t0);
        k[0] = kk.x; k[1] = kk.y; k[2] = kk.z; k[3] = kk.w;
        o[0] = oo.x; o[1] = oo.y; o[2] = oo.z; o[3] = oo.w;
    } else {
#pragma unroll
        for (int p = 0; p < kOrderPerThread; p++)
            if (t0 + p < n_rows) { k[p] = keys[t0 + p]; o[p] = order_in[t0 + p]; }
    }
    unsigned same[kOrderPerThread];
    int base[kOrderPerThread];
#pragma unroll
    for (int p = 0; p < kOrderPerThread; p++) {   // all the atomics first: their round trips overlap
        same[p] = __match_any_sync(0xffffffffu, k[p]);
        base[p] = 0;
        if (k[p] >= 0 && lane == __ffs(same[p]) - 1) base[p] = atomicAdd(cursor + k[p], __popc(same[p]));
    }
#pragma unroll
    for (int p = 0; p < kOrderPerThread; p++) {
        const int b = __shfl_sync(0xffffffffu, base[p], __ffs(same[p]) - 1);
        if (k[p] >= 0) order_out[b + __popc(same[p] & ((1u << lane) - 1u))] = o[p];
    }
}

// ------------------------------------------------------------------------------------------
// gather: repulsive force (unnormalised) from the potentials
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
gather_kernel(const float2 *__restrict__ Y2, long long row_lo, long long n_rows, const IterState *state, int slot,
              InterpConsts ic, const float4 *__restrict__ ytilde, float2 *__restrict__ Frep2)
{
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const GridGeom g = load_geom(state, slot);
    Frep2[row_lo + r] = repulsive_force(Y2[row_lo + r], g, ic, ytilde);
}

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

int launch_minmax_init(const float2 *Y2, int64_t N, IterState *state, int slot, cudaStream_t st)
{
    state_reset_kernel<<<1, 1, 0, st>>>(state, slot, 0);
    B200_CUDA(cudaGetLastError());
    if (N > 0) {
        const unsigned blocks = (unsigned)std::min<long long>(nblk(N, 256), 148 * 8);
        minmax_kernel<<<blocks, 256, 0, st>>>(Y2, N, state, slot);
        B200_CUDA(cudaGetLastError());
    }
    return 0;
}

int launch_state_reset(IterState *state, cudaStream_t st)
{
    state_reset_kernel<<<1, 1, 0, st>>>(state, 0, 1);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_state_swap(IterState *state, cudaStream_t st)
{
    state_swap_kernel<<<1, 1, 0, st>>>(state);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_spread(const float2 *Y2, int64_t row_lo, int64_t row_hi, const int32_t *order, int32_t *hist, const IterState *state,
                  int slot, InterpConsts ic, float4 *w, const FftWorkspace *spectrum, cudaStream_t st)
{
    const long long n = row_hi - row_lo;
    SpectrumRows spec = {nullptr, nullptr, 0};
    if (spectrum) spec = {spectrum->Rk, spectrum->tw, kSpecRowBlocks};
    if (spectrum && !spread_takes_spectrum(n)) return -1;
    if (n <= 0) return 0;
    if (!order && n <= kSpreadDirectMax)
        B200_CUDA(launch_chained(spread_direct_kernel, spec.blocks + nblk(n, kSpreadSmallThreads), kSpreadSmallThreads, 0, st, Y2, row_lo, n, state, slot, ic, w, spec));
    else if (n <= kSpreadSingleMax)
        B200_CUDA(launch_chained(!spectrum       ? spread_kernel<1, SpreadSpectrum::none>
                                 : n < kSortMin ? spread_kernel<1, SpreadSpectrum::registers>
                                                : spread_kernel<1, SpreadSpectrum::late>,
                                 spec.blocks + nblk(n, kSpreadSmallThreads), kSpreadSmallThreads, 0,
                                 st, Y2, row_lo, n, order, state, slot, ic, w, hist, spec));
    else
        B200_CUDA(launch_chained(spread_kernel<kSpreadPerLane, SpreadSpectrum::none>, nblk((n + kSpreadPerLane - 1) / kSpreadPerLane, 256), 256, 0, st, Y2, row_lo, n, order, state,
                                 slot, ic, w, hist, spec));
    return 0;
}

int launch_order_identity(int32_t *order, int64_t n, cudaStream_t st)
{
    if (n <= 0) return 0;
    order_identity_kernel<<<nblk(n, 256), 256, 0, st>>>(order, n);
    B200_CUDA(cudaGetLastError());
    return 0;
}

// `order` sorted anew by the box of the points' current position, in two parts: the first only reads it.  previous, keys: n
// ints of scratch each; hist: kBoxes^2 counters, zero on entry and used up afterwards (the spread clears them where it is told to).
int launch_order_count(const float2 *Y2, int64_t row_lo, int64_t row_hi, const int32_t *order, int32_t *previous, int32_t *keys, int32_t *hist,
                       const IterState *state, int slot, cudaStream_t st)
{
    const long long n = row_hi - row_lo;
    if (n <= 0) return 0;
    const long long n_thr = (n + kOrderPerThread - 1) / kOrderPerThread;
    order_histogram_kernel<<<nblk(n_thr, 256), 256, 0, st>>>(Y2, row_lo, n, order, state, slot, keys, hist, previous);
    B200_CUDA(cudaGetLastError());
    order_scan_kernel<<<1, 1024, 0, st>>>(hist);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_order_scatter(int64_t n, int32_t *order, const int32_t *previous, const int32_t *keys, int32_t *hist, cudaStream_t st)
{
    if (n <= 0) return 0;
    const long long n_thr = (n + kOrderPerThread - 1) / kOrderPerThread;
    order_scatter_kernel<<<nblk(n_thr, 256), 256, 0, st>>>(previous, keys, n, hist, order);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_gather(const float2 *Y2, int64_t row_lo, int64_t row_hi, const IterState *state, int slot, InterpConsts ic,
                  const float4 *ytilde, float2 *Frep2, cudaStream_t st)
{
    const long long n = row_hi - row_lo;
    if (n <= 0) return 0;
    gather_kernel<<<nblk(n, 256), 256, 0, st>>>(Y2, row_lo, n, state, slot, ic, ytilde, Frep2);
    B200_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace b200
