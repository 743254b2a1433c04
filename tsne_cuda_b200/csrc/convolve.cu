// Convolution of the charge grid with the squared-Cauchy kernel (reference: kernel evaluation
// src/kernels/nbodyfft.cu:175-203, cuFFT convolution :3-41 and :395-424).
//
// The linear convolution of two 390-node axes fits any cyclic one of at least 779 points; this one has 784 = 28 x 28,
// the next length that splits evenly over a warp: 28 lanes hold 28 values each, transform them in registers (28 = 4 x 7
// without twiddles between the factors), exchange through shared memory once, and transform again.
//
//  * The four charge grids travel as two complex planes (x, y) and (count, r^2); convolving with a real kernel acts on
//    real and imaginary parts independently, so nothing is unpacked.  A complex FFT leaks rounding error of the larger
//    component into the smaller one, so the x and y charges (same magnitude) share a plane and the r^2 charge is scaled
//    by a power of two to the magnitude of the counts it travels with (exact, undone on the way out).
//  * Only the 390 non-zero rows are transformed on the way in and the 390 needed rows on the way out, and in every
//    one-dimensional transform the fourteen leading registers of a lane hold all of the input (forward) or all of the
//    wanted output (inverse): the other half of the butterflies is left out at compile time.
//  * The kernel is centred at index 0 and even in both axes, so its spectrum is real and even.  It depends on the
//    embedding through the box width alone: its first axis is transformed beside the spread (in the same launch where the map is
//    small, on a stream of its own where the spread is long), its second axis by blocks of the row pass that find SMs idle.
//    Two real columns share a complex transform, and the spectrum of column c serves column 784 - c as well.
//  * Column c, its mirror image 784 - c, and both planes are one block of the column pass, and the product with the spectrum
//    never leaves the SM.  Between the passes four rows of these four columns are one line of 128 bytes: a block of the row
//    passes has four rows, and every block reads and writes whole lines.
//  * The last pass also sums the normalisation on the grid: sum_i Z_i is the bilinear form of charges and potentials
//    (each point's Z_i is interpolated from the potentials with the weights its charges were spread with), so it needs
//    neither a pass over the points nor an exchange between ranks that hold the summed grid.
//
// Bound: three kernels whose blocks each run once: the loads at their start, an exchange and the stores at their end take as
// long as the transforms, and in those the fp32 pipe is three quarters busy (columns pass: 4,900 cycles of packed and scalar
// arithmetic per scheduler in 6,500).  Measured on B200 inside an iteration of 5,000 points (clock stamps): rows 3.3, columns 4.9,
// rows back 4.6 us, and 0.7 to 1.1 us between two of them.  What that came from, per iteration at 1,500 / 5,000 / 20,011 points:
//   a row per block in the row passes (the column pass read and wrote 32 bytes of a line: every access of a warp touched 28
//   different lines), scalar arithmetic, the spectrum in two kernels on a third stream                   31.1 / 32.1 / 34.4 us
//   four rows per block and whole lines between the passes, packed arithmetic                            29.1 / 29.4 / 31.2
//   the spectrum's second axis beside the rows (it was what the column pass waited for, 1.5 us)          27.7 / 27.9 / 31.3
//   copies in the order of their use; point kernels of small blocks (repulsive.cu, update.cu)            27.5 / 28.1 / 31.4
//   chained launches, the spectrum's first axis beside the spread, loads before arithmetic in update.cu  24.0 / 24.1 / 26.9
//   three blocks of the column pass to an SM where that places all of them                               23.0 / 23.4 / 27.1
//   a lane's twiddles in registers, loaded before the kernel in front has ended                          21.7 / 22.2 / 26.1
// A warp's transforms are 750 instructions in 2,800 cycles whether two or three of them share a scheduler, so blocks of three
// rows on 130 SMs instead of four on 98 gained nothing (22.9 -> 23.3: the columns then meet bank conflicts).
// Chained launches gain nothing where the next kernel may start too early: blocks of the column pass that are placed while
// rows still run share the SMs unevenly (27.8 -> 29.0 with the permission at the start of each kernel, 26.7 at its end, 26.4
// before its last stores).
// Rounding: the repulsive force is as far from float64 as with the 1024-point transforms (1e-7 to 4e-7 of its norm for compact
// maps, 7e-6 at spread 10); the sum of Z 1e-7 to 3e-7 for compact maps, where it was 0.5e-7 to 1.5e-7, and the same elsewhere.
#include "fft784.cuh"

#include <math.h>

namespace b200 {
namespace {

__global__ void twiddle_init_kernel(float2 *tw)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kM) {
        double s, c;
        sincospi(-2.0 * (double)((i / kR) * (i % kR)) / (double)kM, &s, &c);
        tw[i] = make_float2((float)c, (float)s);
    }
}

// where the four transforms of column pair c stand in a row of the workspace: plane 0 at c, plane 0 at its mirror image
// 784 - c, plane 1 at c, plane 1 at the mirror image (columns 0 and 392 are their own image: those slots stay unused)
__device__ __forceinline__ int column_of(int k) { return k < kC ? k : kM - k; }
__device__ __forceinline__ int slot_of(int k) { return k < kC ? 0 : 1; }

__global__ void __launch_bounds__(kSpecWarps * 32)
spectrum_rows_kernel(float *Rk, const IterState *state, int slot, const float2 *__restrict__ tw)
{
    spectrum_rows<false>(Rk, state, slot, tw, blockIdx.x);
}

// ---- workspace between the passes ----
// Column pair c (a column, its mirror image, both planes: q = 0 .. 3) and four rows are a line of 128 bytes; the lines of a
// column pair follow one another.  A block of the row passes has four rows, so it writes or reads whole lines, and a block of
// the column pass has one column pair: 12.5 KB in one piece.  Inside its line the place of (row, q) turns with the line, so
// that a half warp that reads one q of sixteen rows meets sixteen bank pairs.
constexpr int kRowsBlock = 4, kLines = (kG + kRowsBlock - 1) / kRowsBlock, kLine = 4 * kRowsBlock;   // kLine: float2
static_assert(kLines * kRowsBlock == kR * kHalf, "rows beyond the grid are the zeros of a transform");
__device__ __forceinline__ int place_in_line(int q, int line, int row) { return kRowsBlock * ((q + line) & 3) + (row & (kRowsBlock - 1)); }
constexpr int kStageLine = kLine + 2;   // float2 per line in shared memory of the row passes: columns apart in their banks

constexpr int kRowThreads = 2 * kRowsBlock * 32;   // a warp per row and plane
constexpr size_t kStageBytes = sizeof(float2) * kC * kStageLine, kRowExBytes = sizeof(float2) * 2 * kRowsBlock * kEx;
constexpr size_t kRowsSmem = kStageBytes > kRowExBytes ? kStageBytes : kRowExBytes;
constexpr size_t kBackSmem = kRowsSmem + sizeof(float4) * kRowsBlock * kG;

// ---- spectrum, second axis: sixteen columns per block, two real ones per warp; Kh[c][k] ----
constexpr int kSpecCols = 2 * kRowThreads / 32, kSpecBlocks = kRkStride / kSpecCols;
constexpr int kSpecRow = kSpecCols + 4;   // floats per row in shared memory
static_assert(kRkStride % kSpecCols == 0 && kSpecBlocks * kSpecCols >= kC, "columns of the spectrum");
static_assert(sizeof(float) * kG * kSpecRow <= kStageBytes, "the columns fit where the lines are staged");
__device__ __forceinline__ void spectrum_columns(float2 *smem, const float *Rk, float *Kh, const float2 *__restrict__ tw, int block)
{
    float2 *ex = smem + (threadIdx.x >> 5) * kEx;
    float *cols = reinterpret_cast<float *>(smem);   // before the exchange
    const int lane = threadIdx.x & 31, own = 2 * (threadIdx.x >> 5), c = kSpecCols * block + own;
    Twiddles t;
    load_twiddles(t, tw, lane);
    after_previous();
    for (int u = threadIdx.x; u < kG * kSpecCols / 4; u += kRowThreads) {
        const int row = u / (kSpecCols / 4), part = u % (kSpecCols / 4);
        copy16(cols + row * kSpecRow + 4 * part, Rk + (size_t)row * kRkStride + kSpecCols * block + 4 * part);
    }
    end_batch();
    copies_done<0>();
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int row = kR * r + lane;
        v[r] = (lane < kR && row < kG) ? *reinterpret_cast<const float2 *>(cols + row * kSpecRow + own) : make_float2(0.0f, 0.0f);
    }
    mirror_input(v, lane);
    fft784_warp<false, kR>(v, ex, t, lane, [] { __syncthreads(); });   // the columns have been read
    let_next_start();
    if (c >= kC || lane >= kR) return;
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const int k = kR * r + lane;
        Kh[(size_t)c * kM + k] = v[r].x;
        if (c + 1 < kC) Kh[(size_t)(c + 1) * kM + k] = v[r].y;
    }
}

// ---- first pass: four rows of the charge grid, both planes; the blocks after those take the spectrum's second axis, on SMs
// that would idle ----
__global__ void __launch_bounds__(kRowThreads)
fft_rows_forward_kernel(const float4 *w, float4 *A, const float *Rk, float *Kh, const IterState *state, int slot, const float2 *__restrict__ tw)
{
    extern __shared__ __align__(16) float2 smem[];
    if (blockIdx.x >= kLines) {
        spectrum_columns(smem, Rk, Kh, tw, blockIdx.x - kLines);
        return;
    }
    float2 *stage = smem;   // the lines, once the exchange is over
    const int lane = threadIdx.x & 31, plane = (threadIdx.x >> 5) & 1, row = kRowsBlock * blockIdx.x + (threadIdx.x >> 6);
    Twiddles t;
    load_twiddles(t, tw, lane);
    after_previous();
    const float2 *wrow = reinterpret_cast<const float2 *>(w + (size_t)row * kG) + plane;   // .xy or .zw of each node
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int j = kR * r + lane;
        v[r] = (lane < kR && j < kG && row < kG) ? wrow[2 * j] : make_float2(0.0f, 0.0f);
    }
    const float imag_scale = plane == 1 ? load_geom(state, slot).r2_scale : 1.0f;
#pragma unroll
    for (int r = 0; r < kHalf; r++) v[r].y *= imag_scale;
    fft784_warp<false, kHalf>(v, stage + (threadIdx.x >> 5) * kEx, t, lane, [] {});
    let_next_start();
    __syncthreads();
    if (lane < kR) {
#pragma unroll
        for (int r = 0; r < kR; r++) {
            const int k = kR * r + lane;
            stage[column_of(k) * kStageLine + place_in_line(2 * plane + slot_of(k), blockIdx.x, row)] = v[r];
        }
    }
    __syncthreads();
#pragma unroll 4
    for (int u = threadIdx.x; u < kC * kLine / 2; u += kRowThreads) {
        const int c = u / (kLine / 2), part = u % (kLine / 2);
        A[((size_t)c * kLines + blockIdx.x) * (kLine / 2) + part] = *reinterpret_cast<const float4 *>(stage + c * kStageLine + 2 * part);
    }
}

// ---- second pass: column c, its mirror image, both planes: forward, product with the spectrum, inverse ----
constexpr size_t kColsSmem = sizeof(float2) * (4 * kEx + kLines * kLine) + sizeof(float) * kM;
// What a block asks for where three to an SM are all there: the blocks come while the rows end, and the SMs that are free by
// then would take four (1,500 / 5,000 points 24.0 -> 22.9 / 24.4 -> 23.5 us an iteration; with fewer SMs, of which some
// have to take four, 20,011 points 27.2 -> 29.7).
constexpr size_t kColsSmemThree = 72 * 1024;
static_assert(kColsSmem <= kColsSmemThree && 4 * kColsSmemThree > 227 * 1024 && 3 * (kColsSmemThree + 1024) <= 227 * 1024, "three blocks to an SM");
__global__ void __launch_bounds__(128)
fft_columns_kernel(const float4 *A, const float *Kh, float4 *B, const float2 *__restrict__ tw)
{
    extern __shared__ __align__(16) float2 smem[];
    float2 *ex = smem + (threadIdx.x >> 5) * kEx, *lines = smem + 4 * kEx;
    float *spec = reinterpret_cast<float *>(lines + kLines * kLine);
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5, c = blockIdx.x;
    constexpr int n4 = kLines * kLine / 2;
    Twiddles t;
    load_twiddles(t, tw, lane);
    after_previous();
    copy_floats<128>(reinterpret_cast<float *>(lines), reinterpret_cast<const float *>(A + (size_t)c * n4), n4);
    end_batch();
    copy_floats<128>(spec, Kh + (size_t)c * kM, kM / 4);
    end_batch();
    copies_done<1>();
    const int sl = min(lane, kR - 1);
    float2 *mine = lines + (sl / kRowsBlock) * kLine;   // rows 28 r + lane: 7 r lines further on; a warp has its q to itself
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        v[r] = mine[r * (kR / kRowsBlock) * kLine + place_in_line(q, r * (kR / kRowsBlock) + sl / kRowsBlock, sl)];
    }
    fft784_warp<false, kHalf>(v, ex, t, lane, [] {});
    copies_done<0>();
#pragma unroll
    for (int r = 0; r < kR; r++) v[r] = times(spec[kR * r + sl], v[r]);
    fft784_warp<true, kR>(v, ex, t, lane, [] {});
    let_next_start();
    if (lane < kR) {
#pragma unroll
        for (int r = 0; r < kHalf; r++) mine[r * (kR / kRowsBlock) * kLine + place_in_line(q, r * (kR / kRowsBlock) + sl / kRowsBlock, sl)] = v[r];
    }
    __syncthreads();
    float4 *dst = B + (size_t)c * n4;
    const float4 *out = reinterpret_cast<const float4 *>(lines);
#pragma unroll
    for (int u = threadIdx.x; u < n4; u += 128) dst[u] = out[u];
}

// ---- third pass: four rows of potentials, both planes; the grid's share of sum_i Z_i ----
__global__ void __launch_bounds__(kRowThreads)
fft_rows_inverse_kernel(const float4 *B, float4 *w, float4 *ytilde, IterState *state, int slot, const float2 *__restrict__ tw, int zero_w)
{
    extern __shared__ __align__(16) float2 smem[];
    float2 *stage = smem;   // the lines, before the exchange
    float4 *charges = reinterpret_cast<float4 *>(smem) + (kBackSmem - sizeof(float4) * kRowsBlock * kG) / sizeof(float4);
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5, plane = wi & 1, row = kRowsBlock * blockIdx.x + (wi >> 1);
    Twiddles t;
    load_twiddles(t, tw, lane);
    after_previous();
    for (int u = threadIdx.x; u < kC * kLine / 2; u += kRowThreads) {
        const int c = u / (kLine / 2), part = u % (kLine / 2);
        copy16(stage + c * kStageLine + 2 * part, B + ((size_t)c * kLines + blockIdx.x) * (kLine / 2) + part);
    }
    end_batch();
    float4 *wrows = w + (size_t)kRowsBlock * blockIdx.x * kG;
    const int nodes = min(kRowsBlock, kG - kRowsBlock * (int)blockIdx.x) * kG;
    for (int j = threadIdx.x; j < nodes; j += kRowThreads) copy16(charges + j, wrows + j);
    end_batch();
    const float scale = 1.0f / ((float)kM * (float)kM);
    const float imag_scale = plane == 1 ? scale * load_geom(state, slot).r2_unscale : scale;
    copies_done<1>();
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const int k = kR * r + min(lane, kR - 1);
        v[r] = stage[column_of(k) * kStageLine + place_in_line(2 * plane + slot_of(k), blockIdx.x, row)];
    }
    fft784_warp<true, kR>(v, stage + wi * kEx, t, lane, [] { __syncthreads(); });   // the lines have been read
    let_next_start();
    copies_done<0>();
    if (zero_w)
        for (int j = threadIdx.x; j < nodes; j += kRowThreads) wrows[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float2 *out = reinterpret_cast<float2 *>(ytilde + (size_t)row * kG) + plane;
    const float4 *charge = charges + (wi >> 1) * kG;
    double z = 0.0;
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int j = kR * r + lane;
        if (lane < kR && j < kG && row < kG) {
            const float2 p = make_float2(v[r].x * scale, v[r].y * imag_scale);
            out[2 * j] = p;
            // node = (x, y, count, r^2) charges and potentials:
            // pot.count (w.count + w.r2) - 2 (pot.x w.x + pot.y w.y) + pot.r2 w.count
            // The two planes' terms are of order |y|^2 and cancel down to Z: products and sums in double.
            const float2 q = reinterpret_cast<const float2 *>(charge + j)[plane];
            const double px = p.x, py = p.y, qx = q.x, qy = q.y;
            z += plane == 0 ? -2.0 * fma(px, qx, py * qy) : fma(px, qx + qy, py * qx);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    __shared__ double zs[2 * kRowsBlock];
    if (lane == 0) zs[wi] = z;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 1; k < 2 * kRowsBlock; k++) z += zs[k];
        atomicAdd(&state->zsum[slot], z);
        if (blockIdx.x == 0) {   // recycle the other slot's min/max and this slot's norm for this iteration's update
            state->min_enc[slot ^ 1] = 0xffffffffu;
            state->max_enc[slot ^ 1] = 0u;
            state->unorm2[slot] = 0.0;
        }
    }
}

}  // namespace

size_t fft_workspace_bytes()
{
    return sizeof(float2) * (size_t)kC * kLines * kLine * 2 + sizeof(float) * ((size_t)kG * kRkStride + (size_t)kC * kM) + sizeof(float2) * kM;
}

int fft_workspace_init(FftWorkspace *ws, void *mem, cudaStream_t st)
{
    char *p = static_cast<char *>(mem);
    ws->A = reinterpret_cast<float4 *>(p); p += sizeof(float2) * (size_t)kC * kLines * kLine;
    ws->B = reinterpret_cast<float4 *>(p); p += sizeof(float2) * (size_t)kC * kLines * kLine;
    ws->tw = reinterpret_cast<float2 *>(p); p += sizeof(float2) * kM;
    ws->Kh = reinterpret_cast<float *>(p); p += sizeof(float) * (size_t)kC * kM;
    ws->Rk = reinterpret_cast<float *>(p);
    B200_CUDA(cudaFuncSetAttribute(fft_rows_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsSmem));
    B200_CUDA(cudaFuncSetAttribute(fft_rows_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBackSmem));
    B200_CUDA(cudaFuncSetAttribute(fft_columns_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kColsSmemThree));
    twiddle_init_kernel<<<(kM + 255) / 256, 256, 0, st>>>(ws->tw);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_kernel_spectrum(const IterState *state, int slot, const FftWorkspace &ws, cudaStream_t st)
{
    spectrum_rows_kernel<<<kSpecRowBlocks, kSpecWarps * 32, 0, st>>>(ws.Rk, state, slot, ws.tw);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_convolve_rows(const float4 *w, const IterState *state, int slot, const FftWorkspace &ws, cudaStream_t st)
{
    B200_CUDA(launch_chained(fft_rows_forward_kernel, kLines + kSpecBlocks, kRowThreads, kRowsSmem, st, w, ws.A, ws.Rk, ws.Kh, state, slot, ws.tw));
    return 0;
}

int launch_convolve(float4 *w, float4 *ytilde, IterState *state, int slot, const FftWorkspace &ws, bool zero_w, int free_sms, cudaStream_t st)
{
    B200_CUDA(launch_chained(fft_columns_kernel, kC, 128, 3 * free_sms >= kC ? kColsSmemThree : kColsSmem, st, ws.A, ws.Kh, ws.B, ws.tw));
    B200_CUDA(launch_chained(fft_rows_inverse_kernel, kLines, kRowThreads, kBackSmem, st, ws.B, w, ytilde, state, slot, ws.tw, zero_w ? 1 : 0));
    return 0;
}

}  // namespace b200
