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
//    embedding through the box width alone: two small kernels (spectrum_rows, spectrum_columns) prepare it on a stream of
//    their own while the points are sorted and spread.  Two real columns share a complex transform, and the spectrum of
//    column c serves column 784 - c as well.
//  * Column c, its mirror image 784 - c, and both planes are one block of the column pass, and the product with the spectrum
//    never leaves the SM.  Between the passes four rows of these four columns are one line of 128 bytes: a block of the row
//    passes has four rows, and every block reads and writes whole lines.
//  * The last pass also sums the normalisation on the grid: sum_i Z_i is the bilinear form of charges and potentials
//    (each point's Z_i is interpolated from the potentials with the weights its charges were spread with), so it needs
//    neither a pass over the points nor an exchange between ranks that hold the summed grid.
//
// Bound: three kernels whose blocks each run once: the loads at their start, an exchange and the stores at their end take as
// long as the transforms, and in those the fp32 pipe is three quarters busy (columns pass: 4,900 cycles of packed and scalar
// arithmetic per scheduler in 6,500).  Measured on B200 inside an iteration of 5,000 points: rows 5.1, columns 6.9, rows
// back 6.2 us.  With a row (390 blocks of two warps) as the unit of the row passes, so that the column pass read and wrote
// 32 bytes per row (every load and store of a warp 28 different lines), and scalar arithmetic: 4.8, 9.8, 6.2.  Iteration at
// 1,500 / 5,000 / 20,011 points 31.1 -> 29.1, 32.1 -> 29.4, 34.4 -> 31.2 us; 60,000 exaggerated 46.2 -> 43.9.
// Rounding: the repulsive force is as far from float64 as with the 1024-point transforms (1e-7 to 4e-7 of its norm for compact
// maps, 7e-6 at spread 10); the sum of Z 1e-7 to 3e-7 for compact maps, where it was 0.5e-7 to 1.5e-7, and the same elsewhere.
#include "grid_geom.cuh"

#include <math.h>

#include <algorithm>

namespace b200 {
namespace {

constexpr int kR = 28;                       // kM = kR * kR
constexpr int kHalf = kR / 2;                // registers that hold a 390-point input or output: 28 * 14 >= 390
constexpr int kC = kM / 2 + 1;               // distinct columns of an even spectrum: 0 .. 392
constexpr int kRkStride = (kC + 15) / 16 * 16;   // row of Rk: whole groups of the columns that a block of the second axis takes
constexpr int kExStride = kR + 1;            // float2 per row of the exchange buffer (odd: no bank conflicts)
constexpr int kEx = kR * kExStride;
static_assert(kM == kR * kR && kM >= 2 * kG - 1 && kR * kHalf >= kG && kR * (kHalf - 1) < kG, "transform length");

// Sums and products with a real coefficient act on both halves of a complex number alike: one packed instruction each, with
// the results of the two it stands for.  The fp32 pipe is as fast either way; the issue slots go to everything else.
__device__ __forceinline__ uint64_t pack(float2 a)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 unpack(uint64_t r)
{
    float2 a;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
    return a;
}
__device__ __forceinline__ float2 operator+(float2 a, float2 b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack(a)), "l"(pack(b)));
    return unpack(r);
}
// a + c * t, a real coefficient
__device__ __forceinline__ float2 axpy(float c, float2 t, float2 a)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack(make_float2(c, c))), "l"(pack(t)), "l"(pack(a)));
    return unpack(r);
}
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return axpy(-1.0f, b, a); }
__device__ __forceinline__ float2 times(float c, float2 t)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack(make_float2(c, c))), "l"(pack(t)));
    return unpack(r);
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a plus or minus b turned by -90 degrees (forward) or +90 (inverse)
template <bool INV> __device__ __forceinline__ float2 add_turned(float2 a, float2 b) { return INV ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, a.y - b.x); }
template <bool INV> __device__ __forceinline__ float2 sub_turned(float2 a, float2 b) { return add_turned<!INV>(a, b); }

// Seven-point transform, natural order.  Z1..Z6: the input of that index is zero.
template <bool INV, bool Z0, bool Z1, bool Z2, bool Z3, bool Z4, bool Z5, bool Z6> __device__ __forceinline__ void dft7(float2 (&v)[7])
{
    constexpr float c1 = 0.62348980185873353f, c2 = -0.22252093395631440f, c3 = -0.90096886790241913f;   // cos(2 pi j / 7)
    constexpr float s1 = 0.78183148246802981f, s2 = 0.97492791218182361f, s3 = 0.43388373911755812f;     // sin(2 pi j / 7)
    const float2 zero = make_float2(0.0f, 0.0f);
    // sums and differences of the pairs (j, 7 - j); a missing partner costs nothing
    const float2 t1 = Z6 ? v[1] : (Z1 ? v[6] : v[1] + v[6]), d1 = Z6 ? v[1] : (Z1 ? zero - v[6] : v[1] - v[6]);
    const float2 t2 = Z5 ? v[2] : (Z2 ? v[5] : v[2] + v[5]), d2 = Z5 ? v[2] : (Z2 ? zero - v[5] : v[2] - v[5]);
    const float2 t3 = Z4 ? v[3] : (Z3 ? v[4] : v[3] + v[4]), d3 = Z4 ? v[3] : (Z3 ? zero - v[4] : v[3] - v[4]);
    constexpr bool none1 = Z1 && Z6, none2 = Z2 && Z5, none3 = Z3 && Z4;
    float2 a1 = Z0 ? zero : v[0], a2 = a1, a3 = a1, sum = a1, b1 = zero, b2 = zero, b3 = zero;
    if (!none1) {
        sum = Z0 ? t1 : sum + t1;
        a1 = axpy(c1, t1, a1); a2 = axpy(c2, t1, a2); a3 = axpy(c3, t1, a3);
        b1 = times(s1, d1); b2 = times(s2, d1); b3 = times(s3, d1);
    }
    if (!none2) {
        sum = sum + t2;
        a1 = axpy(c2, t2, a1); a2 = axpy(c3, t2, a2); a3 = axpy(c1, t2, a3);
        b1 = axpy(s2, d2, b1); b2 = axpy(-s3, d2, b2); b3 = axpy(-s1, d2, b3);
    }
    if (!none3) {
        sum = sum + t3;
        a1 = axpy(c3, t3, a1); a2 = axpy(c1, t3, a2); a3 = axpy(c2, t3, a3);
        b1 = axpy(s3, d3, b1); b2 = axpy(-s1, d3, b2); b3 = axpy(s2, d3, b3);
    }
    v[0] = sum;
    v[1] = add_turned<INV>(a1, b1); v[6] = sub_turned<INV>(a1, b1);
    v[2] = add_turned<INV>(a2, b2); v[5] = sub_turned<INV>(a2, b2);
    v[3] = add_turned<INV>(a3, b3); v[4] = sub_turned<INV>(a3, b3);
}

// input b of the a-th seven-point transform of fft28 is one of the zeros
__host__ __device__ constexpr bool zero_at(int a, int b, int nz) { return (7 * a + 4 * b) % 28 >= nz; }

// 28-point transform in registers, natural order in and out, by the coprime factors 4 and 7: input index
// (7 a + 4 b) mod 28, output index (21 ka + 8 kb) mod 28.  NZ: inputs from NZ on are zero.
template <bool INV, int NZ> __device__ __forceinline__ void fft28(float2 (&v)[kR])
{
    float2 y[4][7];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 7; b++) y[a][b] = v[(7 * a + 4 * b) % 28];
    dft7<INV, zero_at(0, 0, NZ), zero_at(0, 1, NZ), zero_at(0, 2, NZ), zero_at(0, 3, NZ), zero_at(0, 4, NZ), zero_at(0, 5, NZ), zero_at(0, 6, NZ)>(y[0]);
    dft7<INV, zero_at(1, 0, NZ), zero_at(1, 1, NZ), zero_at(1, 2, NZ), zero_at(1, 3, NZ), zero_at(1, 4, NZ), zero_at(1, 5, NZ), zero_at(1, 6, NZ)>(y[1]);
    dft7<INV, zero_at(2, 0, NZ), zero_at(2, 1, NZ), zero_at(2, 2, NZ), zero_at(2, 3, NZ), zero_at(2, 4, NZ), zero_at(2, 5, NZ), zero_at(2, 6, NZ)>(y[2]);
    dft7<INV, zero_at(3, 0, NZ), zero_at(3, 1, NZ), zero_at(3, 2, NZ), zero_at(3, 3, NZ), zero_at(3, 4, NZ), zero_at(3, 5, NZ), zero_at(3, 6, NZ)>(y[3]);
#pragma unroll
    for (int kb = 0; kb < 7; kb++) {
        const float2 p = y[0][kb] + y[2][kb], m = y[0][kb] - y[2][kb];
        const float2 q = y[1][kb] + y[3][kb], r = y[1][kb] - y[3][kb];
        v[(8 * kb) % 28] = p + q;
        v[(21 + 8 * kb) % 28] = add_turned<INV>(m, r);
        v[(42 + 8 * kb) % 28] = p - q;
        v[(63 + 8 * kb) % 28] = sub_turned<INV>(m, r);
    }
}

// Everything a block needs besides the values of its own transforms goes to shared memory with asynchronous copies, all
// in flight at once: a loop of loads and stores waits for L2 once per round (seven to thirteen rounds here), which cost
// more than the transforms.
__device__ __forceinline__ void copy16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// What is needed first is a batch of its own: copies arrive at 64 bytes a cycle, and the transform starts on the first batch.
__device__ __forceinline__ void end_batch() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LATER> __device__ __forceinline__ void copies_done()   // all but the last LATER batches are there, for the whole block
{
    asm volatile("cp.async.wait_group %0;" ::"n"(LATER) : "memory");
    __syncthreads();
}
template <int THREADS> __device__ __forceinline__ void copy_floats(float *dst, const float *__restrict__ src, int n4)   // n4 times four
{
    for (int k = threadIdx.x; k < n4; k += THREADS) copy16(dst + 4 * k, src + 4 * k);
}
template <int THREADS> __device__ __forceinline__ void copy_twiddles(float2 *tws, const float2 *__restrict__ tw)
{
    copy_floats<THREADS>(reinterpret_cast<float *>(tws), reinterpret_cast<const float *>(tw), kM / 2);
}

// 784-point transform by one warp.  In: lane l < 28 holds x[28 r + l] in v[r] (zero from r = NZ on).  Out: lane l holds
// X[l + 28 r] in v[r], the same pattern.  ex: kEx float2 of this warp; tws[k * 28 + l] = e^{-2 pi i k l / 784}, there
// when twiddles_ready() returns.
template <bool INV, int NZ, class READY>
__device__ __forceinline__ void fft784_warp(float2 (&v)[kR], float2 *ex, const float2 *tws, int lane, READY twiddles_ready)
{
    fft28<INV, NZ>(v);
    twiddles_ready();
    if (lane < kR) {
        ex[lane] = v[0];
#pragma unroll
        for (int k = 1; k < kR; k++) {
            float2 w = tws[k * kR + lane];
            if (INV) w.y = -w.y;
            ex[k * kExStride + lane] = cmul(v[k], w);
        }
    }
    __syncwarp();
    const float2 *row = ex + min(lane, kR - 1) * kExStride;
#pragma unroll
    for (int n = 0; n < kR; n++) v[n] = row[n];
    __syncwarp();
    fft28<INV, kR>(v);
}

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

// ---- spectrum of the kernel, first axis: a row per warp.  Two rows could share a transform, but a lane then evaluates 28
// values instead of 14, and the evaluation is as long as the transform: settled iteration at 1,500 / 20,011 / 45,000 points
// 32.8 / 35.0 / 39.0 us with two rows, 32.2 / 34.6 / 38.2 with one. ----
__device__ __forceinline__ float kernel_value(int row, int j, float h, float cmin)
{
    // node coordinates in float exactly as the reference forms them, summed and inverted in double (nbodyfft.cu:175-195)
    const float x1 = cmin + h / 2, y1 = cmin + h / 2 + row * h, y2 = cmin + h / 2 + j * h;
    const float da = x1 - y1, db = x1 - y2;
    const double s = 1.0 + (double)(da * da) + (double)(db * db), t = s * s;
    // 1 / t by two Newton-Raphson steps from the float reciprocal (off by less than 2^-21): 2^-42, then 2^-84 and one rounding,
    // so the double that a division gives unless 1 / t lies within 2^-31 of an ulp of a tie.  Beyond the range of floats
    // scaled by a power of two.  No branch: a lane's values are independent, and a branch in each (a division's special cases,
    // a range check) puts them in one chain.
    const bool big = t > 1e37;
    const double ts = big ? t * 0x1p-160 : t;
    const double r = (double)__fdividef(1.0f, (float)ts), r1 = fma(r, fma(-ts, r, 1.0), r), r2 = fma(r1, fma(-ts, r1, 1.0), r1);
    return (float)(t > 1e78 ? 0.0 : big ? r2 * 0x1p-160 : r2);
}
// completes a lane's half of an even sequence: v[r], r < 14, holds x[28 r + l]; the rest is x[784 - (28 r + l)]
__device__ __forceinline__ void mirror_input(float2 (&v)[kR], int lane)
{
    const int from = (kR - lane) % kR;
#pragma unroll
    for (int r = kHalf; r < kR; r++) {
        float2 m;                     // lanes 1..27: register 27 - r of lane 28 - l
        m.x = __shfl_sync(0xffffffffu, v[kR - 1 - r].x, from & 31);
        m.y = __shfl_sync(0xffffffffu, v[kR - 1 - r].y, from & 31);
        // lane 0: its own register 28 - r (register 14 would be node 392: beyond the grid)
        const float2 own = r == kHalf ? make_float2(0.0f, 0.0f) : v[kR - r];
        v[r] = lane == 0 ? own : m;
    }
}

constexpr int kSpecWarps = 2;
__global__ void __launch_bounds__(kSpecWarps * 32)
spectrum_rows_kernel(float *__restrict__ Rk, const IterState *state, int slot, const float2 *__restrict__ tw)
{
    __shared__ __align__(16) float2 tws[kM];
    __shared__ float2 exch[kSpecWarps][kEx];
    copy_twiddles<kSpecWarps * 32>(tws, tw);
    end_batch();
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const int row = blockIdx.x * kSpecWarps + wi;
    const GridGeom g = load_geom(state, slot);
    const float h = g.box_width / (float)kInterp;
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int j = kR * r + lane;
        const bool in = lane < kR && j < kG;
        const float value = kernel_value(row, j, h, g.cmin);   // evaluated in all lanes: no branch around it
        v[r] = make_float2(in ? value : 0.0f, 0.0f);
    }
    mirror_input(v, lane);
    fft784_warp<false, kR>(v, exch[wi], tws, lane, copies_done<0>);
    if (row >= kG || lane >= kR) return;
#pragma unroll
    for (int r = 0; r <= kHalf; r++) {
        const int k = kR * r + lane;
        if (k < kRkStride) {
            Rk[(size_t)row * kRkStride + k] = v[r].x;
        }
    }
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
constexpr size_t kRowsSmem = sizeof(float2) * kM + (kStageBytes > kRowExBytes ? kStageBytes : kRowExBytes);
constexpr size_t kBackSmem = kRowsSmem + sizeof(float4) * kRowsBlock * kG;

// ---- spectrum, second axis: sixteen columns per block, two real ones per warp; Kh[c][k] ----
constexpr int kSpecCols = 2 * kRowThreads / 32, kSpecBlocks = kRkStride / kSpecCols;
constexpr int kSpecRow = kSpecCols + 4;   // floats per row in shared memory
static_assert(kRkStride % kSpecCols == 0 && kSpecBlocks * kSpecCols >= kC, "columns of the spectrum");
static_assert(sizeof(float) * kG * kSpecRow <= kStageBytes, "the columns fit where the lines are staged");
__device__ __forceinline__ void spectrum_columns(float2 *smem, const float *__restrict__ Rk, float *__restrict__ Kh, const float2 *__restrict__ tw, int block)
{
    float2 *tws = smem, *ex = smem + kM + (threadIdx.x >> 5) * kEx;
    float *cols = reinterpret_cast<float *>(smem + kM);   // before the exchange
    const int lane = threadIdx.x & 31, own = 2 * (threadIdx.x >> 5), c = kSpecCols * block + own;
    for (int u = threadIdx.x; u < kG * kSpecCols / 4; u += kRowThreads) {
        const int row = u / (kSpecCols / 4), part = u % (kSpecCols / 4);
        copy16(cols + row * kSpecRow + 4 * part, Rk + (size_t)row * kRkStride + kSpecCols * block + 4 * part);
    }
    end_batch();
    copy_twiddles<kRowThreads>(tws, tw);
    end_batch();
    copies_done<1>();
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int row = kR * r + lane;
        v[r] = (lane < kR && row < kG) ? *reinterpret_cast<const float2 *>(cols + row * kSpecRow + own) : make_float2(0.0f, 0.0f);
    }
    mirror_input(v, lane);
    fft784_warp<false, kR>(v, ex, tws, lane, copies_done<0>);
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
fft_rows_forward_kernel(const float4 *__restrict__ w, float4 *__restrict__ A, const float *__restrict__ Rk, float *__restrict__ Kh,
                        const IterState *state, int slot, const float2 *__restrict__ tw)
{
    extern __shared__ __align__(16) float2 smem[];
    if (blockIdx.x >= kLines) {
        spectrum_columns(smem, Rk, Kh, tw, blockIdx.x - kLines);
        return;
    }
    float2 *tws = smem, *stage = smem + kM;   // the lines, once the exchange is over
    const int lane = threadIdx.x & 31, plane = (threadIdx.x >> 5) & 1, row = kRowsBlock * blockIdx.x + (threadIdx.x >> 6);
    copy_twiddles<kRowThreads>(tws, tw);
    end_batch();
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
    fft784_warp<false, kHalf>(v, stage + (threadIdx.x >> 5) * kEx, tws, lane, copies_done<0>);
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
constexpr size_t kColsSmem = sizeof(float2) * (kM + 4 * kEx + kLines * kLine) + sizeof(float) * kM;
__global__ void __launch_bounds__(128)
fft_columns_kernel(const float4 *__restrict__ A, const float *__restrict__ Kh, float4 *__restrict__ B, const float2 *__restrict__ tw)
{
    extern __shared__ __align__(16) float2 smem[];
    float2 *tws = smem, *ex = smem + kM + (threadIdx.x >> 5) * kEx, *lines = smem + kM + 4 * kEx;
    float *spec = reinterpret_cast<float *>(lines + kLines * kLine);
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5, c = blockIdx.x;
    constexpr int n4 = kLines * kLine / 2;
    copy_floats<128>(reinterpret_cast<float *>(lines), reinterpret_cast<const float *>(A + (size_t)c * n4), n4);
    end_batch();
    copy_twiddles<128>(tws, tw);
    end_batch();
    copy_floats<128>(spec, Kh + (size_t)c * kM, kM / 4);
    end_batch();
    copies_done<2>();
    const int sl = min(lane, kR - 1);
    float2 *mine = lines + (sl / kRowsBlock) * kLine;   // rows 28 r + lane: 7 r lines further on; a warp has its q to itself
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        v[r] = mine[r * (kR / kRowsBlock) * kLine + place_in_line(q, r * (kR / kRowsBlock) + sl / kRowsBlock, sl)];
    }
    fft784_warp<false, kHalf>(v, ex, tws, lane, copies_done<1>);
    copies_done<0>();
#pragma unroll
    for (int r = 0; r < kR; r++) v[r] = times(spec[kR * r + sl], v[r]);
    fft784_warp<true, kR>(v, ex, tws, lane, [] {});
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
fft_rows_inverse_kernel(const float4 *__restrict__ B, float4 *__restrict__ w, float4 *__restrict__ ytilde, IterState *state, int slot,
                        const float2 *__restrict__ tw, int zero_w)
{
    extern __shared__ __align__(16) float2 smem[];
    float2 *tws = smem, *stage = smem + kM;   // the lines, before the exchange
    float4 *charges = reinterpret_cast<float4 *>(smem) + (kBackSmem - sizeof(float4) * kRowsBlock * kG) / sizeof(float4);
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5, plane = wi & 1, row = kRowsBlock * blockIdx.x + (wi >> 1);
    for (int u = threadIdx.x; u < kC * kLine / 2; u += kRowThreads) {
        const int c = u / (kLine / 2), part = u % (kLine / 2);
        copy16(stage + c * kStageLine + 2 * part, B + ((size_t)c * kLines + blockIdx.x) * (kLine / 2) + part);
    }
    end_batch();
    copy_twiddles<kRowThreads>(tws, tw);
    end_batch();
    float4 *wrows = w + (size_t)kRowsBlock * blockIdx.x * kG;
    const int nodes = min(kRowsBlock, kG - kRowsBlock * (int)blockIdx.x) * kG;
    for (int j = threadIdx.x; j < nodes; j += kRowThreads) copy16(charges + j, wrows + j);
    end_batch();
    const float scale = 1.0f / ((float)kM * (float)kM);
    const float imag_scale = plane == 1 ? scale * load_geom(state, slot).r2_unscale : scale;
    copies_done<2>();
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const int k = kR * r + min(lane, kR - 1);
        v[r] = stage[column_of(k) * kStageLine + place_in_line(2 * plane + slot_of(k), blockIdx.x, row)];
    }
    fft784_warp<true, kR>(v, stage + wi * kEx, tws, lane, copies_done<1>);   // (a barrier: the lines have been read)
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
    static_assert(kColsSmem <= 48 * 1024, "columns pass: no more than a kernel may have unasked");
    twiddle_init_kernel<<<(kM + 255) / 256, 256, 0, st>>>(ws->tw);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int convolve_wave_sms(int *sms)
{
    int per_sm = 0;
    B200_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fft_columns_kernel, 128, kColsSmem));
    *sms = (kC + std::max(per_sm, 1) - 1) / std::max(per_sm, 1);
    return 0;
}

int launch_kernel_spectrum(const IterState *state, int slot, const FftWorkspace &ws, cudaStream_t st)
{
    spectrum_rows_kernel<<<(kG + kSpecWarps - 1) / kSpecWarps, kSpecWarps * 32, 0, st>>>(ws.Rk, state, slot, ws.tw);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_convolve_rows(const float4 *w, const IterState *state, int slot, const FftWorkspace &ws, cudaStream_t st)
{
    fft_rows_forward_kernel<<<kLines + kSpecBlocks, kRowThreads, kRowsSmem, st>>>(w, ws.A, ws.Rk, ws.Kh, state, slot, ws.tw);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_convolve(float4 *w, float4 *ytilde, IterState *state, int slot, const FftWorkspace &ws, bool zero_w, cudaStream_t st)
{
    fft_columns_kernel<<<kC, 128, kColsSmem, st>>>(ws.A, ws.Kh, ws.B, ws.tw);
    B200_CUDA(cudaGetLastError());
    fft_rows_inverse_kernel<<<kLines, kRowThreads, kBackSmem, st>>>(ws.B, w, ytilde, state, slot, ws.tw, zero_w ? 1 : 0);
    B200_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace b200
