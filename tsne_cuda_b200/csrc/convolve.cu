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
//  * Column c, its mirror image 784 - c, and both planes stand side by side in the workspace (32 bytes per row): one
//    block transforms the four of them, every access is a whole sector, and the product with the spectrum never leaves
//    the SM.
//  * The last pass also sums the normalisation on the grid: sum_i Z_i is the bilinear form of charges and potentials
//    (each point's Z_i is interpolated from the potentials with the weights its charges were spread with), so it needs
//    neither a pass over the points nor an exchange between ranks that hold the summed grid.
//
// Bound: about 5,300 warp transforms of 1,100 issue slots are 10,000 cycles of all 592 schedulers, 5 us; the rest is the
// load latency of three dependent kernels.  Measured on B200, each kernel alone with warm caches: rows 5.2, columns 10.4,
// rows back 7.2 us (the three passes over 1024-point transforms, with the kernel as a third plane, took 7.5, 20 and 7 us);
// cold, under the profiler, 7.1, 12.5 and 8.7, and beside them 6.4 + 7.6 for the spectrum.
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
constexpr int kRkStride = kC + 1;            // row of Rk, padded to whole pairs of columns
constexpr int kExStride = kR + 1;            // float2 per row of the exchange buffer (odd: no bank conflicts)
constexpr int kEx = kR * kExStride;
static_assert(kM == kR * kR && kM >= 2 * kG - 1 && kR * kHalf >= kG && kR * (kHalf - 1) < kG, "transform length");

__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a + c * t, a real coefficient
__device__ __forceinline__ float2 axpy(float c, float2 t, float2 a) { return make_float2(fmaf(c, t.x, a.x), fmaf(c, t.y, a.y)); }
// -i b (forward) or +i b (inverse)
template <bool INV> __device__ __forceinline__ float2 turn(float2 b) { return INV ? make_float2(-b.y, b.x) : make_float2(b.y, -b.x); }

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
        b1 = make_float2(s1 * d1.x, s1 * d1.y); b2 = make_float2(s2 * d1.x, s2 * d1.y); b3 = make_float2(s3 * d1.x, s3 * d1.y);
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
    const float2 i1 = turn<INV>(b1), i2 = turn<INV>(b2), i3 = turn<INV>(b3);
    v[0] = sum;
    v[1] = a1 + i1; v[6] = a1 - i1;
    v[2] = a2 + i2; v[5] = a2 - i2;
    v[3] = a3 + i3; v[4] = a3 - i3;
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
        const float2 q = y[1][kb] + y[3][kb], r = turn<INV>(y[1][kb] - y[3][kb]);
        v[(8 * kb) % 28] = p + q;
        v[(21 + 8 * kb) % 28] = m + r;
        v[(42 + 8 * kb) % 28] = p - q;
        v[(63 + 8 * kb) % 28] = m - r;
    }
}

// 784-point transform by one warp.  In: lane l < 28 holds x[28 r + l] in v[r] (zero from r = NZ on).  Out: lane l holds
// X[l + 28 r] in v[r], the same pattern.  ex: kEx float2 of this warp; tws[k * 28 + l] = e^{-2 pi i k l / 784}.
template <bool INV, int NZ> __device__ __forceinline__ void fft784_warp(float2 (&v)[kR], float2 *ex, const float2 *tws, int lane)
{
    fft28<INV, NZ>(v);
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

// Everything a block needs besides the values of its own transforms goes to shared memory with asynchronous copies, all
// in flight at once: a loop of loads and stores waits for L2 once per round (seven to thirteen rounds here), which cost
// more than the transforms.
__device__ __forceinline__ void copy16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
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
    copies_done();
    fft784_warp<false, kR>(v, exch[wi], tws, lane);
    if (row >= kG || lane >= kR) return;
#pragma unroll
    for (int r = 0; r <= kHalf; r++) {
        const int k = kR * r + lane;
        if (k < kRkStride) {
            Rk[(size_t)row * kRkStride + k] = v[r].x;
        }
    }
}

// ---- second axis: two real columns per warp; Kh[c][k] ----
__global__ void __launch_bounds__(kSpecWarps * 32)
spectrum_columns_kernel(const float *__restrict__ Rk, float *__restrict__ Kh, const float2 *__restrict__ tw)
{
    __shared__ __align__(16) float2 tws[kM];
    __shared__ float2 exch[kSpecWarps][kEx];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const int c = 2 * (blockIdx.x * kSpecWarps + wi);
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int row = kR * r + lane;
        v[r] = (lane < kR && row < kG && c < kC) ? *reinterpret_cast<const float2 *>(Rk + (size_t)row * kRkStride + c) : make_float2(0.0f, 0.0f);
    }
    copy_twiddles<kSpecWarps * 32>(tws, tw);
    mirror_input(v, lane);
    copies_done();
    fft784_warp<false, kR>(v, exch[wi], tws, lane);
    if (c >= kC || lane >= kR) return;
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const int k = kR * r + lane;
        Kh[(size_t)c * kM + k] = v[r].x;
        if (c + 1 < kC) Kh[(size_t)(c + 1) * kM + k] = v[r].y;
    }
}

// ---- first pass: a row of the charge grid, both planes ----
__global__ void __launch_bounds__(64)
fft_rows_forward_kernel(const float4 *__restrict__ w, float4 *__restrict__ A, const IterState *state, int slot, const float2 *__restrict__ tw)
{
    __shared__ __align__(16) float2 tws[kM], out[2][kC][2];   // out[plane][column][slot]
    __shared__ float2 exch[2][kEx];
    const int lane = threadIdx.x & 31, plane = threadIdx.x >> 5, row = blockIdx.x;
    copy_twiddles<64>(tws, tw);
    const float2 *wrow = reinterpret_cast<const float2 *>(w + (size_t)row * kG) + plane;   // .xy or .zw of each node
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int j = kR * r + lane;
        v[r] = (lane < kR && j < kG) ? wrow[2 * j] : make_float2(0.0f, 0.0f);
    }
    const float imag_scale = plane == 1 ? load_geom(state, slot).r2_scale : 1.0f;
#pragma unroll
    for (int r = 0; r < kHalf; r++) v[r].y *= imag_scale;
    copies_done();
    fft784_warp<false, kHalf>(v, exch[plane], tws, lane);
    if (lane < kR) {
#pragma unroll
        for (int r = 0; r < kR; r++) {
            const int k = kR * r + lane;
            out[plane][column_of(k)][slot_of(k)] = v[r];
        }
    }
    __syncthreads();
    float4 *dst = A + (size_t)row * kC * 2;
#pragma unroll
    for (int u = threadIdx.x; u < 2 * kC; u += 64) dst[u] = *reinterpret_cast<const float4 *>(out[u & 1][u >> 1]);
}

// ---- second pass: column c, its mirror image, both planes: forward, product with the spectrum, inverse ----
constexpr size_t kColsSmem = sizeof(float2) * (kM + 4 * kEx + 4 * kG) + sizeof(float) * kM;
__global__ void __launch_bounds__(128)
fft_columns_kernel(const float2 *__restrict__ A, const float *__restrict__ Kh, float4 *__restrict__ B, const float2 *__restrict__ tw)
{
    extern __shared__ __align__(16) float2 smem[];
    float2 *tws = smem, *ex = smem + kM + (threadIdx.x >> 5) * kEx, *out = smem + kM + 4 * kEx;
    float *spec = reinterpret_cast<float *>(smem + kM + 4 * kEx + 4 * kG);
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5, c = blockIdx.x;
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int row = kR * r + lane;
        v[r] = (lane < kR && row < kG) ? A[((size_t)row * kC + c) * 4 + q] : make_float2(0.0f, 0.0f);
    }
    copy_twiddles<128>(tws, tw);
    copy_floats<128>(spec, Kh + (size_t)c * kM, kM / 4);
    copies_done();
    fft784_warp<false, kHalf>(v, ex, tws, lane);
    const int sl = min(lane, kR - 1);
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const float k = spec[kR * r + sl];
        v[r].x *= k;
        v[r].y *= k;
    }
    fft784_warp<true, kR>(v, ex, tws, lane);
    if (lane < kR) {
#pragma unroll
        for (int r = 0; r < kHalf; r++) {
            const int row = kR * r + lane;
            if (row < kG) out[q * kG + row] = v[r];
        }
    }
    __syncthreads();
#pragma unroll
    for (int row = threadIdx.x; row < kG; row += 128) {
        const float2 a = out[row], b = out[kG + row], e = out[2 * kG + row], f = out[3 * kG + row];
        float4 *dst = B + ((size_t)row * kC + c) * 2;
        dst[0] = make_float4(a.x, a.y, b.x, b.y);
        dst[1] = make_float4(e.x, e.y, f.x, f.y);
    }
}

// ---- third pass: a row of potentials, both planes; the grid's share of sum_i Z_i ----
__global__ void __launch_bounds__(64)
fft_rows_inverse_kernel(const float4 *__restrict__ B, float4 *__restrict__ w, float4 *__restrict__ ytilde, IterState *state, int slot,
                        const float2 *__restrict__ tw, int zero_w)
{
    __shared__ __align__(16) float2 tws[kM], in[2][kC][2];   // in[plane][column][slot]
    __shared__ __align__(16) float4 charge[kG];
    __shared__ float2 exch[2][kEx];
    const int lane = threadIdx.x & 31, plane = threadIdx.x >> 5, row = blockIdx.x;
    const float4 *src = B + (size_t)row * kC * 2;
    float4 *wrow = w + (size_t)row * kG;
    for (int u = threadIdx.x; u < 2 * kC; u += 64) copy16(in[u & 1][u >> 1], src + u);
    copy_twiddles<64>(tws, tw);
    for (int j = threadIdx.x; j < kG; j += 64) copy16(charge + j, wrow + j);
    const float scale = 1.0f / ((float)kM * (float)kM);
    const float imag_scale = plane == 1 ? scale * load_geom(state, slot).r2_unscale : scale;
    copies_done();
    if (zero_w)
        for (int j = threadIdx.x; j < kG; j += 64) wrow[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float2 v[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const int k = kR * r + min(lane, kR - 1);
        v[r] = in[plane][column_of(k)][slot_of(k)];
    }
    fft784_warp<true, kR>(v, exch[plane], tws, lane);
    float2 *out = reinterpret_cast<float2 *>(ytilde + (size_t)row * kG) + plane;
    double z = 0.0;
#pragma unroll
    for (int r = 0; r < kHalf; r++) {
        const int j = kR * r + lane;
        if (lane < kR && j < kG) {
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
    __shared__ double other;
    if (threadIdx.x == 32) other = z;
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&state->zsum[slot], z + other);
        if (row == 0) {   // recycle the other slot's min/max and this slot's norm for this iteration's update
            state->min_enc[slot ^ 1] = 0xffffffffu;
            state->max_enc[slot ^ 1] = 0u;
            state->unorm2[slot] = 0.0;
        }
    }
}

}  // namespace

size_t fft_workspace_bytes()
{
    return sizeof(float4) * (size_t)kG * kC * 2 * 2 + sizeof(float) * ((size_t)kG * kRkStride + (size_t)kC * kM) + sizeof(float2) * kM;
}

int fft_workspace_init(FftWorkspace *ws, void *mem, cudaStream_t st)
{
    char *p = static_cast<char *>(mem);
    ws->A = reinterpret_cast<float4 *>(p); p += sizeof(float4) * (size_t)kG * kC * 2;
    ws->B = reinterpret_cast<float4 *>(p); p += sizeof(float4) * (size_t)kG * kC * 2;
    ws->tw = reinterpret_cast<float2 *>(p); p += sizeof(float2) * kM;
    ws->Kh = reinterpret_cast<float *>(p); p += sizeof(float) * (size_t)kC * kM;
    ws->Rk = reinterpret_cast<float *>(p);
    static_assert(kColsSmem <= 48 * 1024, "columns pass: three blocks to an SM, and no more than a kernel may have unasked");
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
    constexpr int row_blocks = (kG + kSpecWarps - 1) / kSpecWarps, col_blocks = ((kC + 1) / 2 + kSpecWarps - 1) / kSpecWarps;
    spectrum_rows_kernel<<<row_blocks, kSpecWarps * 32, 0, st>>>(ws.Rk, state, slot, ws.tw);
    B200_CUDA(cudaGetLastError());
    spectrum_columns_kernel<<<col_blocks, kSpecWarps * 32, 0, st>>>(ws.Rk, ws.Kh, ws.tw);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_convolve_rows(const float4 *w, const IterState *state, int slot, const FftWorkspace &ws, cudaStream_t st)
{
    fft_rows_forward_kernel<<<kG, 64, 0, st>>>(w, ws.A, state, slot, ws.tw);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_convolve(float4 *w, float4 *ytilde, IterState *state, int slot, const FftWorkspace &ws, bool zero_w, cudaStream_t st)
{
    fft_columns_kernel<<<kC, 128, kColsSmem, st>>>(reinterpret_cast<const float2 *>(ws.A), ws.Kh, ws.B, ws.tw);
    B200_CUDA(cudaGetLastError());
    fft_rows_inverse_kernel<<<kG, 64, 0, st>>>(ws.B, w, ytilde, state, slot, ws.tw, zero_w ? 1 : 0);
    B200_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace b200
