// 784-point transforms by a warp, and the first axis of the kernel's spectrum, which the spread's launch has on its side
// (see convolve.cu).
#pragma once
#include "grid_geom.cuh"

namespace b200 {

constexpr int kR = 28;                       // kM = kR * kR
constexpr int kHalf = kR / 2;                // registers that hold a 390-point input or output: 28 * 14 >= 390
constexpr int kC = kM / 2 + 1;               // distinct columns of an even spectrum: 0 .. 392
constexpr int kRkStride = (kC + 15) / 16 * 16;   // row of Rk: whole groups of the columns that a block of the second axis takes
constexpr int kExStride = kR + 1;            // float2 per row of the exchange buffer (odd: no bank conflicts)
constexpr int kEx = kR * kExStride;
static_assert(kM == kR * kR && kM >= 2 * kG - 1 && kR * kHalf >= kG && kR * (kHalf - 1) < kG, "transform length");

// Sums and products with a real coefficient act on both halves of a complex number alike: one packed instruction each, with
// the results of the two it stands for.  The fp32 pipe is as fast either way; the issue slots go to everything else.
__device__ __forceinline__ float2 operator+(float2 a, float2 b)
{
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack(a)), "l"(pack(b)));
    return unpack(r);
}
// a + c * t, a real coefficient
__device__ __forceinline__ float2 axpy(float c, float2 t, float2 a)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack(make_float2(c, c))), "l"(pack(t)), "l"(pack(a)));
    return unpack(r);
}
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return axpy(-1.0f, b, a); }
__device__ __forceinline__ float2 times(float c, float2 t)
{
    unsigned long long r;
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

// What a block needs besides the values of its own transforms goes to shared memory with asynchronous copies, all in flight at
// once: a loop of loads and stores waits for L2 once per round (seven to thirteen rounds here), which cost more than the
// transforms.
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

// A lane's twiddles, e^{-2 pi i k l / 784} at tw[k * 28 + l], in registers: they are asked for before the kernel in front has
// ended, serve both transforms of a column, and a transform then waits for its exchange alone (out of shared memory, one
// by one between the products, 1,500 / 5,000 / 20,011 points 23.0 / 23.4 / 27.1 us an iteration; so 21.7 / 22.2 / 26.1).
using Twiddles = float2[kR];
__device__ __forceinline__ void load_twiddles(Twiddles &t, const float2 *__restrict__ tw, int lane)
{
#pragma unroll
    for (int k = 1; k < kR; k++)   // volatile: here and not where they are used
        asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(t[k].x), "=f"(t[k].y) : "l"(tw + k * kR + min(lane, kR - 1)));
}

// The same, each read where it is used: for a kernel whose other blocks want the registers.
struct LateTwiddles {
    const float2 *tw;
    __device__ __forceinline__ float2 operator[](int k) const { return __ldg(tw + k * kR); }
};

// 784-point transform by one warp.  In: lane l < 28 holds x[28 r + l] in v[r] (zero from r = NZ on).  Out: lane l holds
// X[l + 28 r] in v[r], the same pattern.  ex: kEx float2 of this warp, free when exchange_free() returns.
template <bool INV, int NZ, class TWIDDLES, class READY>
__device__ __forceinline__ void fft784_warp(float2 (&v)[kR], float2 *ex, const TWIDDLES &t, int lane, READY exchange_free)
{
    fft28<INV, NZ>(v);
    exchange_free();
    if (lane < kR) {
        ex[lane] = v[0];
#pragma unroll
        for (int k = 1; k < kR; k++) {
            float2 w = t[k];
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

// block: rows kSpecWarps block .. of the kernel, a block of kSpecWarps warps
constexpr int kSpecWarps = 2, kSpecRowBlocks = (kG + kSpecWarps - 1) / kSpecWarps;
template <bool LATE>
__device__ __forceinline__ void spectrum_rows(float *Rk, const IterState *state, int slot, const float2 *__restrict__ tw, int block)
{
    __shared__ float2 exch[kSpecWarps][kEx];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    Twiddles t;
    if (!LATE) load_twiddles(t, tw, lane);
    const int row = block * kSpecWarps + wi;
    after_previous();
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
    if constexpr (LATE) fft784_warp<false, kR>(v, exch[wi], LateTwiddles{tw + min(lane, kR - 1)}, lane, [] {});
    else fft784_warp<false, kR>(v, exch[wi], t, lane, [] {});
    if (row >= kG || lane >= kR) return;
#pragma unroll
    for (int r = 0; r <= kHalf; r++) {
        const int k = kR * r + lane;
        if (k < kRkStride) {
            Rk[(size_t)row * kRkStride + k] = v[r].x;
        }
    }
}

}  // namespace b200
