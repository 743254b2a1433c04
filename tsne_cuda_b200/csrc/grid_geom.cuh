// Geometry of the interpolation grid over the embedding's bounding square, shared by the spread, the convolution and the
// gather (reference: src/kernels/nbodyfft.cu:43-105).
#pragma once
#include "common.cuh"

namespace b200 {

struct GridGeom {
    float cmin, box_width;
    float box_inv;                // 1 / box_width; 0 where the division by it is left to the compiler
    float r2_scale, r2_unscale;   // powers of two: r2_scale * max possible (x^2+y^2) lies in [4, 8)
};

// a / b from r, the reciprocal of b as a float: two Newton-Raphson steps on the quotient.  The first leaves less than one unit
// of the last place, and a step from there rounds correctly (Markstein 1990), so this is the quotient that a division gives as
// long as the remainder a - q b does not underflow.  Eight divisions with their special cases were 900 cycles between a point's
// load and its first access to the grid, half the time of the spread and a fifth of the update at 5,000 points.
__device__ __forceinline__ float divide(float a, float b, float r)
{
    float q = a * r;
    q = fmaf(fmaf(-q, b, a), r, q);
    return fmaf(fmaf(-q, b, a), r, q);
}

__device__ __forceinline__ GridGeom load_geom(const IterState *state, int slot)
{
    GridGeom g;
    const float cmin = dec_float(state->min_enc[slot]);
    const float cmax = dec_float(state->max_enc[slot]);
    g.cmin = cmin;
    g.box_width = (cmax - cmin) / (float)kBoxes;
    // All points identical: the reference divides by zero here.  Use a tiny positive width so that
    // every point falls in box 0 with in-box coordinate 0 and all results stay finite.
    if (!(g.box_width > 0.0f)) g.box_width = 1e-30f;
    g.box_inv = g.box_width > 1e-20f && g.box_width < 1e20f ? 1.0f / g.box_width : 0.0f;
    const float r = fmaxf(fabsf(cmin), fabsf(cmax));
    const float r2max = 2.0f * r * r;
    int e = 0;
    // from the exponent's bits (a subnormal's say -127, which the limit covers)
    if (r2max > 0.0f && r2max < INFINITY) e = min(100, max(-100, 129 - (__float_as_int(r2max) >> 23)));
    g.r2_scale = __int_as_float((127 + e) << 23);
    g.r2_unscale = __int_as_float((127 - e) << 23);
    return g;
}

// c in box widths from the grid's edge
__device__ __forceinline__ float in_boxes(float c, const GridGeom &g)
{
    return g.box_inv != 0.0f ? divide(c, g.box_width, g.box_inv) : c / g.box_width;
}

__device__ __forceinline__ void axis_weights(float c, const GridGeom &g, const InterpConsts &ic, int &box, float (&L)[kInterp])
{
    int idx = (int)in_boxes(c - g.cmin, g);
    idx = max(0, idx);
    idx = min(kBoxes - 1, idx);
    const float lower = idx * g.box_width + g.cmin;
    const float in_box = in_boxes(c - lower, g);
#pragma unroll
    for (int j = 0; j < kInterp; j++) {
        float v = 1;
#pragma unroll
        for (int k = 0; k < kInterp; k++)
            if (j != k) v *= in_box - ic.sp[k];
        L[j] = divide(v, ic.den[j], ic.den_inv[j]);   // |v| is 0 or above 2^-50: a coordinate in its box is a float of about 1
    }
    box = idx;
}

__device__ __forceinline__ float4 load_node(const float4 *p)   // volatile: a point's nodes are asked for one right after the other
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

// the point's repulsive force before the division by Z, interpolated from the potentials
__device__ __forceinline__ float2 repulsive_force(float2 y, const GridGeom &g, const InterpConsts &ic, const float4 *ytilde)
{
    int bx, by;
    float Lx[kInterp], Ly[kInterp];
    axis_weights(y.x, g, ic, bx, Lx);
    axis_weights(y.y, g, ic, by, Ly);
    float4 v[kInterp][kInterp];
#pragma unroll
    for (int a = 0; a < kInterp; a++)
#pragma unroll
        for (int b = 0; b < kInterp; b++) v[a][b] = load_node(ytilde + (size_t)(bx * kInterp + a) * kG + (by * kInterp + b));
    float p1 = 0.0f, p2 = 0.0f, p3 = 0.0f;
#pragma unroll
    for (int a = 0; a < kInterp; a++) {
#pragma unroll
        for (int b = 0; b < kInterp; b++) {
            const float l = Lx[a] * Ly[b];
            p1 += l * v[a][b].z; p2 += l * v[a][b].x; p3 += l * v[a][b].y;  // node = (x, y, count, r^2) potentials
        }
    }
    return make_float2(y.x * p1 - p2, y.y * p1 - p3);
}

}  // namespace b200
