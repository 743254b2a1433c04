// Geometry of the interpolation grid over the embedding's bounding square, shared by the spread, the convolution and the
// gather (reference: src/kernels/nbodyfft.cu:43-105).
#pragma once
#include "common.cuh"

namespace b200 {

struct GridGeom {
    float cmin, box_width;
    float r2_scale, r2_unscale;   // powers of two: r2_scale * max possible (x^2+y^2) lies in [4, 8)
};

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
    const float r = fmaxf(fabsf(cmin), fabsf(cmax));
    const float r2max = 2.0f * r * r;
    int e = 0;
    if (r2max > 0.0f && r2max < INFINITY) e = min(100, max(-100, 2 - ilogbf(r2max)));
    g.r2_scale = scalbnf(1.0f, e);
    g.r2_unscale = scalbnf(1.0f, -e);
    return g;
}

__device__ __forceinline__ void axis_weights(float c, const GridGeom &g, const InterpConsts &ic, int &box, float (&L)[kInterp])
{
    int idx = (int)((c - g.cmin) / g.box_width);
    idx = max(0, idx);
    idx = min(kBoxes - 1, idx);
    const float lower = idx * g.box_width + g.cmin;
    const float in_box = (c - lower) / g.box_width;
#pragma unroll
    for (int j = 0; j < kInterp; j++) {
        float v = 1;
#pragma unroll
        for (int k = 0; k < kInterp; k++)
            if (j != k) v *= in_box - ic.sp[k];
        L[j] = v / ic.den[j];
    }
    box = idx;
}

// the point's repulsive force before the division by Z, interpolated from the potentials
__device__ __forceinline__ float2 repulsive_force(float2 y, const GridGeom &g, const InterpConsts &ic, const float4 *__restrict__ ytilde)
{
    int bx, by;
    float Lx[kInterp], Ly[kInterp];
    axis_weights(y.x, g, ic, bx, Lx);
    axis_weights(y.y, g, ic, by, Ly);
    float p1 = 0.0f, p2 = 0.0f, p3 = 0.0f;
#pragma unroll
    for (int a = 0; a < kInterp; a++) {
#pragma unroll
        for (int b = 0; b < kInterp; b++) {
            const float l = Lx[a] * Ly[b];
            const float4 v = ytilde[(size_t)(bx * kInterp + a) * kG + (by * kInterp + b)];
            p1 += l * v.z; p2 += l * v.x; p3 += l * v.y;  // node = (x, y, count, r^2) potentials
        }
    }
    return make_float2(y.x * p1 - p2, y.y * p1 - p3);
}

}  // namespace b200
