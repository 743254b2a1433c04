// Gradient, gains and momentum update (reference: IntegrationKernel, src/kernels/apply_forces.cu:11-57)
// fused with the min/max reduction the next iteration's grid needs (reference: thrust::minmax_element
// + two host reads, src/fit_tsne.cu:430-432) and the optional update-norm reduction
// (src/fit_tsne.cu:522-527).  40 bytes read and 24 written per point, and nine nodes of 16 bytes out of L2 where the repulsive
// force is interpolated here (10^6 points: 32 us, 22 without).
#include "grid_geom.cuh"

namespace b200 {

namespace {

__device__ __forceinline__ float gain_rule(float g, float grad, float u)
{
    // the reference evaluates g + 0.2 and g * 0.8 in double and rounds once
    g = (signbit(grad) != signbit(u)) ? (float)((double)g + 0.2) : (float)((double)g * 0.8);
    return (g < 0.01) ? (float)0.01 : g;
}

__device__ __forceinline__ void step_point(float2 &y, const float2 fa, const float2 fr, float2 &g, float2 &u, float eta,
                                           float Z, float momentum, float exaggeration)
{
    const float dx = exaggeration * fa.x - (fr.x / Z);
    const float dy = exaggeration * fa.y - (fr.y / Z);
    g.x = gain_rule(g.x, dx, u.x);
    g.y = gain_rule(g.y, dy, u.y);
    u.x = momentum * u.x - eta * g.x * dx;
    u.y = momentum * u.y - eta * g.y * dy;
    y.x += u.x;
    y.y += u.y;
}

// Rows [row_lo, row_lo+n_rows) of the embedding are updated: read from Y2, written to every array of
// `dst` (in place: Y2 itself; sharded over peer memory: the next embedding buffer of every rank, which
// replaces an all-gather).  Reads the normalisation
// from state->zsum[slot] (sum of Z_i; Z = sum - n_total as in src/kernels/rep_forces.cu:51-54),
// accumulates min/max of the new coordinates into slot^1 and clears zsum[slot^1] for the next
// iteration.
// GATHER: the repulsive force is interpolated here instead of read from Fr: one launch and 16 bytes per point less
// (whole iteration at 5 000 / 10^6 points: 38.2 -> 37.4 / 251 -> 238 us, although the interpolation now waits for the
// attractive force).  (Clearing Fa here for the next iteration's additions instead of a memset on the other stream costs
// 2 us at 1 500 points and 5 at 200 000.)
// norm_mode 1: unorm2[slot] = sum of squared updates.  2: and nothing is changed any more once the previous iteration's
// norm is below stop_norm (the iterations the host has queued beyond the reference's stop leave the state alone).
template <bool GATHER, int THREADS>
__global__ void __launch_bounds__(THREADS)
update_kernel(const float2 *Y2, UpdateTargets dst, const float2 *Fa, const float2 *Fr, const float4 *ytilde, InterpConsts ic, float2 *gains,
              float2 *u2, long long row_lo, long long n_rows, long long n_total, IterState *state, int slot, float eta, float momentum, float exaggeration,
              int norm_mode, float stop_norm)
{
    after_previous();
    // Everything that does not depend on a position is loaded before anything is computed: the positions' nodes are the second
    // round trip to L2 then (900 cycles each here) and not the fourth.
    const long long r = (long long)blockIdx.x * THREADS + threadIdx.x, i = row_lo + r;
    const bool mine = r < n_rows;
    float2 y = make_float2(0.0f, 0.0f), g = y, u = y, fa = y, fr = y;
    if (mine) {
        y = Y2[i]; g = gains[r]; u = u2[r];
        fa = __ldcs(Fa + i);
        if (!GATHER) fr = __ldcs(Fr + i);
    }
    const double zsum = state->zsum[slot], last_norm2 = state->unorm2[slot ^ 1];
    const GridGeom geom = load_geom(state, slot);
    float mn = INFINITY, mx = -INFINITY, nrm = 0.0f;
    int bad = 0;
    const bool stopped = norm_mode == 2 && (float)sqrt(last_norm2) < stop_norm;
    if (mine) {
        if (GATHER) fr = repulsive_force(y, geom, ic, ytilde);
        const float Z = (float)zsum - (float)n_total;
        if (!stopped) {
            step_point(y, fa, fr, g, u, eta, Z, momentum, exaggeration);
#pragma unroll
            for (int t = 0; t < (GATHER ? 1 : kMaxUpdateTargets); t++)   // (GATHER: one GPU)
                if (t < dst.n) dst.p[t][i] = y;
            gains[r] = g;
            u2[r] = u;
        }
        mn = fminf(y.x, y.y);
        mx = fmaxf(y.x, y.y);
        nrm = u.x * u.x + u.y * u.y;
        bad = !(isfinite(y.x) && isfinite(y.y));
    }
    // order-preserving encodings: one reduction instruction each (a coordinate that is no number counts for neither)
    unsigned emn = __reduce_min_sync(0xffffffffu, enc_float(fminf(INFINITY, mn))), emx = __reduce_max_sync(0xffffffffu, enc_float(fmaxf(-INFINITY, mx)));
    if (norm_mode) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    }
    bad = __any_sync(0xffffffffu, bad);
    constexpr int kWarps = THREADS / 32;
    __shared__ unsigned s_mn[kWarps], s_mx[kWarps];
    __shared__ float s_n[kWarps];
    __shared__ int s_bad[kWarps];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { s_mn[w] = emn; s_mx[w] = emx; s_n[w] = nrm; s_bad[w] = bad; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
#pragma unroll
        for (int k = 0; k < kWarps; k++) {
            emn = min(emn, s_mn[k]); emx = max(emx, s_mx[k]); tot += (double)s_n[k]; bad |= s_bad[k];
        }
        if (emn <= emx) {
            atomicMin(&state->min_enc[slot ^ 1], emn);
            atomicMax(&state->max_enc[slot ^ 1], emx);
        }
        if (norm_mode && !stopped) atomicAdd(&state->unorm2[slot], tot);
        if (bad) state->bad = 1;
        if (blockIdx.x == 0) {
            state->zsum[slot ^ 1] = 0.0;
            if (!stopped) { state->z_last = zsum; state->done++; }
            else state->unorm2[slot] = state->unorm2[slot ^ 1];   // once stopped, the later iterations are too
        }
    }
}

// Stand-alone form with the reference's SoA buffers and an explicit Z, for the stage entry point.
__global__ void apply_forces_soa_kernel(float *Y, float *attr, float *rep, float *gains, float *old_forces, float eta,
                                        float Z, float momentum, float exaggeration, long long N)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    float2 y = make_float2(Y[i], Y[N + i]), g = make_float2(gains[i], gains[N + i]);
    float2 u = make_float2(old_forces[i], old_forces[N + i]);
    const float2 fa = make_float2(attr[i], attr[N + i]), fr = make_float2(rep[i], rep[N + i]);
    step_point(y, fa, fr, g, u, eta, Z, momentum, exaggeration);
    Y[i] = y.x; Y[N + i] = y.y;
    gains[i] = g.x; gains[N + i] = g.y;
    old_forces[i] = u.x; old_forces[N + i] = u.y;
    attr[i] = 0.0f; attr[N + i] = 0.0f; rep[i] = 0.0f; rep[N + i] = 0.0f;
}

// perm (optional): position q of the pair array holds point perm[q] of the block-wise array
__global__ void soa_to_aos_kernel(const float *soa, float2 *aos, long long N, const int32_t *perm)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) { const long long j = perm ? perm[i] : i; aos[i] = make_float2(soa[j], soa[N + j]); }
}
__global__ void aos_to_soa_kernel(const float2 *aos, float *soa, long long N, const int32_t *perm)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) { const long long j = perm ? perm[i] : i; const float2 v = aos[i]; soa[j] = v.x; soa[N + j] = v.y; }
}
__global__ void __launch_bounds__(256)
load_state_kernel(const float *io, float2 *Y2, float2 *u2, float2 *gains2, long long N, IterState *state, int slot)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float mn = INFINITY, mx = -INFINITY;
    if (i < N) {
        const float2 y = make_float2(io[i], io[N + i]);
        Y2[i] = y;
        u2[i] = make_float2(io[2 * N + i], io[3 * N + i]);
        gains2[i] = make_float2(io[4 * N + i], io[5 * N + i]);
        mn = fminf(y.x, y.y);
        mx = fmaxf(y.x, y.y);
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
__global__ void __launch_bounds__(256)
store_state_kernel(const float2 *Y2, const float2 *u2, const float2 *gains2, float *io, long long N)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const float2 *from[3] = {Y2, u2, gains2};
#pragma unroll
    for (int a = 0; a < 3; a++)
        if (from[a]) {
            const float2 v = from[a][i];
            io[2 * a * N + i] = v.x;
            io[(2 * a + 1) * N + i] = v.y;
        }
}
// dst[q] = src[perm[q]] (gather) or dst[perm[q]] = src[q] (scatter)
__global__ void reorder_pairs_kernel(const float2 *src, float2 *dst, long long N, const int32_t *perm, int scatter)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    if (scatter) dst[perm[i]] = src[i];
    else dst[i] = src[perm[i]];
}
__global__ void fill_kernel(float *p, float v, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

constexpr long long kUpdateSmallMax = 148 * 256;
inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }
}  // namespace

int launch_update(const float2 *Y2, const UpdateTargets &dst, const float2 *Fattr2, const float2 *Frep2, const float4 *ytilde, InterpConsts ic,
                  float2 *gains2, float2 *u2, int64_t N, int64_t row_lo, int64_t row_hi, IterState *state, int slot, float eta,
                  float momentum, float exaggeration, int norm_mode, float stop_norm, cudaStream_t st)
{
    const long long n_rows = row_hi - row_lo;
    // Even an empty shard must run one block so that the state slots are recycled.  A warp's nine node reads touch up to 32
    // lines each, which the SM serves one by one: blocks of two warps as long as larger ones would leave SMs idle.
    const bool small = n_rows <= kUpdateSmallMax;
    const auto chained = [&](auto kernel) {
        const unsigned threads = small ? 64 : 256;
        return launch_chained(kernel, n_rows > 0 ? nblk(n_rows, threads) : 1, threads, 0, st, Y2, dst, Fattr2, Frep2, ytilde, ic, gains2, u2, row_lo, n_rows, N,
                              state, slot, eta, momentum, exaggeration, norm_mode, stop_norm);
    };
    if (ytilde) B200_CUDA(chained(small ? update_kernel<true, 64> : update_kernel<true, 256>));
    else B200_CUDA(chained(small ? update_kernel<false, 64> : update_kernel<false, 256>));
    return 0;
}

int launch_apply_forces_soa(float *Y, float *attr, float *rep, float *gains, float *old_forces, float eta, float Z,
                            float momentum, float exaggeration, int64_t N, cudaStream_t st)
{
    if (N <= 0) return 0;
    apply_forces_soa_kernel<<<nblk(N, 256), 256, 0, st>>>(Y, attr, rep, gains, old_forces, eta, Z, momentum,
                                                         exaggeration, N);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_soa_to_aos(const float *soa, float2 *aos, int64_t N, cudaStream_t st, const int32_t *perm)
{
    if (N <= 0) return 0;
    soa_to_aos_kernel<<<nblk(N, 256), 256, 0, st>>>(soa, aos, N, perm);
    B200_CUDA(cudaGetLastError());
    return 0;
}
int launch_aos_to_soa(const float2 *aos, float *soa, int64_t N, cudaStream_t st, const int32_t *perm)
{
    if (N <= 0) return 0;
    aos_to_soa_kernel<<<nblk(N, 256), 256, 0, st>>>(aos, soa, N, perm);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_load_state(const float *io, float2 *Y2, float2 *u2, float2 *gains2, int64_t N, IterState *state, int slot, cudaStream_t st)
{
    if (N <= 0) return 0;
    load_state_kernel<<<nblk(N, 256), 256, 0, st>>>(io, Y2, u2, gains2, N, state, slot);
    B200_CUDA(cudaGetLastError());
    return 0;
}
int launch_store_state(const float2 *Y2, const float2 *u2, const float2 *gains2, float *io, int64_t N, cudaStream_t st)
{
    if (N <= 0) return 0;
    store_state_kernel<<<nblk(N, 256), 256, 0, st>>>(Y2, u2, gains2, io, N);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_reorder_pairs(const float2 *src, float2 *dst, int64_t N, const int32_t *perm, bool scatter, cudaStream_t st)
{
    if (N <= 0) return 0;
    reorder_pairs_kernel<<<nblk(N, 256), 256, 0, st>>>(src, dst, N, perm, scatter ? 1 : 0);
    B200_CUDA(cudaGetLastError());
    return 0;
}
int launch_fill(float *p, float v, int64_t n, cudaStream_t st)
{
    if (n <= 0) return 0;
    fill_kernel<<<nblk(n, 256), 256, 0, st>>>(p, v, n);
    B200_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace b200
