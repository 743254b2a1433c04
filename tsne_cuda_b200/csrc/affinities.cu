// From neighbour distances to the fixed-width affinity matrix P:
//   global max-normalisation   (reference: util::MaxNormalizeDeviceVector, src/util/math_utils.cu:66-74)
//   per-row perplexity search  (reference: src/kernels/perplexity_search.cu:10-141: two elementwise
//                               kernels, two cuBLAS gemv row reductions and three device syncs per round)
//   symmetrisation             (reference: syv2k, src/util/math_utils.cu:269-291)
//
// Here one warp owns one row for the whole bisection: the row's normalised distances sit in shared
// memory, the row sums are warp shuffles, and p is written once (4*K bytes read + 4*K written per
// point).  The update rule, the fast exp/log intrinsics and the 200-round cap follow the reference.
#include <float.h>

#include "common.cuh"

namespace b200 {
namespace {

__global__ void __launch_bounds__(256) absmax_kernel(const float *__restrict__ v, long long n, unsigned int *max_enc)
{
    float m = 0.0f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float a = fabsf(v[i]);
        if (a > m && a < INFINITY) m = a;  // +inf marks an unfilled slot, never a distance
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(max_enc, enc_float(m));
}

__device__ __forceinline__ float cond_p(int s, float dist, float beta)
{
    // slot 0 is the point itself (distance exactly 0): p_ii = 0   (perplexity_search.cu:32)
    return (s == 0 & dist == 0.0f) ? 0.0f : __expf(-beta * dist);
}

constexpr int kPerpWarps = 8;

__global__ void __launch_bounds__(kPerpWarps * 32)
perplexity_kernel(const float *__restrict__ d2, long long n_rows, int K, float perplexity, float eps,
                  const unsigned int *__restrict__ max_enc, float *__restrict__ p, float *__restrict__ betas)
{
    extern __shared__ float srow[];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const long long row = (long long)blockIdx.x * kPerpWarps + wi;
    if (row >= n_rows) return;
    float *d = srow + (size_t)wi * K;
    const float maxv = dec_float(*max_enc);
    for (int s = lane; s < K; s += 32) d[s] = d2[row * K + s] / maxv;
    __syncwarp();
    const float log_perp = __logf(perplexity);
    float beta = 1.0f, lo = -FLT_MAX, hi = FLT_MAX;
    float beta_eval = beta, S = 0.0f;
    for (int it = 0; it < 200; it++) {
        float sum = 0.0f, ent = 0.0f;
        for (int s = lane; s < K; s += 32) {
            const float v = cond_p(s, d[s], beta);
            float e = v * logf(v);
            e = (e != e || isinf(e)) ? 0.0f : e;  // FunctionalEntropy, thrust_transform_functions.h:32-37
            sum += v;
            ent += e;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
            ent += __shfl_xor_sync(0xffffffffu, ent, o);
        }
        S = sum;
        beta_eval = beta;
        const float neg_ent = -ent;
        const float H = (neg_ent / S) + __logf(S);
        const float diff = H - log_perp;
        if (diff < eps && -diff < eps) break;
        if (diff > 0) {
            lo = beta;
            beta = (hi == FLT_MAX || hi == -FLT_MAX) ? beta * 2.0f : (beta + hi) / 2.0f;
        } else {
            hi = beta;
            beta = (lo == -FLT_MAX || lo == FLT_MAX) ? beta / 2.0f : (beta + lo) / 2.0f;
        }
    }
    // p of the last evaluated beta divided by its row sum.  A row that exhausts the 200 rounds keeps,
    // like the reference, the values of the beta evaluated last, not of the beta it would try next.
    for (int s = lane; s < K; s += 32) p[row * K + s] = cond_p(s, d[s], beta_eval) / S;
    if (lane == 0 && betas) betas[row] = beta;
}

// One warp per row i.  For each slot s: j = ids[i][s]; scan the K ids of row j for i and add the
// matching p[j][.]; divide by 2N in double like the reference.
// visit (optional, n_rows entries, all inside [row_lo, row_lo + n_rows)): the order in which the warps take the rows.
// The kernel is bound by the K random row reads per row (32 GB at N = 10^6, K = 90); rows visited cluster by cluster
// find the rows of their neighbours, which lie in the same cluster, in L2.
// d2 (optional): the lists' distances, ascending in a row and the same in both directions, and furthest[j] the last of row j.
// With them a lane finds its point in a neighbour's row by its distance: 10^6 points, K = 90 7.4 -> 2.9 ms, 60,000 x 90 0.44 -> 0.08, 50,000
// x 150 0.75 -> 0.11 (with the rows that cannot have it left out, but the others read whole: 6.3, 0.33, 0.56).
constexpr int kSymWarps = 8;
constexpr int kSymAhead = 4;   // neighbour rows whose loads are in flight together (8: 15.9 ms against 7.0 at N = 10^6, K = 90; 1: 8.5)
__global__ void furthest_kernel(const float *__restrict__ d2, long long N, int K, float *__restrict__ furthest)
{
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < N) furthest[j] = d2[j * K + K - 1];
}
template <bool BY_DISTANCE>
__global__ void __launch_bounds__(kSymWarps * 32)
symmetrize_kernel(const float *__restrict__ p, const int32_t *__restrict__ ids, long long N, int K, long long row_lo,
                  long long n_rows, const int32_t *__restrict__ visit, const float *__restrict__ d2, const float *__restrict__ furthest,
                  float *__restrict__ P_rows)
{
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * kSymWarps + (threadIdx.x >> 5);
    if (w >= n_rows) return;
    const long long i = visit ? (long long)visit[w] : row_lo + w;
    const long long r = i - row_lo;
    if (r < 0 || r >= n_rows) return;
    const double inv = 2.0 * (double)N;
    for (int s0 = 0; s0 < K; s0 += 32) {
        const int s_mine = s0 + lane;
        int j_mine = -1;
        float p_mine = 0.0f;
        if (s_mine < K) {
            j_mine = ids[i * K + s_mine];
            p_mine = p[i * K + s_mine];
        }
        float acc_mine = p_mine;
        const bool valid = (unsigned long long)j_mine < (unsigned long long)N;
        if constexpr (BY_DISTANCE) {
            // A neighbour whose own last one is nearer than this point does not have it in its row; in the others it stands
            // among those at its distance, by id (unfilled slots, id -1, last).  A lane a neighbour: fewer sectors than the ids
            // have, and 32 searches in flight.
            const float d = valid ? d2[i * K + s_mine] : 0.0f;
            if (valid && d <= furthest[j_mine]) {
                const float *dj = d2 + (long long)j_mine * K;
                const int32_t *ij = ids + (long long)j_mine * K;
                int lo = 0, hi = K;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (dj[mid] < d) lo = mid + 1;
                    else hi = mid;
                }
                // Whole numbers and copies have most of a row at one distance, so its equals are searched too: 60,000 x 32 binary
                // features, K = 150 0.73 ms (walked through 3.6, by ids alone 0.93, points without equals 0.17).
                if (lo < K && ij[lo] != (int32_t)i) {
                    hi = K;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (dj[mid] == d && (uint32_t)ij[mid] < (uint32_t)i) lo = mid + 1;
                        else hi = mid;
                    }
                }
                if (lo < K && ij[lo] == (int32_t)i) acc_mine += p[(long long)j_mine * K + lo];
            }
            if (s_mine < K) P_rows[r * K + s_mine] = (float)((double)acc_mine / inv);
            continue;
        }
        unsigned left = __ballot_sync(0xffffffffu, valid);
        // kSymAhead neighbours' rows at a time: their loads are independent and in flight together (a warp that takes
        // one row after the other waits for each round trip to L2 in turn)
        while (left) {
            int j[kSymAhead], at[kSymAhead];
            const int32_t *rj[kSymAhead];
#pragma unroll
            for (int q = 0; q < kSymAhead; q++) {
                at[q] = left ? __ffs(left) - 1 : 32;
                left &= left - 1;
                j[q] = __shfl_sync(0xffffffffu, j_mine, at[q] & 31);
                if (at[q] == 32) j[q] = -1;
                rj[q] = ids + (long long)max(j[q], 0) * K;
            }
            float add[kSymAhead];
#pragma unroll
            for (int q = 0; q < kSymAhead; q++) add[q] = 0.0f;
            for (int u0 = 0; u0 < K; u0 += 32) {
                const int u = u0 + lane;
                int32_t v[kSymAhead];
#pragma unroll
                for (int q = 0; q < kSymAhead; q++) v[q] = (u < K && j[q] >= 0) ? rj[q][u] : -1;
#pragma unroll
                for (int q = 0; q < kSymAhead; q++)
                    if (v[q] == (int32_t)i && j[q] >= 0) add[q] += p[(long long)j[q] * K + u];
            }
            // matches are rare (at most one for a valid neighbour list): reduce only when some lane has one
#pragma unroll
            for (int q = 0; q < kSymAhead; q++) {
                if (__any_sync(0xffffffffu, add[q] != 0.0f)) {
                    float a = add[q];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                    if (lane == at[q]) acc_mine += a;
                }
            }
        }
        if (s_mine < K) P_rows[r * K + s_mine] = (float)((double)acc_mine / inv);
    }
}

// The entries the fixed-width P leaves out.  The fixed-width symmetrisation stores P_ij only where j is a neighbour
// of i; where j has i as a neighbour but not the other way round, the reference drops P_ji's mirror image
// (src/util/math_utils.cu:269-291).  A truly symmetric P = (p + p^T) / 2N has it: for every edge i -> j whose
// reverse is missing, row j gets the extra entry (column i, p_j|i / 2N).
// One warp per source row i (all N rows); PASS 0 counts the extra entries of the owned target rows, PASS 1 writes them
// (order inside a row: as the atomics fall, which only reorders a row's sum).
template <int PASS>
__global__ void __launch_bounds__(kSymWarps * 32)
reverse_only_kernel(const float *__restrict__ p, const int32_t *__restrict__ ids, long long N, int K, long long row_lo, long long row_hi,
                    int *__restrict__ count, const int *__restrict__ ptr, int *__restrict__ cursor, int32_t *__restrict__ ext_ids,
                    float *__restrict__ ext_val)
{
    const int lane = threadIdx.x & 31;
    const long long i = (long long)blockIdx.x * kSymWarps + (threadIdx.x >> 5);
    if (i >= N) return;
    const double inv = 2.0 * (double)N;
    for (int s0 = 0; s0 < K; s0 += 32) {
        const int s_mine = s0 + lane;
        int j_mine = -1;
        float p_mine = 0.0f;
        if (s_mine < K) {
            j_mine = ids[i * K + s_mine];
            p_mine = p[i * K + s_mine];
        }
        const int cnt = min(32, K - s0);
        for (int t = 0; t < cnt; t++) {
            const int j = __shfl_sync(0xffffffffu, j_mine, t);
            if (j < row_lo || j >= row_hi || j == i) continue;          // not an owned target, or the point itself
            const int32_t *rj = ids + (long long)j * K;
            bool found = false;
            for (int u = lane; u < K; u += 32) found |= rj[u] == (int32_t)i;
            if (__any_sync(0xffffffffu, found)) continue;               // mutual: the fixed-width entry has both halves
            if (lane == t) {
                const long long r = j - row_lo;
                if (PASS == 0) {
                    atomicAdd(&count[r], 1);
                } else {
                    const int at = ptr[r] + atomicAdd(&cursor[r], 1);
                    ext_ids[at] = (int32_t)i;
                    ext_val[at] = (float)((double)p_mine / inv);
                }
            }
        }
    }
}

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }
}  // namespace

// ptr: [rows + 1] ints (device), filled here; returns the number of extra entries in *count_host (synchronises st).
int launch_reverse_only_count(const float *p_all, const int32_t *ids_all, int64_t N, int K, int64_t row_lo, int64_t row_hi, int *ptr,
                              int64_t *count_host, cudaStream_t st)
{
    const long long rows = row_hi - row_lo;
    *count_host = 0;
    if (rows <= 0) return 0;
    B200_CUDA(cudaMemsetAsync(ptr, 0, sizeof(int) * (rows + 1), st));
    reverse_only_kernel<0><<<nblk(N, kSymWarps), kSymWarps * 32, 0, st>>>(p_all, ids_all, N, K, row_lo, row_hi, ptr, nullptr, nullptr, nullptr,
                                                                          nullptr);
    B200_CUDA(cudaGetLastError());
    B200_TRY(launch_exclusive_scan_i32(ptr, rows + 1, st));
    int total = 0;
    B200_CUDA(cudaMemcpyAsync(&total, ptr + rows, sizeof(int), cudaMemcpyDeviceToHost, st));
    B200_CUDA(cudaStreamSynchronize(st));
    if (total < 0) { set_error("symmetric P: more than 2^31 reverse-only entries"); return -4; }
    *count_host = total;
    return 0;
}

// cursor: [rows] ints of scratch (device)
int launch_reverse_only_fill(const float *p_all, const int32_t *ids_all, int64_t N, int K, int64_t row_lo, int64_t row_hi, const int *ptr,
                             int *cursor, int32_t *ext_ids, float *ext_val, cudaStream_t st)
{
    const long long rows = row_hi - row_lo;
    if (rows <= 0) return 0;
    B200_CUDA(cudaMemsetAsync(cursor, 0, sizeof(int) * rows, st));
    reverse_only_kernel<1><<<nblk(N, kSymWarps), kSymWarps * 32, 0, st>>>(p_all, ids_all, N, K, row_lo, row_hi, nullptr, ptr, cursor, ext_ids,
                                                                          ext_val);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_absmax(const float *v, int64_t n, unsigned int *max_enc, cudaStream_t st)
{
    if (n <= 0) return 0;
    const unsigned blocks = (unsigned)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
    absmax_kernel<<<blocks, 256, 0, st>>>(v, n, max_enc);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_perplexity(const float *d2, int64_t n_rows, int K, float perplexity, float eps, const unsigned int *max_enc,
                      float *p, float *betas, cudaStream_t st)
{
    if (n_rows <= 0) return 0;
    const size_t smem = (size_t)kPerpWarps * K * sizeof(float);
    constexpr size_t most = 200 * 1024;
    if (smem > most) { set_error("perplexity: num_neighbors too large for the shared-memory row buffer"); return -4; }
    // always to the most: another thread may be between this and its launch
    if (smem > 48 * 1024) B200_CUDA(cudaFuncSetAttribute(perplexity_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    perplexity_kernel<<<nblk(n_rows, kPerpWarps), kPerpWarps * 32, smem, st>>>(d2, n_rows, K, perplexity, eps, max_enc, p,
                                                                              betas);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int launch_symmetrize(const float *p_all, const int32_t *ids_all, int64_t N, int K, int64_t row_lo, int64_t row_hi,
                      float *P_rows, cudaStream_t st, const int32_t *visit, const float *d2, float *furthest)
{
    const long long n_rows = row_hi - row_lo;
    if (n_rows <= 0) return 0;
    if (d2 && furthest) {
        furthest_kernel<<<nblk(N, 256), 256, 0, st>>>(d2, N, K, furthest);
        B200_CUDA(cudaGetLastError());
    }
    if (d2 && furthest) symmetrize_kernel<true><<<nblk(n_rows, kSymWarps), kSymWarps * 32, 0, st>>>(p_all, ids_all, N, K, row_lo, n_rows, visit, d2, furthest, P_rows);
    else symmetrize_kernel<false><<<nblk(n_rows, kSymWarps), kSymWarps * 32, 0, st>>>(p_all, ids_all, N, K, row_lo, n_rows, visit, nullptr, nullptr, P_rows);
    B200_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace b200
