// A coarse partition of the points: nearest of at most kMaxCells sample points ("centres").
//
// The neighbour search visits queries and database rows cell by cell and skips database cells that no query of a block
// can reach (triangle inequality on these distances, knn_tc.cu); the blocked copy of P numbers the points by cells chained
// by distance (attractive_blocked.cu).  One assignment serves both.
#include <algorithm>

#include "session.h"

namespace b200 {
namespace {

constexpr int kPts = 128, kDims = 32, kThreads = 256;

// dist[i][c] = |x_i - centre_c| for rows lo + i, or for the centres themselves (lo < 0); cell[i] = the nearest (ties: lower
// index), own[i] = its distance (each optional).  Differences are squared and
// summed in fp32 (relative error below (D + 2) 2^-24: what the users of the distances allow for).  A block takes 128 rows
// and all centres, eight rows and four centres a thread: two instructions per row, centre and dimension, 0.2 ms for
// 10^6 x 50 and for 60,000 x 784 (a thread per row with its coordinates in registers: 0.53 ms at D = 50, and a kernel of
// its own for wide rows 0.63).
__global__ void __launch_bounds__(kThreads)
cell_distance_kernel(const float *__restrict__ X, int D, long long lo, long long n, const CellTable *__restrict__ tab, int cells,
                     float *__restrict__ dist, float *__restrict__ own, unsigned char *__restrict__ cell)
{
    __shared__ __align__(16) float xs[kDims][kPts + 4], cs[kDims][kMaxCells + 4];
    __shared__ float s_best[kPts][17];
    __shared__ unsigned char s_arg[kPts][16];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31, warp = tid >> 5;
    const long long i0 = (long long)blockIdx.x * kPts;
    float acc[8][4];
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] = 0.0f;
    for (int d0 = 0; d0 < D; d0 += kDims) {
        const int dlen = min(kDims, D - d0);
        __syncthreads();
        for (int r = warp; r < kPts; r += kThreads / 32)
            xs[lane][r] = (i0 + r < n && lane < dlen) ? X[(lo < 0 ? tab->centre_row[i0 + r] : lo + i0 + r) * D + d0 + lane] : 0.0f;
        for (int c = warp; c < kMaxCells; c += kThreads / 32)
            cs[lane][c] = (c < cells && lane < dlen) ? X[tab->centre_row[c] * D + d0 + lane] : 0.0f;
        __syncthreads();
#pragma unroll 4
        for (int d = 0; d < dlen; d++) {
            const float4 x0 = *reinterpret_cast<const float4 *>(&xs[d][ty * 8]), x1 = *reinterpret_cast<const float4 *>(&xs[d][ty * 8 + 4]);
            const float4 c4 = *reinterpret_cast<const float4 *>(&cs[d][tx * 4]);
            const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w}, c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    const float t = x[a] - c[b];
                    acc[a][b] = fmaf(t, t, acc[a][b]);
                }
        }
    }
#pragma unroll
    for (int a = 0; a < 8; a++) {
        const int r = ty * 8 + a;
        float best = INFINITY;
        int arg = 0;
#pragma unroll
        for (int b = 0; b < 4; b++) {
            acc[a][b] = sqrtf(acc[a][b]);
            if (tx * 4 + b < cells && acc[a][b] < best) { best = acc[a][b]; arg = tx * 4 + b; }
        }
        if (dist && i0 + r < n)
            *reinterpret_cast<float4 *>(dist + (size_t)(i0 + r) * kMaxCells + tx * 4) = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
        s_best[r][tx] = best;
        s_arg[r][tx] = (unsigned char)arg;
    }
    __syncthreads();
    if (tid < kPts && i0 + tid < n) {
        float best = s_best[tid][0];
        int arg = s_arg[tid][0];
        for (int t = 1; t < 16; t++)
            if (s_best[tid][t] < best) { best = s_best[tid][t]; arg = s_arg[tid][t]; }
        if (cell) cell[i0 + tid] = (unsigned char)arg;
        if (own) own[i0 + tid] = best;   // (+inf for a row of NaN: its cell is never skipped)
    }
}

// centres: one row from each of `cells` equal stretches of [lo, lo + n) at a hashed offset (an even spacing would alias with
// any periodic ordering of the data and could leave whole clusters without a centre)
__global__ void cell_centres_kernel(long long lo, long long n, int cells, CellTable *tab)
{
    const int c = threadIdx.x;
    if (c >= cells) return;
    const long long stretch = n / cells;
    const unsigned long long h = ((unsigned long long)(c + 1) * 0x9E3779B97F4A7C15ull) >> 20;
    tab->centre_row[c] = lo + (long long)c * stretch + (long long)(h % (unsigned long long)stretch);
}

// rank[c] = position of cell c in a greedy nearest-neighbour chain through the centres (start: cell 0), so that cells of one
// cluster end up next to each other.  One warp; dist: the centres' distances to one another.
__global__ void __launch_bounds__(32) cell_chain_kernel(const float *__restrict__ dist, int cells, int *__restrict__ rank)
{
    __shared__ float s_d[kMaxCells][kMaxCells + 1];
    const int lane = threadIdx.x;
    for (int a = 0; a < cells; a++)
        for (int b = lane; b < cells; b += 32) s_d[a][b] = dist[a * kMaxCells + b];
    __syncwarp();
    bool used0 = lane == 0, used1 = false;   // cells lane and lane + 32
    int cur = 0;
    if (lane == 0) rank[0] = 0;
    for (int k = 1; k < cells; k++) {
        // key: distance bits, then index (distances are >= 0)
        unsigned long long best = ~0ull;
        if (!used0 && lane < cells) best = (unsigned long long)__float_as_uint(s_d[cur][lane]) << 32 | (unsigned)lane;
        if (!used1 && lane + 32 < cells) {
            const unsigned long long o = (unsigned long long)__float_as_uint(s_d[cur][lane + 32]) << 32 | (unsigned)(lane + 32);
            best = o < best ? o : best;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
            best = t < best ? t : best;
        }
        cur = (int)(unsigned)best & (kMaxCells - 1);
        if (cur == lane) used0 = true;
        if (cur == lane + 32) used1 = true;
        if (lane == 0) rank[cur] = k;
    }
}

}  // namespace

// Cells of rows [lo, lo + n); buffers from the arena.  distances: keep those to all centres, for up to kCellRowsMax rows
// (256 bytes each, a fifth of what a set-up holds per point, and a search that goes through its queries in batches of as
// many computes them again for 0.2 ms a batch).  At least 2,048 rows a cell: cells are padded to whole tiles of 128
// where that matters, 3 % then.
int point_cells_build(PointCells *pc, const float *X, int D, int64_t lo, int64_t n, bool distances, DeviceArena &arena, cudaStream_t st)
{
    *pc = PointCells();
    pc->lo = lo;
    pc->n = n;
    pc->cells = point_cells_count(n);
    B200_TRY(arena.alloc((void **)&pc->tab, sizeof(CellTable)));
    if (distances && n <= kCellRowsMax) B200_TRY(arena.alloc((void **)&pc->dist, sizeof(float) * kMaxCells * (size_t)n));
    B200_TRY(arena.alloc((void **)&pc->own, sizeof(float) * (size_t)n));
    B200_TRY(arena.alloc((void **)&pc->cell, (size_t)n));
    cell_centres_kernel<<<1, kMaxCells, 0, st>>>(lo, n, pc->cells, pc->tab);
    B200_CUDA(cudaGetLastError());
    return point_cells_assign(*pc, X, D, lo, n, pc->dist, pc->own, pc->cell, st);
}

// distances and cells of other rows to the same centres
int point_cells_assign(const PointCells &pc, const float *X, int D, int64_t lo, int64_t n, float *dist, float *own, unsigned char *cell, cudaStream_t st)
{
    if (n <= 0) return 0;
    cell_distance_kernel<<<(unsigned)((n + kPts - 1) / kPts), kThreads, 0, st>>>(X, D, lo, n, pc.tab, pc.cells, dist, own, cell);
    B200_CUDA(cudaGetLastError());
    return 0;
}

int point_cells_chain(const PointCells &pc, const float *X, int D, int *rank, DeviceArena &arena, cudaStream_t st)
{
    float *between = nullptr;
    B200_TRY(arena.alloc((void **)&between, sizeof(float) * kMaxCells * kMaxCells));
    cell_distance_kernel<<<1, kThreads, 0, st>>>(X, D, -1, pc.cells, pc.tab, pc.cells, between, nullptr, nullptr);
    B200_CUDA(cudaGetLastError());
    cell_chain_kernel<<<1, 32, 0, st>>>(between, pc.cells, rank);
    B200_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace b200
