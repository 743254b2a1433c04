// Exact k-nearest-neighbour search by whole rows of distances: every canonical distance of a group of queries is
// written out, then a block per query selects its K smallest.
//
// Used where the query x database product is small: databases below the tensor-core search's range, the rows that
// search could not certify, and callers that must not allocate.  A search that keeps a running list per query
// (knn_exact_kernel) serves 64 queries per block and inserts survivors one at a time: at 1,500 points that is 24 blocks on
// 148 SMs, and half of the time goes into insertions.  Here the distances are a plain tiled product over all SMs (three
// rounded fp32 operations per pair and dimension, issued for two pairs at a time, the bound), and the selection ranks the few keys, held in registers, that
// lie below a bound from the smallest keys of groups (short rows, long lists: bisection on the keys' bits).  Measured on B200 (lists / now):
// 4,099 points of 64 dimensions, K = 16: 1.69 / 0.18 ms; 1,500 x 20, K = 32: 1.63 / 0.03 ms; five rows of 60,000 x 784:
// 4.4 / 0.4 ms.
#include <limits.h>

#include <type_traits>

#include <algorithm>

#include "session.h"

namespace b200 {
namespace {

constexpr int kTileP = 128;    // database points per tile
constexpr int kDims = 32;      // dimensions per shared-memory chunk
constexpr int kThreads = 256;

// Two canonical operations at a time: each half rounds as the single instruction does (kMinusZero2: common.cuh).  The fp32 pipe
// is as busy as with single instructions, but half as many are issued: 4,099 x 64, K = 16 211 -> 201 us,
// 10,000 x 100, K = 40 1,943 -> 1,827 (whole searches).
__device__ __forceinline__ void add_square2(unsigned long long &acc, unsigned long long q, unsigned long long minus_p, unsigned long long minus_zero)
{
    asm("{\n\t.reg .b64 t;\n\t"
        "add.rn.f32x2 t, %1, %2;\n\tfma.rn.f32x2 t, t, t, %3;\n\tadd.rn.f32x2 %0, %0, t;\n\t}"
        : "+l"(acc)
        : "l"(q), "l"(minus_p), "l"(minus_zero));
}

// dist[q * ld + p] = canonical distance (sequential over the dimensions, every operation rounded) of query q of the list
// and database row db_lo + p.  QT queries and eight points a thread, 16 QT queries and 128 points a block.
// Bound: the fp32 pipe, which the packed operations of a dimension take for 96 cycles a warp.
// AHEAD: the next chunk of dimensions is on its way in registers while one is worked on, and a query's value stands twice in
// shared memory, as the operation wants it; three blocks to an SM, as one wave of a round of 832 queries wants (122 registers and
// two blocks: 184 us at 4,099 x 64).  A launch of many waves hides the loads behind a fourth block instead and is bound by the
// pipe alone.  The line is where all blocks find a place at once, four to an SM.  Searches, us, AHEAD | not, blocks of a launch in
// brackets: 3,000 x 33, K = 8 (384) 72 | 83, 4,099 x 64, K = 16 (429) 176 | 208, 6,145 x 20, K = 40 (490) 200 | 210, 10,000 x 100, K = 40
// (474) 1,728 | 1,715; K = 240 2,150 x 257 (578) 215 | 216, 2,300 x 257 (648) 253 | 245, 3,500 x 257 (1,540) 494 | 468, 12,288 x 97 (8,128)
// 2,408 | 2,235.
// Launched behind the selection of the round before, it runs beside it up to its stores (see chained launches in common.cuh): with
// AHEAD 4,099 x 64 (16) 201 -> 181 us, 9,000 x 20 (150) 743 -> 586, 12,288 x 32 (48) 1,125 -> 947.
template <int QT, bool AHEAD>
__global__ void __launch_bounds__(kThreads, AHEAD ? 3 : 4)
dense_distance_kernel(const float *__restrict__ X, int D, long long q_lo, long long nq, const int *__restrict__ q_index, long long db_lo,
                      long long nd, float *dist, long long ld, unsigned long long minus_zero)
{
    constexpr int kTileQ = 16 * QT, kQs = kTileQ + (AHEAD ? 2 : 4), kPs = kTileP + 4, kWarps = kThreads / 32;
    __shared__ __align__(16) std::conditional_t<AHEAD, float2, float> Qs[kDims][kQs];
    __shared__ __align__(16) float Ps[kDims][kPs];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31, warp = tid >> 5;
    const long long p0 = (long long)blockIdx.x * kTileP, q0 = (long long)blockIdx.y * kTileQ;
    unsigned long long acc[QT][4];
#pragma unroll
    for (int a = 0; a < QT; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] = 0ull;
    // a warp reads 32 dimensions of one row at a time (coalesced) and stores them as a column
    auto query_at = [&](int k, int d0, bool in) {
        const long long pos = q0 + warp + k * kWarps;
        return in && pos < nq ? X[(q_index ? (long long)q_index[pos] : q_lo + pos) * D + d0 + lane] : 0.0f;
    };
    auto point_at = [&](int k, int d0, bool in) {
        const long long pos = p0 + warp + k * kWarps;
        return in && pos < nd ? X[(db_lo + pos) * D + d0 + lane] : 0.0f;
    };
    [[maybe_unused]] float qn[kTileQ / kWarps], pn[kTileP / kWarps];
    [[maybe_unused]] auto fetch = [&](int d0) {
        const bool in = lane < D - d0;
#pragma unroll
        for (int k = 0; k < kTileQ / kWarps; k++) qn[k] = query_at(k, d0, in);
#pragma unroll
        for (int k = 0; k < kTileP / kWarps; k++) pn[k] = point_at(k, d0, in);
    };
    if constexpr (AHEAD) fetch(0);
    for (int d0 = 0; d0 < D; d0 += kDims) {
        const int dlen = min(kDims, D - d0);
        __syncthreads();
        if constexpr (AHEAD) {
#pragma unroll
            for (int k = 0; k < kTileQ / kWarps; k++) Qs[lane][warp + k * kWarps] = make_float2(qn[k], qn[k]);
#pragma unroll
            for (int k = 0; k < kTileP / kWarps; k++) Ps[lane][warp + k * kWarps] = -pn[k];   // the difference as a sum
        } else {
#pragma unroll 4
            for (int k = 0; k < kTileQ / kWarps; k++) Qs[lane][warp + k * kWarps] = query_at(k, d0, lane < dlen);
#pragma unroll 4
            for (int k = 0; k < kTileP / kWarps; k++) Ps[lane][warp + k * kWarps] = -point_at(k, d0, lane < dlen);
        }
        __syncthreads();
        if constexpr (AHEAD)
            if (d0 + kDims < D) fetch(d0 + kDims);
#pragma unroll (AHEAD ? 8 : 4)
        for (int d = 0; d < dlen; d++) {
            unsigned long long qq[QT];
            if constexpr (!AHEAD) {
                float qv[QT];
                if constexpr (QT == 4) *reinterpret_cast<float4 *>(qv) = *reinterpret_cast<const float4 *>(&Qs[d][ty * 4]);
                else qv[0] = Qs[d][ty];
#pragma unroll
                for (int a = 0; a < QT; a++) qq[a] = pack(make_float2(qv[a], qv[a]));
            } else if constexpr (QT == 4) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(&Qs[d][ty * 4]), b = *reinterpret_cast<const ulonglong2 *>(&Qs[d][ty * 4 + 2]);
                qq[0] = a.x; qq[1] = a.y; qq[2] = b.x; qq[3] = b.y;
            } else {
                qq[0] = *reinterpret_cast<const unsigned long long *>(&Qs[d][ty]);
            }
            const ulonglong2 pa = *reinterpret_cast<const ulonglong2 *>(&Ps[d][tx * 4]), pb = *reinterpret_cast<const ulonglong2 *>(&Ps[d][64 + tx * 4]);
            const unsigned long long pv[4] = {pa.x, pa.y, pb.x, pb.y};
#pragma unroll
            for (int a = 0; a < QT; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) add_square2(acc[a][b], qq[a], pv[b], minus_zero);
        }
    }
    let_next_start();
    after_previous();   // the selection before this round reads dist
    // (rows of dist are padded to whole tiles: every store stays inside)
#pragma unroll
    for (int a = 0; a < QT; a++) {
        const long long q = q0 + ty * QT + a;
        if (q >= nq) continue;
        float *row = dist + q * ld + p0;
        const float2 d0 = unpack(acc[a][0]), d1 = unpack(acc[a][1]), d2 = unpack(acc[a][2]), d3 = unpack(acc[a][3]);
        *reinterpret_cast<float4 *>(row + tx * 4) = make_float4(d0.x, d0.y, d1.x, d1.y);
        *reinterpret_cast<float4 *>(row + 64 + tx * 4) = make_float4(d2.x, d2.y, d3.x, d3.y);
    }
}

// The sum over the block, for every thread.  buf: one int per warp and parity (two calls in flight share no slot).
__device__ __forceinline__ int block_sum(int v, int *buf)
{
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) t += buf[w];
    return t;
}

constexpr unsigned kInfBits = 0x7f800000u;   // distances are >= 0: their bits order like them; NaN lies above and never ranks
constexpr int kMaxDenseK = 512;
constexpr int kFewMore = 64;      // keys beyond K that are ranked rather than sorted out by further rounds of bisection
// Lists of up to kFoursMaxK take the groups of the bound from four threads' keys each, longer ones from one thread's, and beyond kGroupMaxK, or
// in rows of at most 2,048 keys, none: 256 smallest keys are ranked whatever the row's length (1,500 x 20, K = 90 39.5 us by a bound,
// 35 by bisection, 2,047 x 20, K = 150 66 / 54, 3,000 x 20, K = 150 118 / 118), and ranking the 256 ln(256 / (256 - K)) or so that lie at or
// below the bound takes their number's square (9,000 x 20, K = 150 758 / 887, K = 192 929 / 928).
constexpr int kFoursMaxK = 48;
constexpr int kGroupMaxK = 160;

// Blocks an SM: what the keys leave registers for (unasked, the compiler took 64 instead of 48 for 24 keys, 201 -> 209 us at 4,099 x 64).
constexpr int select_blocks(int kpt) { return kpt > 32 ? 3 : kpt > 16 ? 4 : kpt > 8 ? 5 : kpt > 4 ? 6 : 8; }

// One block per (query, segment).  The n values of segment s of query q start at val + q * ld + s * seg; with `ids` (IDS) they
// carry the ids at the same place (equal values in ascending order of id), else value j has id id_lo + s * seg + j.  The K
// smallest by (value, id), ascending, go to out row (q * segments + s), or, with out_rows, to row out_rows[q] - out_base;
// slots without a value get (+inf, INT_MAX), and where such slots of shorter lists come in again (ids given) they are no
// values: a neighbour infinitely far away is one, and precedes them.  KPT * 256 >= seg.
// LONG: lists of more than kFoursMaxK.
template <int KPT, bool IDS, bool LONG>
__global__ void __launch_bounds__(kThreads, select_blocks(KPT))
dense_select_kernel(const float *val, const int32_t *ids, long long ld, long long n_total, long long seg, int id_lo,
                    int K, const int *__restrict__ out_rows, long long out_base, float *out_d, int32_t *out_i)
{
    let_next_start();   // the distances of the next round touch nothing of this one's before they wait
    after_previous();
    __shared__ unsigned long long s_key[kMaxDenseK];
    __shared__ __align__(16) unsigned s_min[kThreads], s_four[kThreads / 4];
    __shared__ unsigned s_bound, s_least;
    __shared__ int s_sum[2][kThreads / 32];
    __shared__ unsigned s_lo[kThreads / 32], s_hi[kThreads / 32];
    __shared__ int s_n, s_before;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long q = blockIdx.y, s = blockIdx.x;
    const long long base = q * ld + s * seg;
    const int n = (int)min(seg, n_total - s * seg);
    unsigned key[KPT];
    unsigned lo = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < KPT; j++) {
        const int e = j * kThreads + tid;
        key[j] = e < n ? __float_as_uint(val[base + e]) : 0xffffffffu;
        if (IDS && key[j] == kInfBits && ids[base + e] == INT_MAX) key[j] = 0xffffffffu;
        lo = min(lo, key[j]);
        // A group's smallest key so far goes from thread to thread of the warp.  Were a group the keys of one thread, points whose
        // neighbours stand 256 apart (classes in turn, lines of a raster) would have whole classes in one group, and a bound with
        // thousands of keys below: 4,099 x 16, K = 90 255 us, so 155; 9,000 x 40, K = 16 1,166, so 784 (without a period: 151, 798).
        if (LONG || (j & 1)) lo = __shfl_sync(0xffffffffu, lo, (lane + 5) & 31);
    }
    auto id_of = [&](int e) { return IDS ? ids[base + e] : (int32_t)(id_lo + s * seg + e); };
    auto composed = [&](int j) { return (unsigned long long)key[j] << 32 | (unsigned)id_of(j * kThreads + tid); };
    const long long row = out_rows ? out_rows[q] - out_base : q * gridDim.x + s;
    if (tid == 0) { s_n = 0; s_before = 0; s_bound = s_least = 0xffffffffu; }
    unsigned hi = 0u;
    int known = 0;   // 1: hi is a key with at least K keys <= it; 2: and it is the K-th smallest
    // The K-th smallest of the smallest keys of disjoint groups bounds the K-th smallest key from above, and little more than K
    // keys lie below it.  Three barriers instead of the bisection's thirty: whole search of 4,099 x 64, K = 16 317 -> 226 us,
    // 1,500 x 20, K = 32 33 -> 25, 9,000 x 40 1,095 -> 840.
    if (!LONG || (KPT > 8 && K <= kGroupMaxK)) {
        constexpr int groups = LONG ? kThreads : kThreads / 4;
        s_min[tid] = lo;
        __syncthreads();
        if (tid < groups) {
            unsigned m = s_min[tid];
            if constexpr (!LONG) {   // the same lane of four warps; this is two warps' work
                const unsigned *const four = s_min + warp * 128 + lane;
                m = min(min(four[0], four[32]), min(four[64], four[96]));
                s_four[tid] = m;
                asm volatile("bar.sync 1, %0;" ::"n"(kThreads / 4) : "memory");
            }
            const unsigned *const all = LONG ? s_min : s_four;
            int at_or_below = 0;
#pragma unroll 4
            for (int u = 0; u < groups; u += 4) {
                const uint4 o = *reinterpret_cast<const uint4 *>(all + u);
                at_or_below += (o.x <= m) + (o.y <= m) + (o.z <= m) + (o.w <= m);
            }
            const unsigned least = __reduce_min_sync(0xffffffffu, m);
            m = __reduce_min_sync(0xffffffffu, at_or_below >= K ? m : 0xffffffffu);
            if (lane == 0) { atomicMin(&s_bound, m); atomicMin(&s_least, least); }
        }
        __syncthreads();
        const unsigned bound = s_bound;
        // 0: fewer than K groups have a key at all; 2: K groups have the smallest key of the row (copies of a point: 9,000 x 40, K = 16,
        // four points in five equal, 1,391 -> 850 us)
        known = bound > kInfBits ? 0 : bound == s_least ? 2 : 1;
        if (known == 1) {
            // one trip to the shared counter a thread (one a key: 9,000 x 20, K = 150 797 us, so 758; 6,145 x 20, K = 40 282, so 265)
            int mine_below = 0;
#pragma unroll
            for (int j = 0; j < KPT; j++) mine_below += key[j] <= bound;
            int slot = mine_below > 0 ? atomicAdd(&s_n, mine_below) : 0;
            if (mine_below > 0 && slot + mine_below <= kMaxDenseK)
#pragma unroll
                for (int j = 0; j < KPT; j++)
                    if (key[j] <= bound) s_key[slot++] = composed(j);
            __syncthreads();
            const int below = s_n;
            if (below <= kMaxDenseK) {
                for (int e = tid; e < below; e += kThreads) {
                    const unsigned long long mine = s_key[e];
                    int rank = 0;
                    for (int u = 0; u < below; u++) rank += s_key[u] < mine;
                    if (rank < K) {
                        out_d[row * K + rank] = __uint_as_float((unsigned)(mine >> 32));
                        out_i[row * K + rank] = (int32_t)(unsigned)mine;
                    }
                }
                return;
            }
            __syncthreads();   // more than there is room for
            if (tid == 0) s_n = 0;
        }
        if (known) hi = bound;
    }
    int valid = 0;
#pragma unroll
    for (int j = 0; j < KPT; j++)
        if (key[j] <= kInfBits) { valid++; if (!known) hi = max(hi, key[j]); }
    lo = __reduce_min_sync(0xffffffffu, lo);
    if (!known) hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) { s_lo[warp] = lo; s_hi[warp] = hi; }
    int turn = 0;
    valid = block_sum(valid, s_sum[turn++ & 1]);
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) { lo = min(lo, s_lo[w]); hi = max(hi, s_hi[w]); }
    // v: a bound with at least K keys <= v, few enough to rank, or else (ties) the K-th smallest key itself
    const int few = min(K + kFewMore, kMaxDenseK);
    bool ties = valid > few;
    unsigned v = ties ? hi : kInfBits;
    if (ties && known < 2) {
        unsigned a = lo, b = hi;
        bool first = known;   // the bound often is the K-th smallest key, one of many equal ones: the largest key below it first
        while (a < b) {
            const unsigned mid = first ? b - 1 : a + ((b - a) >> 1);
            first = false;
            int c = 0;
#pragma unroll
            for (int j = 0; j < KPT; j++) c += key[j] <= mid;
            c = block_sum(c, s_sum[turn++ & 1]);
            if (c >= K) { b = mid; if (c <= few) { ties = false; valid = c; break; } }
            else a = mid + 1;
        }
        v = b;
    }
    if (valid > 0) {
#pragma unroll
        for (int j = 0; j < KPT; j++)
            if (key[j] <= kInfBits && (ties ? key[j] < v : key[j] <= v)) s_key[atomicAdd(&s_n, 1)] = composed(j);
    }
    __syncthreads();
    if (ties) {
        const int room = K - s_n;
        const int at = s_n;
        for (int j = 0; j < KPT && s_before < room; j++) {
            bool eq = false;
#pragma unroll
            for (int t = 0; t < KPT; t++) eq = t == j ? key[t] == v : eq;
            const unsigned m = __ballot_sync(0xffffffffu, eq);
            if (lane == 0) s_sum[0][warp] = __popc(m);
            __syncthreads();
            int before = s_before + __popc(m & ((1u << lane) - 1u));
            for (int w = 0; w < warp; w++) before += s_sum[0][w];
            if (eq && before < room) s_key[at + before] = (unsigned long long)v << 32 | (unsigned)id_of(j * kThreads + tid);
            __syncthreads();
            if (tid == 0)
                for (int w = 0; w < kThreads / 32; w++) s_before += s_sum[0][w];
            __syncthreads();
        }
    }
    __syncthreads();
    // rank by counting: a few hundred keys at most
    const int got = ties ? K : valid;
    for (int e = tid; e < got; e += kThreads) {
        const unsigned long long mine = s_key[e];
        int rank = 0;
        for (int u = 0; u < got; u++) rank += s_key[u] < mine;
        if (rank < K) {
            out_d[row * K + rank] = __uint_as_float((unsigned)(mine >> 32));
            out_i[row * K + rank] = (int32_t)(unsigned)mine;
        }
    }
    for (int e = got + tid; e < K; e += kThreads) {
        out_d[row * K + e] = INFINITY;
        out_i[row * K + e] = INT_MAX;
    }
}

constexpr long long kMaxSegment = 48 * kThreads;   // values one block selects from (12,288)

template <bool IDS, bool LONG>
int launch_select_as(const float *val, const int32_t *ids, long long ld, long long n, long long seg, int segments, long long nq, int id_lo, int K,
                  const int *out_rows, long long out_base, float *out_d, int32_t *out_i, cudaStream_t st)
{
    const long long longest = std::min(n, seg);
    for (long long q = 0; q < nq; q += 65535) {   // grid.y
        const dim3 grid((unsigned)segments, (unsigned)std::min<long long>(65535, nq - q));
        const float *v = val + q * ld;
        const int32_t *i = ids ? ids + q * ld : nullptr;
        const int *r = out_rows ? out_rows + q : nullptr;
        float *od = out_rows ? out_d : out_d + q * segments * K;
        int32_t *oi = out_rows ? out_i : out_i + q * segments * K;
        cudaError_t launched = cudaSuccess;
        // A merge waits for the selection in front to end: placed beside it, its blocks share the few SMs that have room left
        // (200 of 20,000 rows, K = 240: merge 22 us for 11, all three kernels 68 for 62).
        auto launch = [&](auto kernel) {
            if (!IDS) {
                launched = launch_chained(kernel, grid, kThreads, 0, st, v, i, ld, n, seg, id_lo, K, r, out_base, od, oi);
                return;
            }
            kernel<<<grid, kThreads, 0, st>>>(v, i, ld, n, seg, id_lo, K, r, out_base, od, oi);
            launched = cudaGetLastError();
        };
        if (longest <= 4 * kThreads) launch(dense_select_kernel<4, IDS, LONG>);
        else if (longest <= 8 * kThreads) launch(dense_select_kernel<8, IDS, LONG>);
        else if (longest <= 16 * kThreads) launch(dense_select_kernel<16, IDS, LONG>);
        else if (longest <= 24 * kThreads) launch(dense_select_kernel<24, IDS, LONG>);
        else if (longest <= 32 * kThreads) launch(dense_select_kernel<32, IDS, LONG>);
        else launch(dense_select_kernel<48, IDS, LONG>);
        B200_CUDA(launched);
    }
    return 0;
}

template <bool IDS>
int launch_select(const float *val, const int32_t *ids, long long ld, long long n, long long seg, int segments, long long nq, int id_lo, int K,
                  const int *out_rows, long long out_base, float *out_d, int32_t *out_i, cudaStream_t st)
{
    const auto as = K > kFoursMaxK ? launch_select_as<IDS, true> : launch_select_as<IDS, false>;
    return as(val, ids, ld, n, seg, segments, nq, id_lo, K, out_rows, out_base, out_d, out_i, st);
}

// first: of a call.  What was queued before the call may write the points, so that launch waits for all of it; the later ones
// find this call's selection in front.
int launch_distances(const float *X, int D, int64_t q_lo, int64_t nq, const int *q_index, int64_t db_lo, int64_t nd, float *dist, long long ld, bool first,
                     cudaStream_t st)
{
    if (nd <= 0) return 0;
    const auto launch = [&](auto kernel, dim3 grid, int64_t q, int64_t m) {
        const int *index = q_index ? q_index + q : nullptr;
        if (!first) return launch_chained(kernel, grid, kThreads, 0, st, X, D, q_lo + q, m, index, db_lo, nd, dist + q * ld, ld, kMinusZero2);
        kernel<<<grid, kThreads, 0, st>>>(X, D, q_lo + q, m, index, db_lo, nd, dist + q * ld, ld, kMinusZero2);
        return cudaGetLastError();
    };
    const unsigned tiles = (unsigned)((nd + kTileP - 1) / kTileP);
    int device = 0, sms = 0;
    B200_CUDA(cudaGetDevice(&device));
    B200_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const auto launch_tiles = [&](auto ahead, auto plain, unsigned rows, int64_t q, int64_t m) {
        return launch((long long)tiles * rows <= 4ll * sms ? ahead : plain, dim3(tiles, rows), q, m);
    };
    // a short list of queries: 16 a block waste less of the tile
    if (nq > 48) {
        for (int64_t q = 0; q < nq; q += 65535 * 64) {
            const int64_t m = std::min<int64_t>(65535 * 64, nq - q);
            B200_CUDA(launch_tiles(dense_distance_kernel<4, true>, dense_distance_kernel<4, false>, (unsigned)((m + 63) / 64), q, m));
        }
    } else {
        B200_CUDA(launch_tiles(dense_distance_kernel<1, true>, dense_distance_kernel<1, false>, (unsigned)((nq + 15) / 16), 0, nq));
    }
    return 0;
}

long long padded(long long nd) { return (nd + kTileP - 1) / kTileP * kTileP; }
}  // namespace

// Queries of one round of several: alike, in whole blocks of 64, where `most` would leave a short last round (4,099 x 64: five
// rounds of 832, three blocks of distances an SM in each, instead of four of 960 and one of 259: 226 -> 211 us).
static int64_t even_round(int64_t nq, int64_t most)
{
    if (nq <= most || most < 64) return most;
    const int64_t rounds = (nq + most - 1) / most;
    return std::min(most, ((nq + rounds - 1) / rounds + 63) / 64 * 64);
}

bool knn_dense_supported(int K) { return K <= kMaxDenseK; }

// Queries [q_lo, q_lo + nq), or the nq rows that q_index lists, against database rows [db_lo, db_hi); the list of query
// number p goes to row p of ids / d2, of listed row g to row g - out_base.  Queues everything on st; the buffers come
// from tmp, which must outlive the work.
int knn_dense(const float *X, int D, int K, int64_t q_lo, int64_t nq, const int *q_index, int64_t out_base, int64_t db_lo, int64_t db_hi,
              int32_t *ids, float *d2, DeviceArena &tmp, cudaStream_t st)
{
    const long long nd = db_hi - db_lo, ld = padded(std::max<long long>(nd, 1));
    if (nq <= 0) return 0;
    if (!knn_dense_supported(K)) { set_error("knn_dense: K too large"); return -4; }
    const long long seg = nd <= kMaxSegment ? std::max<long long>(nd, 1) : kMaxSegment;
    const int segments = (int)std::max<long long>(1, (nd + seg - 1) / seg);
    // queries per round: at most 2^26 distances (256 MB), in whole blocks of the distance kernel (67 at 10^6 rows are two
    // blocks, the second with three queries: 3,000 rows 49 ms against 33)
    int64_t round = std::max<int64_t>(1, std::min<int64_t>(nq, (1ll << 26) / ld));
    if (round < nq && round >= 16) round -= round % (round >= 64 ? 64 : 16);
    round = even_round(nq, round);
    float *dist = nullptr, *part_d[2] = {nullptr, nullptr};
    int32_t *part_i[2] = {nullptr, nullptr};
    B200_TRY(tmp.alloc((void **)&dist, sizeof(float) * (size_t)round * ld));
    if (segments > 1)
        for (int k = 0; k < 2; k++) {
            B200_TRY(tmp.alloc((void **)&part_d[k], sizeof(float) * (size_t)round * segments * K));
            B200_TRY(tmp.alloc((void **)&part_i[k], sizeof(int32_t) * (size_t)round * segments * K));
        }
    for (int64_t q = 0; q < nq; q += round) {
        const int64_t m = std::min<int64_t>(round, nq - q);
        const int *index = q_index ? q_index + q : nullptr;
        float *final_d = q_index ? d2 : d2 + q * K;
        int32_t *final_i = q_index ? ids : ids + q * K;
        B200_TRY(launch_distances(X, D, q_lo + q, m, index, db_lo, nd, dist, ld, q == 0, st));
        if (segments == 1) {
            B200_TRY(launch_select<false>(dist, nullptr, ld, nd, seg, 1, m, (int)db_lo, K, index, out_base, final_d, final_i, st));
            continue;
        }
        // the best of every segment, then of those lists (a level more while they are too long for a block)
        B200_TRY(launch_select<false>(dist, nullptr, ld, nd, seg, segments, m, (int)db_lo, K, nullptr, 0, part_d[0], part_i[0], st));
        long long lists = segments;
        int from = 0;
        while (lists * K > kMaxSegment) {
            const long long per = kMaxSegment / K;   // lists that one block merges
            const long long next = (lists + per - 1) / per;
            B200_TRY(launch_select<true>(part_d[from], part_i[from], lists * K, lists * K, per * K, (int)next, m, 0, K, nullptr, 0, part_d[from ^ 1],
                                   part_i[from ^ 1], st));
            lists = next;
            from ^= 1;
        }
        B200_TRY(launch_select<true>(part_d[from], part_i[from], lists * K, lists * K, lists * K, 1, m, 0, K, index, out_base, final_d, final_i, st));
    }
    return 0;
}

template <bool LONG> static int load_select()
{
    cudaFuncAttributes a;
    const void *kernels[] = {(const void *)dense_select_kernel<4, false, LONG>,  (const void *)dense_select_kernel<8, false, LONG>,
                             (const void *)dense_select_kernel<16, false, LONG>, (const void *)dense_select_kernel<24, false, LONG>,
                             (const void *)dense_select_kernel<32, false, LONG>, (const void *)dense_select_kernel<48, false, LONG>};
    for (const void *k : kernels) B200_CUDA(cudaFuncGetAttributes(&a, k));
    return 0;
}

// loads every kernel that knn_dense_in_scratch may launch (a look at its attributes does)
int knn_dense_load()
{
    cudaFuncAttributes a;
    const void *kernels[] = {(const void *)dense_distance_kernel<1, true>, (const void *)dense_distance_kernel<1, false>, (const void *)dense_distance_kernel<4, true>,
                             (const void *)dense_distance_kernel<4, false>};
    for (const void *k : kernels) B200_CUDA(cudaFuncGetAttributes(&a, k));
    B200_TRY(load_select<false>());
    return load_select<true>();
}

// The same for all points against all, in scratch of `floats` floats that the caller owns; -1 when it is too small for
// that to be worth it (the caller then searches another way).
int knn_dense_in_scratch(const float *X, int64_t N, int D, int K, float *scratch, long long floats, int32_t *ids, float *d2, cudaStream_t st)
{
    const long long ld = padded(N);
    const int64_t most = floats / ld / 64 * 64;
    if (N > kMaxSegment || !knn_dense_supported(K) || most < 64) return -1;
    const int64_t round = even_round(N, most);
    for (int64_t q = 0; q < N; q += round) {
        const int64_t m = std::min<int64_t>(round, N - q);
        B200_TRY(launch_distances(X, D, q, m, nullptr, 0, N, scratch, ld, q == 0, st));
        B200_TRY(launch_select<false>(scratch, nullptr, ld, N, N, 1, m, 0, K, nullptr, 0, d2 + q * K, ids + q * K, st));
    }
    return 0;
}

}  // namespace b200
