// Exact k-nearest-neighbour search on the tensor cores (tcgen05 + TMEM): a kernel that keeps the whole inner
// dimension in shared memory (D <= 63) and a chunked one for wider points (knn_tc_wide_kernel).
//
// Replaces the reference's FAISS IVF-Flat call (src/util/distance_utils.cu:79-121, approximate).
// The result is the same as that of knn.cu's search: ids ordered by the canonical fp32 distance
// (sequential, unfused) with ties broken by index.  It is obtained in three steps:
//
//  1. Filter.  Ranking keys  key_ij = |x_j|^2 - 2 x_i.x_j  come straight out of the tensor cores: the
//     query operand is [x_i, 1], the database operand [-2 x_j, |x_j|^2] (padding columns of the inner
//     dimension carry the norm), each value split in a pair v = hi + lo and multiplied as three products
//     hi.hi + lo.hi + hi.lo accumulated in fp32 in TMEM.  By default the pairs are bf16 (kind::f16, K steps
//     of 16, keys accurate to 3 * 2^-16 of sum_k |x_ik||2 x_jk|; the norm travels in three or four columns);
//     B200TSNE_KNN_FILTER=tf32 selects TF32 pairs (K steps of 8, about 2^-20 of |x_i||x_j|) at nearly twice
//     the tensor-core time.  Either error is covered by the proof of step 3.  A block owns 256 queries (one
//     TMEM lane each per query tile) and
//     walks the database in tiles of 128 points; each epilogue thread compares its row of the
//     accumulator tile with a per-query threshold and appends the rare survivors to the query's
//     candidate buffer with plain stores, about 3 L of them (L = 128 or 256).  No N x N matrix is written.
//  2. Re-rank.  The canonical distance of the candidates that can be among the K best (their key is within twice the
//     filter's error of the K-th smallest; at most L) is evaluated exactly and they are ordered by (distance, id).
//  3. Proof.  Every point that is not evaluated has a key >= T (the threshold, or the smallest one left out), hence a
//     canonical distance >= (|x_i|^2 + T - E)(1 - theta) with E bounding the filter's error and theta the
//     rounding of the canonical sum.  If the K-th candidate distance is strictly below that bound the
//     first K are provably the exact answer; otherwise the row is flagged and recomputed by
//     an exact search.  The observed filter error on the candidates is checked against E as well.
//
// Operand staging: the prepared operands live in global memory as ready-made shared-memory images, one per 128-row tile
// (and chunk of the inner dimension for wide points), bf16 pairs in swizzled rows, TF32 pairs in no-swizzle core matrices
// (8 rows x 16 bytes contiguous; the two 16-byte halves of a K step 128 bytes apart; 8-row groups 256 bytes apart).  A
// tile is therefore ONE contiguous bulk copy (cp.async.bulk + mbarrier complete_tx) with no tensor map.
//
// Thresholds are FIXED per query before the scan that uses them.  Up to 393,216 rows a sample (16 N / 3 L points, spread over
// the database and scanned with a top-16 epilogue in registers) sets it at the key of rank ~16; beyond, in two further
// steps: every 16th tile against the sample's threshold (~300 candidates), then all tiles against the key of rank
// ~3L/16 of those, which about 3L points beat.  Nothing is compacted during a scan; the re-rank picks from the buffer by
// bisection on the key bits.  A row whose buffer overflows or ends with too few candidates is recomputed.
//
// Epilogue: a thread first reduces its 32 keys of a chunk to their minimum (a tree of independent
// min operations); only if that minimum beats the threshold, which becomes rare as the scan
// proceeds, does it locate and append the survivors.
//
// Order of the scan.  Queries and database rows are visited by Voronoi cells around sample points; a block
// skips the database cells none of its queries can reach under their thresholds (triangle inequality, see
// the knn_cells_* kernels), which leaves the result untouched and removes most tile pairs on clustered
// data.  A database image much larger than L2 is scanned in windows, one launch per window.
//
// Warp roles: a block serves QH = 2 query tiles (256 queries; 1 when the operand images are too wide for
// that) against every database tile, so a database image is fetched from L2 once per 256 queries.
// Warps 0 .. 8 QH - 1 are the epilogue, in 2 QH groups of four (TMEM lane quarter = warp % 4), then the
// bulk-copy producer warp and the MMA issuer / TMEM owner warp.  Two database stages and two accumulator
// buffers (of QH tiles each), so the MMAs of tile t+1 overlap the epilogue of tile t.  Measured at 400,000 x 50 before the
// last change of the epilogue: issue slots 77 % busy (390 instructions per MMA, most of them survivors' stores in divergent
// warps), tensor pipe 50 %: the epilogue bounds the narrow kernel; the wide one runs at the tensor pipe's rate
// (50,000 x 1,024: 15.4 TFLOP in 10.4 ms).
// Every wait has a time limit; on expiry the kernel sets an error flag, drains and frees its TMEM.
#include <limits.h>
#include <stdio.h>
#include <string.h>
#include <stdlib.h>

#include "common.cuh"

#include <cuda_bf16.h>

#include <algorithm>

namespace b200 {
namespace {

constexpr int TM = 128;             // queries per block = accumulator rows = TMEM lanes
constexpr int TN = 128;             // database points per tile = accumulator columns
constexpr int kBStages = 2;
constexpr int kAccBufs = 2;
// A block serves QH query tiles (QH = 2 when two query images and two database stages fit in shared
// memory, else 1): every database tile is multiplied with each of them, so the database image is read
// from L2 once per 128 * QH queries.  8 * QH epilogue warps, then the producer warp and the MMA warp;
// TMEM columns = kAccBufs * QH * TN.
constexpr int tc_threads(int QH) { return (8 * QH + 2) * 32; }
// Thresholds stay below the keys of padding rows, whose norm is 3e38: without the limit a sample of infinite keys (norms
// beyond the range of floats) lets padding pass.  Rows that find too few candidates below it are recomputed.
constexpr float kTauLimit = 2.9e38f;

// ------------------------------------------------------------------------------------------------
// PTX helpers
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: gives up after 4 s or as soon as another thread of the block has given up.  A waiting
// thread sleeps between polls: the producer and the MMA issuer share their schedulers with epilogue
// warps, and a busy poll would take every other issue slot from them.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, unsigned sleep_ns = 128,
                                          unsigned long long limit_ns = 4000000000ull)
{
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    int spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        __nanosleep(sleep_ns);
        if ((++spins & 63) == 0) {
            if (*abort_flag) return false;
            if (global_ns() - t0 > limit_ns) { *abort_flag = 1; return false; }
        }
    }
    return true;
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, 128 x 128 x 8, TF32 operands, fp32 accumulation
__device__ __forceinline__ void tc_mma_tf32(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, 128 x 128 x 16, bf16 operands, fp32 accumulation
__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
// 32 consecutive accumulator columns of this thread's TMEM lane: asynchronous issue ...
__device__ __forceinline__ void tc_ld32_issue(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32"
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15,"
        " %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
// ... and the wait that makes the registers valid (they are listed so that no use is scheduled above it)
__device__ __forceinline__ void tc_ld32_wait(uint32_t (&r)[32])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                   "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                   "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}

// three-input minimum (one instruction on sm_100)
__device__ __forceinline__ float min3(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Shared-memory matrix descriptor, K-major, no swizzle: core matrices of 8 rows x 16 bytes, the two
// 16-byte halves of a K step 128 bytes apart (leading offset), 8-row groups 256 bytes apart (stride
// offset); offsets are encoded in 16-byte units; bits 46-47 carry the descriptor version (1).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fff);
    d |= (uint64_t)(128 >> 4) << 16;
    d |= (uint64_t)(256 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}
// The same for a swizzled K-major image: rows of sw = 32, 64 or 128 bytes, 8-row groups 8 * sw bytes apart, the
// 16-byte pieces of a row exchanged by the XOR pattern of that width (layout type 6, 4 or 2 in bits 61-63; the
// leading offset is not used).  A K step inside a row is reached by adding its byte offset to the start address.
__device__ __forceinline__ uint64_t make_desc_swizzled(uint32_t saddr, uint32_t sw)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fff);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)((8u * sw) >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)(sw == 128u ? 2u : (sw == 64u ? 4u : 6u)) << 61;
    return d;
}
// Instruction descriptor: fp32 accumulate (bits 4-5 = 1), TF32 A and B (bits 7-9, 10-12 = 2), both
// K-major (bits 15, 16 = 0), N/8 in bits 17-22, M/16 in bits 24-28.
constexpr uint32_t kInstrDesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
// the same with bf16 A and B (format 1 of kind::f16); one K step is 32 operand bytes per row in either kind
constexpr uint32_t kInstrDescBf16 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
// two database tiles at once: 128 x 256 x 16
constexpr uint32_t kInstrDescBf16Pair = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(2 * TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);

// ------------------------------------------------------------------------------------------------
// operand preparation
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float to_tf32(float x)
{
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// offset (in floats) of element (row r, dimension k) inside a tile image part (hi or lo)
__device__ __forceinline__ size_t image_offset(int r, int k)
{
    return (size_t)(k >> 3) * 1024 + (size_t)(r >> 3) * 64 + (size_t)((k >> 2) & 1) * 32 + (size_t)(r & 7) * 4 + (k & 3);
}

// Rows of X named by `list` (-1 = padding) -> tile images [tiles][Dp/KC chunks][2 (hi, lo)][KC/8][1024 floats] (the
// narrow path has one chunk, KC = Dp; the wide path chunks of kWideKC inner dimensions) in query form
// [x, 1, 0...] or database form [-2x, |x|^2, 0...]; a padding row is all zeros as a query and carries a huge
// finite norm as a database point, so it never ranks.  norms (queries only): exact squared norms, double.
__global__ void __launch_bounds__(128)
knn_tc_prepare_kernel(const float *__restrict__ X, const int *__restrict__ list, int D, int Dp, int KC, int db_form,
                      float *__restrict__ img, double *__restrict__ norms)
{
    const long long tile = blockIdx.x;
    const int r = threadIdx.x;
    const long long pos = tile * TM + r;
    const int i = list[pos];
    float *im_tile = img + (size_t)tile * 2 * Dp * 128;
    const size_t part = (size_t)KC * 128;
    double n2 = 0.0;
    for (int k = 0; k < D; k++) {
        const float x = (i >= 0) ? X[(long long)i * D + k] : 0.0f;
        n2 += (double)x * (double)x;
    }
    for (int k = 0; k < Dp; k++) {
        float v = 0.0f;
        if (k < D) {
            const float x = (i >= 0) ? X[(long long)i * D + k] : 0.0f;
            v = db_form ? -2.0f * x : x;
        } else if (k == D) {
            v = db_form ? ((i >= 0) ? (float)n2 : 3.0e38f) : ((i >= 0) ? 1.0f : 0.0f);
        }
        const float vh = to_tf32(v);
        float *im = im_tile + (size_t)(k / KC) * 2 * part;
        im[image_offset(r, k % KC)] = vh;
        im[part + image_offset(r, k % KC)] = to_tf32(v - vh);
    }
    if (norms) norms[pos] = n2;
}

// The bf16 form of the images: v = hi + lo + r with hi, lo in bf16 (round to nearest) and |r| <= 2^-16 |v|; an image
// has half the bytes per inner dimension of a TF32 one, [tiles][Dp/KC chunks][2 (hi, lo)][KC * 128 values].  Two columns
// carry the norm (its bf16 pair and the pair of what that pair leaves over: 32 significant bits), against 1, 1 in the
// query form.  A part is rows of sw bytes (sw / 2 values), blocks of 128 rows one after the other along
// the inner dimension; inside a block the 16-byte piece p of row r sits where piece p ^ ((r * sw / 128) mod (sw / 16))
// would (the shared-memory swizzle of that width, which the tensor core undoes when it reads: operands in this
// form are fetched about twice as fast as core matrices without swizzle, measured).  Offset in values.
__device__ __forceinline__ size_t image_offset_bf16(int r, int k, int sw)
{
    const int per_row = sw >> 1;
    const int block = k / per_row;
    unsigned off = (unsigned)r * (unsigned)sw + (unsigned)(k % per_row) * 2u;   // bytes inside the block
    off ^= ((off >> 7) & ((unsigned)(sw >> 4) - 1u)) << 4;
    return (size_t)block * 64 * sw + (off >> 1);
}

// The narrow kernel's images are packed (whole >= 0): K steps of 16 columns, first the hi parts of the `whole` full groups of 16
// dimensions, then their lo parts, then the r = D mod 16 dimensions left over with all three products side by side:
//   query     [x_hi | x_lo | x_hi | 1 1 1]        database  [b_hi | b_hi | b_lo | the norm in three pieces]
// in ceil((3 r + 3) / 16) steps that are multiplied once.  With whole steps for what is left (and the norm's pair of columns)
// 50 dimensions took 12 MMAs a tile pair instead of 10, 20 took 6 instead of 4, and 57 to 63 an image of 64 KB.

// What the three products drop is bounded per pair from the actual leftovers: with a, b the data columns of a
// query and a database operand, a = a_hi + a_lo + a_r,  |dropped| <= |a_lo||b_lo| + |a - a_r||b_r| + |a_r||b - b_r|
// + |a_r||b_r| (Cauchy-Schwarz on the leftover vectors).  Queries record |a_lo| and |a_r| (res), the database the
// largest |b_lo|/|b| and |b_r|/|b| over its rows (rho_bits: float bits, raised with atomicMax).
//
// A block makes one tile image: 64 dimensions of its 128 rows at a time go through shared memory, so that rows are read
// and 16-byte pieces of the image written coalesced (a thread per row, as the TF32 form has it, touches 32 sectors per
// load: 1.2 ms for 10^6 rows of 50 dimensions, 0.56 ms for 50,000 of 1,024; now 0.12 and 0.10).  Xp (optional): the rows in
// list order, Xp[pos] = X[list[pos]], zeros for padding: the re-rank reads ~100 candidate rows per query, and in cell order
// the candidates of neighbouring queries share a few megabytes that stay in L2.
constexpr int kPrepDims = 64;
__global__ void __launch_bounds__(256)
knn_tc_prepare_bf16_kernel(const float *__restrict__ X, const int *__restrict__ list, int D, int Dp, int KC, int sw, int whole, int db_form,
                           __nv_bfloat16 *__restrict__ img, double *__restrict__ norms, float2 *__restrict__ res,
                           int *__restrict__ rho_bits, float *__restrict__ Xp)
{
    __shared__ float xs[TM][kPrepDims + 1];
    __shared__ float s_nf[TM], s_rest[TM];
    __shared__ int s_row[TM];
    const long long tile = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < TM) s_row[tid] = list[tile * TM + tid];
    __nv_bfloat16 *im_tile = img + (size_t)tile * 2 * Dp * 128;
    const size_t part = (size_t)KC * 128;
    const int row = tid >> 1, half = tid & 1;   // two threads share a row's sums
    double n2 = 0.0, lo2 = 0.0, r2 = 0.0;       // squared norms of the row, of its lo parts and of its leftovers
    const int k_end = whole >= 0 ? kPrepDims : Dp;   // (a packed row has fewer than 64 dimensions)
    for (int k0 = 0; k0 < k_end; k0 += kPrepDims) {
        __syncthreads();
        for (int r = warp; r < TM; r += 8) {
            const int i = s_row[r];
#pragma unroll
            for (int h = 0; h < kPrepDims; h += 32) {
                const int k = k0 + h + lane;
                const float x = (i >= 0 && k < D) ? X[(long long)i * D + k] : 0.0f;
                xs[r][h + lane] = x;
                if (Xp && k < D) Xp[(tile * TM + r) * D + k] = x;
            }
        }
        __syncthreads();
        if (k0 < D) {
            float lo_sum = 0.0f, left_sum = 0.0f;   // bounds, rounded up below: float sums of 32 squares will do
            for (int m = 0; m < kPrepDims / 2; m++) {
                const float x = xs[row][2 * m + half];
                n2 += (double)x * (double)x;
                const float rest = x - __bfloat162float(__float2bfloat16_rn(x));
                const float lo = __bfloat162float(__float2bfloat16_rn(rest)), left = rest - lo;
                lo_sum = fmaf(lo, lo, lo_sum);
                left_sum = fmaf(left, left, left_sum);
            }
            lo2 += (double)lo_sum;
            r2 += (double)left_sum;
        }
        if (k0 + kPrepDims > D) {   // the columns from D on carry the norm
            const double total = n2 + __shfl_xor_sync(0xffffffffu, n2, 1);
            const float nf = s_row[row] >= 0 ? (float)total : 3.0e38f;
            const float hi = __bfloat162float(__float2bfloat16_rn(nf));
            if (half == 0) {
                s_nf[row] = nf;
                s_rest[row] = (nf - hi) - __bfloat162float(__float2bfloat16_rn(nf - hi));   // both differences are exact in fp32
            }
            __syncthreads();
        }
        if (whole >= 0) {
            const int n16 = 16 * whole, rest = D - n16;
            for (int idx = tid; idx < TM * (Dp / 4); idx += 256) {
                const int r = idx & (TM - 1), c0 = (idx >> 7) * 8;
                __align__(16) __nv_bfloat16 out[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const int c = c0 + e, j = c - 2 * n16;   // j: column of the remainder's steps
                    int k = c < n16 ? c : c - n16;
                    bool low = c >= n16;
                    if (j >= 0) {
                        const int third = j < rest ? 0 : (j < 2 * rest ? 1 : (j < 3 * rest ? 2 : 3));
                        k = third < 3 ? n16 + j - third * rest : -1;
                        low = third == (db_form ? 2 : 1);
                    }
                    float v = 0.0f;
                    if (k >= 0) {
                        v = db_form ? -2.0f * xs[r][k] : xs[r][k];
                        const float hi = __bfloat162float(__float2bfloat16_rn(v));
                        v = low ? v - hi : hi;
                    } else if (j < 3 * rest + 3) {   // the norm in three pieces of 8 bits, against ones
                        const float nf = s_nf[r], hi = __bfloat162float(__float2bfloat16_rn(nf));
                        const int piece = j - 3 * rest;
                        v = piece == 0 ? hi : (piece == 1 ? nf - hi : s_rest[r]);
                        if (!db_form) v = s_row[r] >= 0 ? 1.0f : 0.0f;
                    }
                    out[e] = __float2bfloat16_rn(v);
                }
                *reinterpret_cast<uint4 *>(im_tile + image_offset_bf16(r, c0, sw)) = *reinterpret_cast<const uint4 *>(out);
            }
            break;
        }
        for (int idx = tid; idx < TM * (kPrepDims / 8); idx += 256) {
            const int r = idx & (TM - 1), o = (idx >> 7) * 8, k = k0 + o;
            if (k >= Dp) break;
            const bool real = s_row[r] >= 0;
            __align__(16) __nv_bfloat162 hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                float v[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int kk = k + e + u;
                    const float x = xs[r][o + e + u];
                    v[u] = kk < D ? (db_form ? -2.0f * x : x) : 0.0f;
                    if (kk == D) v[u] = db_form ? s_nf[r] : (real ? 1.0f : 0.0f);
                    if (kk == D + 1) v[u] = db_form ? s_rest[r] : (real ? 1.0f : 0.0f);
                }
                hi[e / 2] = __floats2bfloat162_rn(v[0], v[1]);
                lo[e / 2] = __floats2bfloat162_rn(v[0] - __low2float(hi[e / 2]), v[1] - __high2float(hi[e / 2]));
            }
            __nv_bfloat16 *im = im_tile + (size_t)(k / KC) * 2 * part;
            const size_t at = image_offset_bf16(r, k % KC, sw);
            *reinterpret_cast<uint4 *>(im + at) = *reinterpret_cast<const uint4 *>(hi);
            *reinterpret_cast<uint4 *>(im + part + at) = *reinterpret_cast<const uint4 *>(lo);
        }
    }
    n2 += __shfl_xor_sync(0xffffffffu, n2, 1);
    lo2 += __shfl_xor_sync(0xffffffffu, lo2, 1);
    r2 += __shfl_xor_sync(0xffffffffu, r2, 1);
    const long long pos = tile * TM + row;
    if (half == 0) {
        if (norms) norms[pos] = n2;
        if (res) res[pos] = make_float2((float)(sqrt(lo2) * 1.00001), (float)(sqrt(r2) * 1.00001));   // rounded up
    }
    if (rho_bits) {
        float rl = 0.0f, rr = 0.0f;   // relative to the row: the factor -2 of the database form cancels
        if (s_row[row] >= 0 && n2 > 0.0) {
            rl = (float)(sqrt(lo2 / n2) * 1.00001);
            rr = (float)(sqrt(r2 / n2) * 1.00001);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            rl = fmaxf(rl, __shfl_xor_sync(0xffffffffu, rl, o));
            rr = fmaxf(rr, __shfl_xor_sync(0xffffffffu, rr, o));
        }
        if (lane == 0) {   // non-negative floats: integer order == float order
            atomicMax(rho_bits + 0, __float_as_int(rl));
            atomicMax(rho_bits + 1, __float_as_int(rr));
        }
    }
}

// ------------------------------------------------------------------------------------------------
// cells: a coarse partition of the points that lets a block skip database tiles no query of it can reach
// ------------------------------------------------------------------------------------------------
// Both the database rows and the queries of a search are visited in the order of a partition into at
// most kMaxCells Voronoi cells around sample points (cells.cu).  Database cells start on tile
// boundaries (padding rows in between), so a cell is a run of whole tiles; for every cell the largest
// distance r_c of a member to its centre is known.  Once a query's threshold is fixed, no point of cell c
// can pass it if  |x_q - centre_c| - r_c  exceeds the threshold distance (triangle inequality), and a block
// skips the cells that none of its queries can reach.  On clustered data most tile pairs disappear; on
// data without structure nothing is lost but a fraction of a millisecond.  The visiting order also keeps the rows that the
// re-rank of neighbouring queries reads together in L2.
constexpr int kCellThreads = 256;

__global__ void knn_cells_reset_kernel(CellTable *tab)
{
    const int c = threadIdx.x;
    if (c >= kMaxCells) return;
    tab->radius_bits[c] = 0u;
    tab->db_count[c] = tab->q_count[c] = 0;
    tab->db_cursor[c] = tab->q_cursor[c] = 0;
}

// members of every cell among the n rows of cell and, for the database, r_c from the rows' distances to their own centre
__global__ void __launch_bounds__(kCellThreads)
knn_cells_count_kernel(const unsigned char *__restrict__ cell, const float *__restrict__ own, long long n, CellTable *tab, int is_db)
{
    __shared__ int s_cnt[kMaxCells];
    __shared__ unsigned int s_rad[kMaxCells];
    for (int c = threadIdx.x; c < kMaxCells; c += kCellThreads) { s_cnt[c] = 0; s_rad[c] = 0u; }
    __syncthreads();
    for (long long i = (long long)blockIdx.x * kCellThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kCellThreads) {
        const int c = cell[i];
        atomicAdd(&s_cnt[c], 1);
        if (is_db) atomicMax(&s_rad[c], __float_as_uint(own[i]));   // >= 0: orders like the bits
    }
    __syncthreads();
    for (int c = threadIdx.x; c < kMaxCells; c += kCellThreads) {
        if (s_cnt[c]) atomicAdd(is_db ? &tab->db_count[c] : &tab->q_count[c], s_cnt[c]);
        if (is_db && s_rad[c]) atomicMax(&tab->radius_bits[c], s_rad[c]);
    }
}

// list positions of the cells: database cells padded to whole tiles, query cells back to back
__global__ void knn_cells_layout_kernel(int cells, CellTable *tab)
{
    if (threadIdx.x != 0) return;
    int db = 0, q = 0;
    for (int c = 0; c < cells; c++) {
        tab->db_start[c] = db;
        tab->q_start[c] = q;
        db += (tab->db_count[c] + TN - 1) / TN * TN;
        q += tab->q_count[c];
    }
    for (int c = cells; c <= kMaxCells; c++) { tab->db_start[c] = db; tab->q_start[c] = q; }
}

// list[start(cell) + rank within the cell] = row; the order inside a cell is arbitrary (it decides which
// points share a tile, never the result)
__global__ void __launch_bounds__(kCellThreads)
knn_cells_scatter_kernel(const unsigned char *__restrict__ cell, long long lo, long long n, int cells, CellTable *tab, int is_db,
                         int *__restrict__ list)
{
    __shared__ int s_cnt[kMaxCells], s_base[kMaxCells];
    for (int c = threadIdx.x; c < kMaxCells; c += kCellThreads) s_cnt[c] = 0;
    __syncthreads();
    const long long i = (long long)blockIdx.x * kCellThreads + threadIdx.x;
    int c = 0, local = 0;
    if (i < n) {
        c = cell[i];
        local = atomicAdd(&s_cnt[c], 1);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < cells; k += kCellThreads)
        if (s_cnt[k]) s_base[k] = atomicAdd(is_db ? &tab->db_cursor[k] : &tab->q_cursor[k], s_cnt[k]);
    __syncthreads();
    if (i < n) list[(is_db ? tab->db_start[c] : tab->q_start[c]) + s_base[c] + local] = (int)(lo + i);
}

__global__ void knn_iota_kernel(int *__restrict__ list, long long lo, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) list[i] = (int)(lo + i);
}

// One block per filter block (qpc = its queries): which cells can hold a point that passes the threshold of
// at least one of its queries?  Their tile ranges (in units of two tiles for the wide kernel), merged where adjacent, are
// the block's segments.
// q_dist: distances of row q_lo + r to the centres at row r.  Rounding: a distance carries a relative error of at most
// (D + 2) 2^-25, the inequality is tested with `margin` = 1e-4 more than twice that; a comparison that involves a NaN keeps
// the cell.
__global__ void __launch_bounds__(kCellThreads)
knn_cells_segments_kernel(const float *__restrict__ q_dist, long long q_lo, const int *__restrict__ qlist, long long nq, int qpc,
                          const float *__restrict__ tau, const double *__restrict__ norms_q, int cells, float margin, int pair_tiles,
                          const CellTable *__restrict__ tab, int2 *__restrict__ segs, int *__restrict__ nseg)
{
    __shared__ int s_keep[kMaxCells];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = threadIdx.x; c < kMaxCells; c += kCellThreads) s_keep[c] = 0;
    __syncthreads();
    float radius[2];
    bool keep[2] = {false, false};
#pragma unroll
    for (int h = 0; h < 2; h++) radius[h] = __uint_as_float(tab->radius_bits[lane + 32 * h]) * (1.0f + margin);
    // a warp per query, a lane per cell (and the cell 32 further on)
    for (int j = warp; j < qpc; j += kCellThreads / 32) {
        const long long q = (long long)blockIdx.x * qpc + j;
        if (q >= nq) break;
        const double R2 = norms_q[q] + (double)tau[q];   // a point passes if its squared distance is below this
        if (R2 <= 0.0) continue;
        const float R = (float)sqrt(R2) * 1.0001f;
        const float *d = q_dist + (size_t)(qlist[q] - q_lo) * kMaxCells;
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (!(d[lane + 32 * h] * (1.0f - margin) - radius[h] > R)) keep[h] = true;
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
        if (keep[h]) s_keep[lane + 32 * h] = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        int n = 0;
        int2 *out = segs + (size_t)blockIdx.x * kMaxCells;
        for (int c = 0; c < cells; c++) {
            if (!s_keep[c] || tab->db_count[c] == 0) continue;
            int a = tab->db_start[c] / TN, b = tab->db_start[c + 1] / TN;
            if (pair_tiles) { a /= 2; b = (b + 1) / 2; }   // a pair may hold the edge tiles of two cells
            if (n > 0 && out[n - 1].y >= a) out[n - 1].y = max(out[n - 1].y, b);
            else out[n++] = make_int2(a, b);
        }
        nseg[blockIdx.x] = n;
    }
}

__global__ void knn_single_segment_kernel(int2 *segs, int *nseg, int tiles)
{
    segs[0] = make_int2(0, tiles);
    nseg[0] = 1;
}

// How many blocks divide the tiles of one block of queries: `most` are launched, and as the cells leave a block of queries
// anything between all tiles and a handful, each decides by what is left of its walk: shares of at least `share` tiles, or
// of four where that only takes SMs that would idle (`idle` blocks a block of queries).
struct ScanParts {
    int most = 1, idle = 1, share = 1;
    __host__ __device__ int of(int tiles) const
    {
        int n = tiles / share;
        const int free = tiles / 4 < idle ? tiles / 4 : idle;
        if (n < free) n = free;
        if (n > most) n = most;
        return n < 1 ? 1 : n;
    }
};
// The database tiles of a block in scan order: the tiles of its segments that are multiples of `stride` and lie
// in the window [win_lo, win_hi) of the launch, and of these the share of block `part` where several blocks divide them.
// The producer, the MMA issuer and the epilogue each walk the same sequence.
template <bool DIVIDED>
struct TileWalk {
    const int2 *segs;
    int nseg, stride, win_lo, win_hi, s, t, end, skip, left, parts;
    __device__ TileWalk(const int2 *segs_, int nseg_, int stride_, int win_lo_, int win_hi_, int part = 0, ScanParts p = ScanParts())
        : segs(segs_), nseg(nseg_), stride(stride_), win_lo(win_lo_), win_hi(win_hi_), s(-1), t(0), end(0), skip(0), left(INT_MAX), parts(1)
    {
        if (DIVIDED && p.most > 1) {
            long long total = 0;
            for (int i = 0; i < nseg; i++) {
                open(i);
                total += tiles();
            }
            t = end = 0;
            parts = p.of((int)total);
            skip = part < parts ? (int)(total * part / parts) : 0;
            left = part < parts ? (int)(total * (part + 1) / parts) - skip : 0;
        }
    }
    __device__ void open(int i)
    {
        const int2 g = segs[i];
        t = (max(g.x, win_lo) + stride - 1) / stride * stride;
        end = min(g.y, win_hi);
    }
    __device__ int tiles() const { return t < end ? (end - t + stride - 1) / stride : 0; }
    __device__ bool next(int &tile)
    {
        if (DIVIDED && left <= 0) return false;
        while (t >= end) {
            if (++s >= nseg) return false;
            open(s);
            if (DIVIDED && skip > 0) {
                const int over = min(skip, tiles());
                skip -= over;
                t += over * stride;
            }
        }
        if (DIVIDED) left--;
        tile = t;
        t += stride;
        return true;
    }
};

// Where several blocks share a query's buffer, the slots for the n keys of a chunk that passed are taken with one atomic
// addition.  Returns the first; `room` = how many of them exist.  A count beyond the segment says that keys were lost (and
// bit 30, which the thread that met the end sets, stops every block that starts on the query later).
__device__ __forceinline__ int take_slots(int *count, int n, int seg_cap, int &room)
{
    const int c = atomicAdd(count, n);
    const int first = c & 0x3fffffff;
    room = seg_cap - first;
    if (room < n && !(c & 0x40000000)) atomicOr(count, 0x40000000);
    return first;
}

// ------------------------------------------------------------------------------------------------
// filter kernel
// ------------------------------------------------------------------------------------------------
struct TcShared {
    uint64_t full_a;
    uint64_t full_b[kBStages];
    uint64_t empty_b[kBStages];
    uint64_t acc_full[kAccBufs];
    uint64_t acc_empty[kAccBufs];
    uint32_t tmem_base;
    int abort_flag;
};

// The MMAs of one accumulator tile: three products over F K steps, then S K steps once (the packed remainder of bf16
// images); off16: offsets of the image's K steps, hi, lo, remainder.  Every descriptor is a register plus a register.
// F and S are template arguments so that the loops unroll into independent instruction sequences: one thread issues
// every MMA of the block, and whatever it computes per MMA shows in the kernel's time.
template <bool BF16, int F, int S>
__device__ __forceinline__ void tc_issue_products(uint32_t d_tmem, uint64_t a, uint64_t b, const uint32_t (&off16)[2 * F + S])
{
    auto mma = [&](int i, int j, uint32_t accumulate) {
        if (BF16) tc_mma_bf16(d_tmem, a + off16[i], b + off16[j], kInstrDescBf16, accumulate);
        else tc_mma_tf32(d_tmem, a + off16[i], b + off16[j], kInstrDesc, accumulate);
    };
#pragma unroll
    for (int ks = 0; ks < F; ks++) mma(ks, ks, ks ? 1u : 0u);      // hi . hi
#pragma unroll
    for (int ks = 0; ks < F; ks++) mma(F + ks, ks, 1u);            // lo . hi
#pragma unroll
    for (int ks = 0; ks < F; ks++) mma(ks, F + ks, 1u);            // hi . lo
#pragma unroll
    for (int ks = 0; ks < S; ks++) mma(2 * F + ks, 2 * F + ks, (F || ks) ? 1u : 0u);
}

// The MMA issuer's walk over the block's database tiles (one thread).  a16 / b16 / end16: the block's images in
// 16-byte units of shared memory; span16: what one K step reads beyond its start.  Every tile's descriptors are
// checked against that range before they are used (an MMA that reads outside the block's shared memory is a fault).
template <int QH, bool BF16, int F, int S, bool DIVIDED>
__device__ __noinline__ void tc_issue_walk(TcShared *shp, volatile int *abort_flag, TileWalk<DIVIDED> walk, uint32_t tmem_base, uint64_t no_addr,
                                           uint32_t a16, uint32_t b16, uint32_t image16, uint32_t spr_log, uint32_t block16,
                                           uint32_t in_row16, uint32_t span16, uint32_t end16)
{
    TcShared &sh = *shp;
    const uint32_t spr_mask = (1u << spr_log) - 1u;
    uint32_t off16[2 * F + S];
    uint32_t reach16 = 0;   // the furthest an image's K steps read
#pragma unroll
    for (int ks = 0; ks < 2 * F + S; ks++) {
        off16[ks] = ((uint32_t)ks >> spr_log) * block16 + ((uint32_t)ks & spr_mask) * in_row16;
        reach16 = max(reach16, off16[ks] + span16);
    }
    int tile;
    for (long long t = 0; walk.next(tile); t++) {
        const int s = (int)(t % kBStages), acc = (int)(t % kAccBufs);
        const uint32_t ph_s = (uint32_t)((t / kBStages) & 1), ph_b = (uint32_t)((t / kAccBufs) & 1);
        if (!mbar_wait(&sh.acc_empty[acc], ph_b ^ 1u, abort_flag)) break;
        if (!mbar_wait(&sh.full_b[s], ph_s, abort_flag)) break;
        tc_fence_after();
        const uint32_t bs16 = b16 + (uint32_t)s * image16;
        if (reach16 > image16 || a16 + QH * image16 > b16 || bs16 + image16 > end16) { *abort_flag = 1; break; }
        const uint64_t b = no_addr + (uint64_t)bs16;
#pragma unroll
        for (int h = 0; h < QH; h++) {
            const uint64_t a = no_addr + (uint64_t)(a16 + (uint32_t)h * image16);
            tc_issue_products<BF16, F, S>(tmem_base + (uint32_t)((acc * QH + h) * TN), a, b, off16);
        }
        tc_commit(&sh.empty_b[s]);    // the stage may be refilled once these MMAs have read it
        tc_commit(&sh.acc_full[acc]);   // the accumulator tiles are complete
    }
}

// img_q / img_db: tile images of the query list and of the database list.  A block serves the queries
// [blockIdx.x * QH * 128, ...) of the list (nq in all) against the database tiles of its segments
// (segs + blockIdx.x * seg_stride, nseg[blockIdx.x * (seg_stride != 0)] of them; seg_stride = 0: one list shared by
// all blocks), taking every tile_stride-th tile.  Candidate ids are database list positions; positions from
// nd_pos on are padding and never kept.
// cand: [nq][cap] candidate buffers (key bits, list position), two segments of cap/2 entries per query; threshold tau[query];
// counts[2*query + buffer] receives the number of entries appended to each (bit 30 set if it overflowed).
// RANKED: no candidate buffers at all; every query thread keeps its 16 smallest keys in
// registers and rank_out[query] receives the one of rank `rank` (0-based, < 16) when the scan ends: the first
// threshold level, a scan of a few thousand sample points.
// SHARED: the tiles of a block of queries are dealt to gridDim.y blocks, which append to the same buffers (take_slots).
// sparse: survivors are rare (see the dispatch).
template <int QH, bool RANKED, bool SHARED>
__global__ void __launch_bounds__(tc_threads(QH), 1)
knn_tc_filter_kernel(const float *__restrict__ img_q, const float *__restrict__ img_db, int Dp, long long nq, long long nd_pos,
                     const int2 *__restrict__ segs, const int *__restrict__ nseg, int seg_stride, int tile_stride, int win_lo,
                     int win_hi, const float *__restrict__ tau, int cap, uint2 *cand, int *counts,
                     int *error_flag, int bf16, int sw, int nks, int n_rest, ScanParts parts, int sparse, int rank = 0, float *__restrict__ rank_out = nullptr)
{
    // bf16: the images hold bf16 pairs; sw != 0: in swizzled rows of sw bytes (else core matrices without swizzle);
    // nks: K steps of 32 operand bytes per row to multiply threefold, n_rest: once (packed remainder)
    constexpr int kProducerWarp = 8 * QH, kMmaWarp = 8 * QH + 1;
    constexpr uint32_t kTmemCols = kAccBufs * QH * TN;
    extern __shared__ __align__(1024) unsigned char smem[];   // swizzled images want their 8-row groups on 8 * sw bytes
    __shared__ __align__(8) TcShared sh;
    const uint32_t image_bytes = (uint32_t)Dp * (bf16 ? 512u : 1024u);        // hi + lo
    float *sA = reinterpret_cast<float *>(smem);                          // [QH] images
    float *sB = reinterpret_cast<float *>(smem + QH * image_bytes);       // [kBStages] images
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long qt = (long long)blockIdx.x * QH;   // first query tile of the block
    const int2 *my_segs = segs + (size_t)blockIdx.x * seg_stride;
    const int my_nseg = nseg[seg_stride ? blockIdx.x : 0];
    const int part = SHARED ? blockIdx.y : 0;
    {   // nothing of this block's segments in the window: leave before any barrier or TMEM is set up
        TileWalk<SHARED> probe(my_segs, my_nseg, tile_stride, win_lo, win_hi, part, parts);
        int first;
        if (!probe.next(first)) return;
    }
    volatile int *abort_flag = &sh.abort_flag;

    if (threadIdx.x == 0) {
        mbar_init(&sh.full_a, 1);
        for (int s = 0; s < kBStages; s++) { mbar_init(&sh.full_b[s], 1); mbar_init(&sh.empty_b[s], 1); }
        for (int b = 0; b < kAccBufs; b++) { mbar_init(&sh.acc_full[b], 1); mbar_init(&sh.acc_empty[b], (RANKED ? 4 : 8) * QH); }
        sh.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = sh.tmem_base;

    if (warp == kProducerWarp) {
        // ---------------- producer: one bulk copy per tile image ----------------
        if (lane == 0) {
            // the images of the block's QH query tiles are adjacent (the image array is padded to a
            // multiple of QH tiles)
            mbar_expect_tx(&sh.full_a, QH * image_bytes);
            for (int h = 0; h < QH; h++)
                bulk_load(sA + (size_t)h * (image_bytes / 4), img_q + (size_t)(qt + h) * (image_bytes / 4), image_bytes, &sh.full_a);
            TileWalk<SHARED> walk(my_segs, my_nseg, tile_stride, win_lo, win_hi, part, parts);
            int tile;
            for (long long t = 0; walk.next(tile); t++) {
                const int s = (int)(t % kBStages);
                const uint32_t ph = (uint32_t)((t / kBStages) & 1);
                if (!mbar_wait(&sh.empty_b[s], ph ^ 1u, abort_flag)) break;
                mbar_expect_tx(&sh.full_b[s], image_bytes);
                bulk_load(sB + (size_t)s * (image_bytes / 4), img_db + (size_t)tile * (image_bytes / 4), image_bytes, &sh.full_b[s]);
            }
        }
    } else if (warp == kMmaWarp) {
        // ---------------- MMA issuer ----------------
        // One thread issues every MMA, and a thread runs its dependent instructions several cycles apart: what it
        // computes per MMA shows in the kernel's time (descriptors built inside the K loop: 170 cycles per MMA
        // measured, with additions only 125).  tc_issue_walk is instantiated per number of K steps, so that the
        // MMAs of a tile are unrolled, independent instruction sequences.
        if (lane == 0 && mbar_wait(&sh.full_a, 0, abort_flag)) {
            // offset of K step ks inside a part, in 16-byte units: 4 KB blocks without swizzle; with it, sw / 32
            // steps side by side in a row (2 units apart) and blocks of 128 rows
            const uint32_t spr_log = sw == 128 ? 2u : (sw == 64 ? 1u : 0u);
            const uint32_t block16 = sw ? (128u * (uint32_t)sw) >> 4 : 256u, in_row16 = sw ? 2u : 0u;
            const uint32_t span16 = sw ? (127u * (uint32_t)sw + 32u) >> 4 : 256u;
            const uint64_t no_addr = sw ? make_desc_swizzled(0u, (uint32_t)sw) : make_desc(0u);
            const uint32_t a16 = smem_u32(sA) >> 4, b16 = smem_u32(sB) >> 4, image16 = image_bytes >> 4;
            const uint32_t end16 = (smem_u32(smem) + (uint32_t)(QH + kBStages) * image_bytes) >> 4;
            const TileWalk<SHARED> walk(my_segs, my_nseg, tile_stride, win_lo, win_hi, part, parts);
#define B200_ISSUE(BF16_, F_, S_)                                                                                               \
    case (F_) * 4 + (S_):                                                                                                       \
        tc_issue_walk<QH, BF16_, F_, S_, SHARED>(&sh, abort_flag, walk, tmem_base, no_addr, a16, b16, image16, spr_log, block16, \
                                                 in_row16, span16, end16);                                                      \
        break;
            if (bf16) {
                switch (nks * 4 + n_rest) {
                    B200_ISSUE(true, 0, 1) B200_ISSUE(true, 0, 2) B200_ISSUE(true, 0, 3)
                    B200_ISSUE(true, 1, 1) B200_ISSUE(true, 1, 2) B200_ISSUE(true, 1, 3)
                    B200_ISSUE(true, 2, 1) B200_ISSUE(true, 2, 2) B200_ISSUE(true, 2, 3)
                    B200_ISSUE(true, 3, 1) B200_ISSUE(true, 3, 2) B200_ISSUE(true, 3, 3)
                    default: sh.abort_flag = 1; break;   // more K steps than a narrow image holds
                }
            } else {
                switch (nks * 4 + n_rest) {
                    B200_ISSUE(false, 1, 0) B200_ISSUE(false, 2, 0) B200_ISSUE(false, 3, 0) B200_ISSUE(false, 4, 0)
                    B200_ISSUE(false, 5, 0) B200_ISSUE(false, 6, 0) B200_ISSUE(false, 7, 0) B200_ISSUE(false, 8, 0)
                    default: sh.abort_flag = 1; break;
                }
            }
#undef B200_ISSUE
        }
    } else {
        // ---------------- epilogue: one query per thread ----------------
        // 2 * QH groups of four warps; a warp reaches the TMEM lane quarter (warp % 4).  Group g belongs to
        // query tile g % QH of the block.  With a fixed threshold every group works on every database tile: it
        // takes the 64 accumulator columns buf * 64 ... (buf = g / QH) and appends to segment buf of the query's
        // candidate buffer, so the groups share nothing.  (A warp walks its keys as one dependent chain, about
        // 800 cycles per 32 keys: with all sixteen warps on a tile its epilogue takes half as long as with the
        // groups taking whole tiles in turn, and the accumulator goes back to the MMAs that much earlier.)  In the
        // ranked scan (per-query state that cannot be shared) only the groups with buf = 0 work, on
        // all columns of every tile.
        const int group = warp >> 2, quarter = warp & 3;
        const int buf = group / QH, half = group % QH;
        const bool active = !RANKED || buf == 0;
        const int seg_cap = cap / kAccBufs;
        const int row = quarter * 32 + lane;                    // TMEM lane
        const long long gq = (qt + half) * TM + row;
        const bool serve = gq < nq && active;
        uint2 *const segment = cand + (serve ? gq : 0) * cap + buf * seg_cap;
        uint2 *next = segment;   // where the next candidate goes
        float thr = serve ? (RANKED ? INFINITY : tau[gq]) : -INFINITY;
        // a fixed-threshold scan may be split into several launches (windows of the database): a launch
        // continues the buffers where the previous one stopped (counts are zeroed before the first)
        bool overflow = false;
        if (!RANKED && serve) {
            const int c0 = counts[gq * kAccBufs + buf];
            next += c0 & 0x3fffffff;
            overflow = (c0 & 0x40000000) != 0;
            if (overflow) thr = -INFINITY;
        }
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * TN);

        // One chunk = 32 accumulator columns = 32 keys of this thread's query.  Fast path: a tree of
        // independent three-input min operations and one comparison.  Only if the minimum beats the
        // threshold (rare once the scan is under way) are the quarters whose minimum does so compared
        // element by element; everything is indexed statically, so the keys never leave the registers.
        // What a survivor costs decides the scan: nearly every chunk of a warp has one.  Comparison, one 8-byte store, one
        // addition to the pointer; with key and id in two arrays, an index and a test for padding the scans took 80.3
        // instead of 63.2 ms (10^6 x 50), 7.16 instead of 4.34 (300 000 x 20), 0.48 instead of 0.31 (30 011 x 32).
        float top[RANKED ? 16 : 1];
#pragma unroll
        for (int i = 0; i < (RANKED ? 16 : 1); i++) top[i] = INFINITY;
        auto process_chunk = [&](const uint32_t (&r)[32], long long col0, bool tile_inside) {
            float m4[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float a = min3(__uint_as_float(r[8 * q]), __uint_as_float(r[8 * q + 1]), __uint_as_float(r[8 * q + 2]));
                const float b = min3(__uint_as_float(r[8 * q + 3]), __uint_as_float(r[8 * q + 4]), __uint_as_float(r[8 * q + 5]));
                const float c = fminf(__uint_as_float(r[8 * q + 6]), __uint_as_float(r[8 * q + 7]));
                m4[q] = min3(a, b, c);
            }
            const float mn = fminf(min3(m4[0], m4[1], m4[2]), m4[3]);
            if (mn < thr) {
                if constexpr (SHARED) {
                    int n = 0, room = 0;
#pragma unroll
                    for (int c = 0; c < 32; c++) n += __uint_as_float(r[c]) < thr ? 1 : 0;
                    next = segment + take_slots(counts + gq * kAccBufs + buf, n, seg_cap, room);
                    if (room < n) { overflow = true; thr = -INFINITY; }   // the row is lost: nothing more is written
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (m4[q] < thr) {
                        if constexpr (RANKED) {
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                const int c = q * 8 + e;
                                const float key = __uint_as_float(r[c]);
                                if (key < thr && (tile_inside || col0 + c < nd_pos)) {   // replaces the largest of the 16 and sinks to its place
                                    top[15] = key;
#pragma unroll
                                    for (int i = 15; i > 0; i--) {
                                        const float lo = fminf(top[i - 1], top[i]), hi = fmaxf(top[i - 1], top[i]);
                                        top[i - 1] = lo;
                                        top[i] = hi;
                                    }
                                    thr = top[15];
                                }
                            }
                        } else {   // padding rows carry a huge norm and never pass (kTauLimit)
                            unsigned which = 16u;   // 8 + index of the survivor when there is one, 16 or more when there are several
                            if (!SHARED && sparse) {
                                which = 0u;
#pragma unroll
                                for (int e = 0; e < 8; e++) which += __uint_as_float(r[q * 8 + e]) < thr ? 8u + e : 0u;
                            }
                            if (!SHARED && which < 16u) {   // its key is the minimum
                                __stcg(next, make_uint2(__float_as_uint(m4[q]), (unsigned)col0 + q * 8 - 8 + which));
                                next++;
                            } else {
#pragma unroll
                                for (int e = 0; e < 8; e++) {
                                    if (__uint_as_float(r[q * 8 + e]) < thr) {
                                        __stcg(next, make_uint2(r[q * 8 + e], (unsigned)col0 + q * 8 + e));
                                        next++;
                                    }
                                }
                            }
                        }
                    }
                }
            }
            // a chunk appends at most 32 entries: stop a buffer that could overflow in the next one
            if (!RANKED && !SHARED && next > segment + (seg_cap - 32)) { overflow = true; thr = -INFINITY; }
        };

        TileWalk<SHARED> walk(my_segs, active ? my_nseg : 0, tile_stride, win_lo, win_hi, part, parts);
        int tile;
        for (long long t = 0; walk.next(tile); t++) {
            const int b = (int)(t % kAccBufs);
            const uint32_t ph_b = (uint32_t)((t / kAccBufs) & 1);
            if (!mbar_wait(&sh.acc_full[b], ph_b, abort_flag, 32)) break;
            tc_fence_after();
            const long long p0 = (long long)tile * TN;
            const bool inside = p0 + TN <= nd_pos;
            const uint32_t tcol = lane_base + (uint32_t)(b * QH * TN);
            // one copy of the chunk code, executed once per 32 columns: small code beats overlapping the TMEM reads
            // (16 keys per read with the next read in flight while these are compared was 4 % slower)
            const int c_lo = RANKED ? 0 : buf * (TN / 2), c_hi = RANKED ? TN : c_lo + TN / 2;   // this group's columns
#pragma unroll 1
            for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
                uint32_t r[32];
                tc_ld32_issue(tcol + (uint32_t)c0, r);
                tc_ld32_wait(r);
                if (c0 == c_hi - 32) {   // the last read has landed: hand the accumulator buffer back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.acc_empty[b]);
                }
                process_chunk(r, p0 + c0, inside);
            }
        }
        if constexpr (RANKED) {
            if (serve) {
                float t = top[0];
#pragma unroll
                for (int i = 1; i < 16; i++) t = (i == rank) ? top[i] : t;
                rank_out[gq] = fminf(t, kTauLimit);
            }
        } else if constexpr (!SHARED) {
            // The final selection is a separate kernel (one warp per query, thousands in flight): it is a chain of
            // dependent global round trips, which the warps of this block would walk through one query at a time.
            if (serve) counts[gq * kAccBufs + buf] = (int)(next - segment) | (overflow ? 0x40000000 : 0);
        }
    }
    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0 && sh.abort_flag) atomicExch(error_flag, 1);
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// filter kernel for wide points (D + 1 > 64): the inner dimension no longer fits in shared memory at once
// ------------------------------------------------------------------------------------------------
// A block multiplies two query tiles with two database tiles (a "unit" of 256 database rows) at a time,
// walking the inner dimension in chunks of kWideKC: a stage holds the chunk images of the four tiles
// (4 x 16 KB), three stages alternate, the four 128 x 128 accumulators fill the 512 TMEM columns.  The query
// images are streamed again for every unit, so the kernel leans on L2 bandwidth (64 KB per 12.6 Mi products).
// bf16 images are in rows of 64 bytes with the 64-byte swizzle, and one MMA multiplies a query tile with both
// database tiles (N = 256): their parts are placed one after the other in the stage, which costs the producer
// two more copies and saves a third of what the tensor core reads from shared memory (no swizzle, N = 128, two
// stages of 96 KB: 5 to 9 % slower, 50 000 x 1 024 14.4 against 13.8 ms a scan).  After the
// last chunk of a unit the sixteen epilogue warps (query tile x database tile x TMEM lane quarter) compare
// the keys with the fixed thresholds exactly as in the narrow kernel; the next unit's MMAs wait until the
// accumulators have been read.
constexpr int kWideKC = 16;                       // words of 32 bits per row, chunk and part (32 bf16 values, 16 TF32) = 2 MMA K steps
constexpr int kWideSwizzle = 64;                  // bytes of such a row: the swizzle of the bf16 images
constexpr uint32_t kWideChunkBytes = kWideKC * 1024;   // hi + lo of one tile and chunk
constexpr int kWideStages = 3;
constexpr int kWideUnit = 2 * TN;                 // database rows per unit

struct WideShared {
    uint64_t full[kWideStages];
    uint64_t empty[kWideStages];
    uint64_t acc_full;
    uint64_t acc_empty;
    uint32_t tmem_base;
    int abort_flag;
};

// RANKED: the first threshold level (see the narrow kernel): no buffers, the warps of the unit's first database tile
// read both tiles and keep the 16 smallest keys of their queries in registers; positions from n_pos on are padding.
template <bool RANKED>
__global__ void __launch_bounds__(tc_threads(2), 1)
knn_tc_wide_kernel(const float *__restrict__ img_q, const float *__restrict__ img_db, int n_chunks, long long nq,
                   const int2 *__restrict__ segs, const int *__restrict__ nseg, int seg_stride, int unit_stride, int win_lo,
                   int win_hi, const float *__restrict__ tau, int cap, uint2 *cand, int *counts,
                   int *error_flag, int bf16, ScanParts parts, int rank = 0, float *__restrict__ rank_out = nullptr, long long n_pos = 0)
{
    constexpr int kProducerWarp = 16, kMmaWarp = 17;
    constexpr uint32_t kTmemCols = 512;
    constexpr int kSteps = kWideKC / 8;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) WideShared sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long qt = (long long)blockIdx.x * 2;   // first query tile of the block
    const int2 *my_segs = segs + (size_t)blockIdx.x * seg_stride;
    const int my_nseg = nseg[seg_stride ? blockIdx.x : 0];
    const int part = RANKED ? 0 : blockIdx.y;
    {   // nothing of this block's segments in the window
        TileWalk<!RANKED> probe(my_segs, my_nseg, unit_stride, win_lo, win_hi, part, parts);
        int first;
        if (!probe.next(first)) return;
    }
    volatile int *abort_flag = &sh.abort_flag;
    const size_t tile_floats = (size_t)n_chunks * (kWideChunkBytes / 4);   // one tile's image, all chunks
    // stage layout: [A0 hi][A0 lo][A1 hi][A1 lo][B0 hi][B1 hi][B0 lo][B1 lo]
    constexpr uint32_t kPartBytes = kWideChunkBytes / 2;
    auto stage_ptr = [&](int s, int part) { return smem + ((size_t)s * 8 + part) * kPartBytes; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kWideStages; s++) { mbar_init(&sh.full[s], 1); mbar_init(&sh.empty[s], 1); }
        mbar_init(&sh.acc_full, 1);
        mbar_init(&sh.acc_empty, RANKED ? 8 : 16);
        sh.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = sh.tmem_base;

    if (warp == kProducerWarp) {
        if (lane == 0) {
            TileWalk<!RANKED> walk(my_segs, my_nseg, unit_stride, win_lo, win_hi, part, parts);
            int unit;
            long long it = 0;   // stage counter over (unit, chunk)
            bool ok = true;
            while (ok && walk.next(unit)) {
                for (int c = 0; c < n_chunks; c++, it++) {
                    const int s = (int)(it % kWideStages);
                    const uint32_t ph = (uint32_t)((it / kWideStages) & 1);
                    if (!mbar_wait(&sh.empty[s], ph ^ 1u, abort_flag)) { ok = false; break; }
                    mbar_expect_tx(&sh.full[s], 4 * kWideChunkBytes);
                    const size_t coff = (size_t)c * (kWideChunkBytes / 4);
                    bulk_load(stage_ptr(s, 0), img_q + (size_t)qt * tile_floats + coff, kWideChunkBytes, &sh.full[s]);
                    bulk_load(stage_ptr(s, 2), img_q + (size_t)(qt + 1) * tile_floats + coff, kWideChunkBytes, &sh.full[s]);
#pragma unroll
                    for (int g = 0; g < 2; g++) {
                        const float *b = img_db + (size_t)(2 * (long long)unit + g) * tile_floats + coff;
                        bulk_load(stage_ptr(s, 4 + g), b, kPartBytes, &sh.full[s]);
                        bulk_load(stage_ptr(s, 6 + g), b + kPartBytes / 4, kPartBytes, &sh.full[s]);
                    }
                }
            }
        }
    } else if (warp == kMmaWarp) {
        if (lane == 0) {
            TileWalk<!RANKED> walk(my_segs, my_nseg, unit_stride, win_lo, win_hi, part, parts);
            int unit;
            long long it = 0, n_unit = 0;
            bool ok = true;
            const uint64_t no_addr = bf16 ? make_desc_swizzled(0u, kWideSwizzle) : make_desc(0u);
            const uint32_t stage16 = smem_u32(smem) >> 4, part16 = kPartBytes >> 4;
            while (ok && walk.next(unit)) {
                // the accumulators of the previous unit must have been read
                if (!mbar_wait(&sh.acc_empty, (uint32_t)((n_unit & 1) ^ 1), abort_flag)) break;
                for (int c = 0; c < n_chunks; c++, it++) {
                    const int s = (int)(it % kWideStages);
                    const uint32_t ph = (uint32_t)((it / kWideStages) & 1);
                    if (!mbar_wait(&sh.full[s], ph, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    // descriptors by addition only (see the narrow kernel's issuer)
                    const uint64_t st0 = no_addr + (uint64_t)(stage16 + (uint32_t)s * 8u * part16);
                    const uint32_t acc0 = (c > 0) ? 1u : 0u;
                    if (bf16) {
#pragma unroll
                        for (int h = 0; h < 2; h++) {   // both database tiles at once; a K step is 32 bytes of a row
                            const uint64_t a_hi = st0 + (uint64_t)(2u * (uint32_t)h * part16), a_lo = a_hi + part16;
                            const uint64_t b_hi = st0 + (uint64_t)(4u * part16), b_lo = b_hi + 2u * part16;
                            const uint32_t d_tmem = tmem_base + (uint32_t)(h * 2 * TN);
#pragma unroll
                            for (int ks = 0; ks < kSteps; ks++)        // hi . hi
                                tc_mma_bf16(d_tmem, a_hi + ks * 2u, b_hi + ks * 2u, kInstrDescBf16Pair, ks ? 1u : acc0);
#pragma unroll
                            for (int ks = 0; ks < kSteps; ks++)        // lo . hi
                                tc_mma_bf16(d_tmem, a_lo + ks * 2u, b_hi + ks * 2u, kInstrDescBf16Pair, 1u);
#pragma unroll
                            for (int ks = 0; ks < kSteps; ks++)        // hi . lo
                                tc_mma_bf16(d_tmem, a_hi + ks * 2u, b_lo + ks * 2u, kInstrDescBf16Pair, 1u);
                        }
                    } else {
#pragma unroll
                        for (int pair = 0; pair < 4; pair++) {   // a K step is a block of 4 KB
                            const int h = pair >> 1, g = pair & 1;
                            const uint64_t a_hi = st0 + (uint64_t)(2u * (uint32_t)h * part16), a_lo = a_hi + part16;
                            const uint64_t b_hi = st0 + (uint64_t)((4u + (uint32_t)g) * part16), b_lo = b_hi + 2u * part16;
                            const uint32_t d_tmem = tmem_base + (uint32_t)((h * 2 + g) * TN);
#pragma unroll
                            for (int ks = 0; ks < kSteps; ks++)        // hi . hi
                                tc_mma_tf32(d_tmem, a_hi + ks * 256u, b_hi + ks * 256u, kInstrDesc, ks ? 1u : acc0);
#pragma unroll
                            for (int ks = 0; ks < kSteps; ks++)        // lo . hi
                                tc_mma_tf32(d_tmem, a_lo + ks * 256u, b_hi + ks * 256u, kInstrDesc, 1u);
#pragma unroll
                            for (int ks = 0; ks < kSteps; ks++)        // hi . lo
                                tc_mma_tf32(d_tmem, a_hi + ks * 256u, b_lo + ks * 256u, kInstrDesc, 1u);
                        }
                    }
                    tc_commit(&sh.empty[s]);
                }
                if (ok) tc_commit(&sh.acc_full);
                n_unit++;
            }
        }
    } else {
        // ---------------- epilogue: one query per thread, one database tile of the unit per warp group ----------------
        const int quarter = warp & 3, half = (warp >> 2) & 1, g = warp >> 3;
        const int seg_cap = cap / 2;
        const int row = quarter * 32 + lane;
        const long long gq = (qt + half) * TM + row;
        const bool active = !RANKED || g == 0;
        const bool serve = gq < nq && active;
        uint2 *const segment = cand + (serve ? gq : 0) * cap + g * seg_cap;
        uint2 *next = segment;
        float thr = serve ? (RANKED ? INFINITY : tau[gq]) : -INFINITY;
        bool overflow = false;
        if (!RANKED && serve) {
            const int c0 = counts[gq * 2 + g];
            next += c0 & 0x3fffffff;
            overflow = (c0 & 0x40000000) != 0;
            if (overflow) thr = -INFINITY;
        }
        TileWalk<!RANKED> walk(my_segs, active ? my_nseg : 0, unit_stride, win_lo, win_hi, part, parts);
        const bool alone = walk.parts == 1;   // as in the narrow kernel
        int unit;
        float top[RANKED ? 16 : 1];
#pragma unroll
        for (int i = 0; i < (RANKED ? 16 : 1); i++) top[i] = INFINITY;
        // 32 keys of this thread's query: positions pos0 ...
        auto process_chunk = [&](const uint32_t (&r)[32], long long pos0) {
            float m4[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float a = min3(__uint_as_float(r[8 * q]), __uint_as_float(r[8 * q + 1]), __uint_as_float(r[8 * q + 2]));
                const float b = min3(__uint_as_float(r[8 * q + 3]), __uint_as_float(r[8 * q + 4]), __uint_as_float(r[8 * q + 5]));
                const float c = fminf(__uint_as_float(r[8 * q + 6]), __uint_as_float(r[8 * q + 7]));
                m4[q] = min3(a, b, c);
            }
            const float mn = fminf(min3(m4[0], m4[1], m4[2]), m4[3]);
            if (mn < thr) {
                if (!RANKED && !alone) {
                    int n = 0, room = 0;
#pragma unroll
                    for (int c = 0; c < 32; c++) n += __uint_as_float(r[c]) < thr ? 1 : 0;
                    next = segment + take_slots(counts + gq * 2 + g, n, seg_cap, room);
                    if (room < n) { overflow = true; thr = -INFINITY; }   // the row is lost: nothing more is written
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (m4[q] < thr) {
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            const int c = q * 8 + e;
                            const float key = __uint_as_float(r[c]);
                            if constexpr (RANKED) {
                                if (key < thr && pos0 + c < n_pos) {   // replaces the largest of the 16 and sinks to its place
                                    top[15] = key;
#pragma unroll
                                    for (int i = 15; i > 0; i--) {
                                        const float lo = fminf(top[i - 1], top[i]), hi = fmaxf(top[i - 1], top[i]);
                                        top[i - 1] = lo;
                                        top[i] = hi;
                                    }
                                    thr = top[15];
                                }
                            } else if (key < thr) {   // padding rows carry a huge norm and never pass (kTauLimit)
                                __stcg(next, make_uint2(r[c], (unsigned)pos0 + c));
                                next++;
                            }
                        }
                    }
                }
            }
            if (!RANKED && alone && next > segment + (seg_cap - 32)) { overflow = true; thr = -INFINITY; }
        };
        const uint32_t tlane = tmem_base + ((uint32_t)(quarter * 32) << 16);
        for (long long n_unit = 0; walk.next(unit); n_unit++) {
            if (!mbar_wait(&sh.acc_full, (uint32_t)(n_unit & 1), abort_flag, 32)) break;
            tc_fence_after();
            // this warp's database tiles of the unit: its own, or both when ranked
#pragma unroll 1
            for (int gg = RANKED ? 0 : g; gg <= (RANKED ? 1 : g); gg++) {
                const uint32_t tcol = tlane + (uint32_t)((half * 2 + gg) * TN);
                const long long p0 = (long long)unit * kWideUnit + (long long)gg * TN;
#pragma unroll 1
                for (int c0 = 0; c0 < TN; c0 += 32) {
                    uint32_t r[32];
                    tc_ld32_issue(tcol + (uint32_t)c0, r);
                    tc_ld32_wait(r);
                    if (c0 == TN - 32 && gg == (RANKED ? 1 : g)) {   // the last read has landed: hand the accumulators back
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh.acc_empty);
                    }
                    process_chunk(r, p0 + c0);
                }
            }
        }
        if constexpr (RANKED) {
            if (serve) {
                float t = top[0];
#pragma unroll
                for (int i = 1; i < 16; i++) t = (i == rank) ? top[i] : t;
                rank_out[gq] = fminf(t, kTauLimit);
            }
        } else {
            if (serve && alone) counts[gq * 2 + g] = (int)(next - segment) | (overflow ? 0x40000000 : 0);
        }
    }
    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0 && sh.abort_flag) atomicExch(error_flag, 1);
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// selection after a scan: one warp per query
// ------------------------------------------------------------------------------------------------
// Buffer of query q: two segments of cap/2 entries with counts[2q], counts[2q+1] valid entries (bit 30 of a
// count: the segment overflowed, i.e. keys below tau were lost).  The warp holds the keys in registers as
// order-preserving integers (SLOTS a lane, the two segments one after the other) and finds the k-th smallest by bisection on
// the bits between the smallest and the largest key of the buffer: they share their leading bits, so about half of 32
// steps are enough, 1,500 issue slots (a warp-wide bitonic sort: 17,000).
struct CandidateBuffer {
    const uint2 *entry;   // (key bits, list position)
    int n0, n, half;
    bool lost;
    __device__ CandidateBuffer(const uint2 *cand, int cap, const int *counts, long long q) : entry(cand + q * cap), half(cap / 2)
    {
        const int c0 = counts[2 * q], c1 = counts[2 * q + 1];
        lost = ((c0 | c1) & 0x40000000) != 0;
        n0 = c0 & 0x3fffffff;
        n = n0 + (c1 & 0x3fffffff);
    }
    __device__ int at(int e) const { return e < n0 ? e : half + (e - n0); }
};
template <int SLOTS> __device__ __forceinline__ void load_keys(const CandidateBuffer &b, int lane, unsigned (&enc)[SLOTS], unsigned &lo, unsigned &hi)
{
    lo = 0xffffffffu;
    hi = 0u;
#pragma unroll
    for (int j = 0; j < SLOTS; j++) {
        const int e = lane + 32 * j;
        enc[j] = 0xffffffffu;
        if (e < b.n) {
            enc[j] = enc_float(__uint_as_float(__ldcg(&b.entry[b.at(e)].x)));
            lo = min(lo, enc[j]);
            hi = max(hi, enc[j]);
        }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
}
// the smallest value with at least k keys at or below it; 0 < k <= n
template <int SLOTS> __device__ __forceinline__ unsigned kth_key(const unsigned (&enc)[SLOTS], int n, int k, unsigned lo, unsigned hi)
{
    const int jmax = (n + 31) / 32;
#pragma unroll 1
    while (lo < hi) {
        const unsigned mid = lo + ((hi - lo) >> 1);
        int c = 0;
#pragma unroll
        for (int j = 0; j < SLOTS; j += 4) {
            if (j >= jmax) break;
            c += (enc[j] <= mid) + (enc[j + 1] <= mid) + (enc[j + 2] <= mid) + (enc[j + 3] <= mid);   // (empty slots hold the maximum)
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (c >= k) hi = mid;
        else lo = mid + 1;
        if (c == k) {   // exactly those: the largest of them
            unsigned v = 0u;
#pragma unroll
            for (int j = 0; j < SLOTS; j++)
                if (enc[j] <= hi) v = max(v, enc[j]);
            return __reduce_max_sync(0xffffffffu, v);
        }
    }
    return lo;
}

// kth[q] = the k-th smallest key of the buffer, or -inf when it lost keys or holds fewer than k
template <int SLOTS>
__global__ void __launch_bounds__(128)
knn_tc_pick_kernel(const uint2 *__restrict__ cand, int cap, const int *__restrict__ counts, long long nq, int k, float *__restrict__ kth)
{
    const int lane = threadIdx.x & 31;
    const long long q = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (q >= nq) return;
    const CandidateBuffer b(cand, cap, counts, q);
    float v = -INFINITY;
    if (!b.lost && b.n >= k) {
        unsigned enc[SLOTS], lo, hi;
        load_keys(b, lane, enc, lo, hi);
        v = dec_float(kth_key(enc, b.n, k, lo, hi));
    }
    if (lane == 0) kth[q] = v;
}

// Xp[pos] = X[list[pos]] (zeros for padding): the database rows in visiting order (the bf16 images' kernel writes them
// on the way).
__global__ void knn_gather_rows_kernel(const float *__restrict__ X, const int *__restrict__ list, int D, long long n_pos,
                                       float *__restrict__ Xp)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_pos * D) return;
    const long long pos = t / D;
    const int i = list[pos];
    Xp[t] = (i >= 0) ? X[(long long)i * D + (t - pos * D)] : 0.0f;
}

// ------------------------------------------------------------------------------------------------
// exact re-rank + proof
// ------------------------------------------------------------------------------------------------
// The canonical distance: differences, squares and the running sum rounded one by one, in the order of the dimensions.
__device__ __forceinline__ float canon_step(float acc, float x, float y)
{
    const float t = __fsub_rn(x, y);
    return __fadd_rn(acc, __fmul_rn(t, t));
}

// The rounded squares of two rounded differences: x - y as x + (-1) y, the square as a fused operation with -0 (kMinusZero2:
// common.cuh), each half as the single instruction rounds it.
__device__ __forceinline__ float2 canon_squares(float2 x, float2 y, unsigned long long minus_zero)
{
    float2 q;   // (the moves are part of it: with pack() and unpack() the compiler spills more)
    asm("{\n\t.reg .b64 a, b, m;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 m, 0xbf800000bf800000;\n\t"
        "fma.rn.f32x2 a, b, m, a;\n\tfma.rn.f32x2 a, a, a, %6;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "=f"(q.x), "=f"(q.y)
        : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "l"(minus_zero));
    return q;
}

constexpr int kRerankWarps = 4;
constexpr int kMaxL = 256;
constexpr int kRerankDims = 32;   // dimensions per stage of wide rows
constexpr int kRerankWhole = 64;  // rows of up to this many dimensions are staged whole

// Staged rows are `stride` floats apart: a multiple of 4, but not of 8, so that 32 lanes read 16 bytes of a row of their own
// without bank conflicts.
__host__ __device__ constexpr int rerank_stride(int D) { const int d = D <= kRerankWhole ? (D + 3) / 4 * 4 : kRerankDims; return d % 8 == 0 ? d + 4 : d; }
// Stages of a row that is walked: one hides its latency behind the other warps that its smaller share of shared memory makes room
// for (16 -> 24 on an SM), two where the registers of 256 candidates allow 16 anyway (scan and selection apart, ms, two | one:
// 100,003 x 96, K = 32 0.95 | 0.77, 60,000 x 784, K = 90 2.55 | 2.47, 50,000 x 1,024, K = 150 3.74 | 4.10).
__host__ __device__ constexpr int rerank_stages(int D, int L) { return D <= kRerankWhole || L <= 128 ? 1 : 2; }
// one warp: the stages of 32 candidate rows and the query; L evaluated candidates; 34 row addresses
__host__ __device__ constexpr size_t rerank_floats(int D, int L) { return (size_t)rerank_stages(D, L) * 33 * rerank_stride(D) + 4 * (size_t)L + 68; }

__host__ __device__ constexpr size_t rerank_floats_max(int L) { return rerank_floats(kRerankWhole, L) > rerank_floats(kRerankWhole + 1, L) ? rerank_floats(kRerankWhole, L) : rerank_floats(kRerankWhole + 1, L); }

template <int BYTES> __device__ __forceinline__ void async_copy(void *dst, const void *src)
{
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}

// Warp-wide bitonic sort of 32 EPL keys, ascending; element lane * EPL + r in k[r].
template <int EPL> __device__ __forceinline__ void warp_sort(unsigned long long (&k)[EPL], int lane)
{
#pragma unroll
    for (int size = 2; size <= 32 * EPL; size <<= 1) {
#pragma unroll
        for (int j = size >> 1; j > 0; j >>= 1) {
            if (j >= EPL) {
                const bool lower = ((lane * EPL) & j) == 0, up = ((lane * EPL) & size) == 0;   // alike for all registers: j, size >= EPL
#pragma unroll
                for (int r = 0; r < EPL; r++) {
                    const unsigned long long o = __shfl_xor_sync(0xffffffffu, k[r], j / EPL);
                    if ((o < k[r]) == (lower == up)) k[r] = o;
                }
            } else {
#pragma unroll
                for (int r = 0; r < EPL; r++) {
                    if (r & j) continue;
                    const bool up = ((lane * EPL + r) & size) == 0;
                    const unsigned long long a = k[r], c = k[r + j];
                    const bool swap = (c < a) == up;
                    k[r] = swap ? c : a;
                    k[r + j] = swap ? a : c;
                }
            }
        }
    }
}

// One warp per query of the list (query row qlist[q]; candidate ids are positions in dblist).  Row
// (qlist[q] - out_base) of ids/d2 ([.][K]) receives the K best candidates by (canonical distance, row id);
// failed[q] = 1 when the proof does not close for the query (its output is then unspecified).
//
// Bound: the candidates' rows out of L2 (K rows per query cannot be left out: 17 GB for 60,000 queries of 784
// dimensions, K = 90).  So of the buffer's ~3 L candidates only those are read that can be among the K best: one whose key
// is more than twice the filter's error above the K-th smallest key cannot (95 at K = 90, 40 at K = 32); where the error
// is so large that more than L remain, the L smallest.  32 rows at a time are staged with asynchronous copies, VEC floats
// each, whole or 32 dimensions wide in two stages: whole lines per request, where a lane that walks a row of its own
// touches 32 lines with each.  A lane then reads its row from shared memory and sums in the canonical order.
// Measured, selection included, before (addresses computed per copy, ranking by counting) and now: 60,000 x 784 5.1 -> 2.6 ms,
// 50,000 x 1,024 7.7 -> 3.9, 10^6 x 50 15.2 -> 10.6, 100,003 x 96 (K = 32) 1.0; with squares two at a time and one stage 2.5, 3.7 (two
// stages), 10.2, 0.77.
// EPL: evaluated candidates a lane sorts (L = 32 EPL); the buffer holds up to 8 L.
template <int VEC, int EPL>
__global__ void __launch_bounds__(kRerankWarps * 32, EPL <= 4 ? 6 : 4)
knn_tc_rerank_kernel(const float *__restrict__ X, int D, const int *__restrict__ qlist, const int *__restrict__ dblist,
                     long long out_base, long long nq, const uint2 *__restrict__ cand, int cap,
                     const int *__restrict__ counts, const float *__restrict__ tau, int K, const double *__restrict__ norms_exact,
                     float err_scale, const float2 *__restrict__ res_q, const float *__restrict__ rho, int32_t *__restrict__ ids,
                     float *__restrict__ d2, int *__restrict__ failed, int *__restrict__ n_failed, float *__restrict__ max_err_ratio,
                     const float *__restrict__ Xp, unsigned long long minus_zero)
{
    // Xp (optional): the database rows in list order, Xp[pos] = X[dblist[pos]]
    constexpr int L = 32 * EPL, SLOTS = 8 * EPL;
    constexpr bool ahead = rerank_stages(kRerankWhole + 1, L) > 1;   // a row that is walked: the next stage is fetched while one is summed
    extern __shared__ __align__(16) float stage_mem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long q = (long long)blockIdx.x * kRerankWarps + w;
    if (q >= nq) return;
    const CandidateBuffer b(cand, cap, counts, q);
    if (b.lost || b.n < K) {   // the fixed threshold kept too few or too many
        if (lane == 0) { failed[q] = 1; atomicAdd(n_failed, 1); }
        return;
    }
    const long long gq = qlist[q];
    const long long orow = gq - out_base;
    const double ni = norms_exact[q];
    const int stride = rerank_stride(D);
    const bool whole = D <= kRerankWhole;
    float *stage = stage_mem + (size_t)w * rerank_floats(D, L);
    // evaluated candidates: distance bits and row id, row of `base`, filter key
    unsigned long long *s_key = reinterpret_cast<unsigned long long *>(stage + rerank_stages(D, L) * 33 * stride);
    int *s_src = reinterpret_cast<int *>(s_key + L);
    float *s_fkey = reinterpret_cast<float *>(s_src + L);
    const float **s_row = reinterpret_cast<const float **>(s_fkey + L);   // the rows of a group, then the query
    const float *base = Xp ? Xp : X;
    const float T = tau[q];   // every database point with a key below this is in the buffer
    // Error bound of the filter's key for this row: it scales with |x_i||x_j|, and a point whose key is
    // near T lies within sqrt(|x_i|^2 + T) of x_i, so |x_i||x_j| <= |x_i|^2 + (|x_i|^2 + T)+ up to a factor 2.
    double E = (double)err_scale * (ni + fmax(0.0, ni + (double)T) + 1.0);
    double dropped = 0.0;
    if (res_q) {
        // bf16 pairs: what the three products drop, bounded from the leftovers of this query and the largest
        // relative leftovers of the database, for every point with |x_j| <= |x_i| + sqrt(|x_i|^2 + T) (a point
        // further out cannot come closer than the threshold whatever the error of its key); the last term is
        // the fp32 rounding of the norm column.  err_scale then covers the accumulation only.
        const double xi = sqrt(ni), xj = xi + sqrt(fmax(0.0, ni + (double)T));
        const float2 rq = res_q[q];
        dropped = 1.001 * 2.0 * xj * ((double)rq.x * (double)rho[0] + xi * (double)rho[1] + (double)rq.y) + 1.2e-7 * xj * xj;
        E += dropped;
    }
    const double theta = (double)(D + 4) * 5.9604644775390625e-08;   // (D+4) * 2^-24
    int m = 0;
    float outside = T;   // what is not evaluated has a key of at least this
    {
        unsigned enc[SLOTS], lo, hi;
        load_keys(b, lane, enc, lo, hi);
        const double kk = (double)dec_float(kth_key(enc, b.n, K, lo, hi));
        // one with a key above key_K + 2 E (and the rounding of the canonical sums) has K others before it
        unsigned cut = enc_float(__double2float_ru(kk + 2.0 * E + 4.0 * theta * fmax(0.0, ni + kk + E) + 1e-30));
        int c = 0;
#pragma unroll
        for (int j = 0; j < SLOTS; j++) c += (lane + 32 * j < b.n && enc[j] <= cut) ? 1 : 0;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c > L) {
            cut = kth_key(enc, b.n, L, lo, hi);
            c = 0;
#pragma unroll
            for (int j = 0; j < SLOTS; j++) c += (lane + 32 * j < b.n && enc[j] <= cut) ? 1 : 0;
            c = __reduce_add_sync(0xffffffffu, c);
            if (c > L) cut--;   // ties beyond the last place stay out
        }
        const int jmax = (b.n + 31) / 32;
#pragma unroll
        for (int j = 0; j < SLOTS; j++) {
            if (j >= jmax) break;
            const int e = lane + 32 * j;
            const bool take = e < b.n && enc[j] <= cut;
            if (e < b.n && !take) outside = fminf(outside, dec_float(enc[j]));
            const unsigned mask = __ballot_sync(0xffffffffu, take);
            if (take) {
                const int at = m + __popc(mask & ((1u << lane) - 1u));
                const int p = (int)__ldcg(&b.entry[b.at(e)].y);
                s_src[at] = Xp ? p : dblist[p];
                s_fkey[at] = dec_float(enc[j]);
            }
            m += __popc(mask);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) outside = fminf(outside, __shfl_xor_sync(0xffffffffu, outside, o));
    __syncwarp();
    float worst = 0.0f;   // largest observed |filter distance - canonical distance|
    const float *xq = X + gq * D;
    const int width = whole ? D : kRerankDims, chunks = whole ? 1 : (D + kRerankDims - 1) / kRerankDims;
    // lanes per row of a copy: the power of two that covers the width, at most the warp
    const int lanes_log = width <= 8 * VEC ? 3 : (width <= 16 * VEC ? 4 : 5);
    const int col = (lane & ((1 << lanes_log) - 1)) * VEC, sub = lane >> lanes_log, rows_per_copy = 32 >> lanes_log;
    const float *mine = stage + lane * stride, *query = stage + 32 * stride;
    if (lane == 0) s_row[32] = xq;
    for (int g = 0; g < m; g += 32) {
        const int rows = min(32, m - g);
        // lanes without a candidate point at the query: their copies and sums are done and not used
        s_row[lane] = lane < rows ? base + (size_t)s_src[g + lane] * D : xq;
        __syncwarp();
        auto fetch = [&](int c) {
            float *to = stage + (size_t)(ahead ? c & 1 : 0) * 33 * stride + sub * stride + col;
            const int d = c * width + col;
            if (col < width && d < D) {
#pragma unroll 4
                for (int r = sub; r < 32; r += rows_per_copy, to += rows_per_copy * stride) async_copy<4 * VEC>(to, s_row[r] + d);
                if (sub == 0) async_copy<4 * VEC>(to, s_row[32] + d);
                if (VEC == 1 && width > 32 && d + 32 < D) {   // an odd row of up to 64 dimensions: its second half
                    for (int r = 0; r < 33; r++) async_copy<4>(stage + r * stride + col + 32, s_row[r] + d + 32);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float acc = 0.0f;
        if (ahead) fetch(0);
        for (int c = 0; c < chunks; c++) {
            if (!ahead) fetch(c);
            if (ahead && c + 1 < chunks) {
                fetch(c + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncwarp();
            const float *x = query + (size_t)(ahead ? c & 1 : 0) * 33 * stride, *y = mine + (size_t)(ahead ? c & 1 : 0) * 33 * stride;
            auto four = [&](int d) {
                const float4 u = *reinterpret_cast<const float4 *>(x + d), v = *reinterpret_cast<const float4 *>(y + d);
                const float2 a = canon_squares(make_float2(u.x, u.y), make_float2(v.x, v.y), minus_zero);
                const float2 b = canon_squares(make_float2(u.z, u.w), make_float2(v.z, v.w), minus_zero);
                acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, a.x), a.y), b.x), b.y);
            };
            const int len = min(width, D - c * width);
            if (len == kRerankDims) {
#pragma unroll
                for (int d = 0; d < kRerankDims; d += 4) four(d);
            } else {
                int d = 0;
#pragma unroll 4
                for (; d + 4 <= len; d += 4) four(d);
                for (; d < len; d++) acc = canon_step(acc, x[d], y[d]);
            }
            __syncwarp();
        }
        if (lane < rows) {
            const double approx = ni + (double)s_fkey[g + lane];
            worst = fmaxf(worst, (float)fabs(approx - (double)acc));
            const int src = s_src[g + lane];
            s_key[g + lane] = (unsigned long long)__float_as_uint(acc) << 32 | (unsigned)(Xp ? dblist[src] : src);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    __syncwarp();
    // in order of (distance, id)
    unsigned long long key[EPL];
#pragma unroll
    for (int r = 0; r < EPL; r++) key[r] = lane * EPL + r < m ? s_key[lane * EPL + r] : ~0ull;
    warp_sort<EPL>(key, lane);
    float dK = INFINITY;
#pragma unroll
    for (int r = 0; r < EPL; r++) {
        const int e = lane * EPL + r;
        const float de = __uint_as_float((unsigned)(key[r] >> 32));
        if (e < K) {
            ids[orow * K + e] = (int32_t)(unsigned)key[r];
            d2[orow * K + e] = de;
        }
        if (e == K - 1) dK = de;
    }
    dK = __shfl_sync(0xffffffffu, dK, (K - 1) / EPL);
    if (lane == 0) {
        // outsiders: key >= outside  =>  canonical distance >= (ni + outside - E) * (1 - theta)
        const double bound = (ni + (double)outside - E) * (1.0 - theta);
        bool ok = (double)dK < bound;
        const float ratio = (float)(fmax(0.0, (double)worst - dropped) / (E - dropped));
        if (!(ratio <= 0.5f)) ok = false;   // the filter was less accurate than the bound assumes
        failed[q] = ok ? 0 : 1;
        if (!ok) atomicAdd(n_failed, 1);
        atomicMax(reinterpret_cast<int *>(max_err_ratio), __float_as_int(ratio));   // ratio >= 0: int order == float order
    }
}

// First threshold level on the CUDA cores: tau[q] = the key of rank `rank` (0-based, < 16) among m sample
// points X[s_lo + k * s_stride + jitter_k], k = 0..m-1, for each of the nq queries of the list.  Keys are
// plain fp32 FMA sums: this threshold only has to be roughly right (it sizes the candidate set of the
// next level).  One query per thread, held in registers; sample points staged 32 at a time in shared
// memory and read as broadcast float4.
// The sample of the first threshold level as a list of rows: position k < m holds the jittered systematic sample
// point s_lo + k * s_stride + jitter_k (a plain stride would alias with any periodic ordering of the data), the
// positions from m on are padding.
__global__ void knn_sample_list_kernel(int *__restrict__ list, long long n_pos, int m, long long s_lo, long long s_stride)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_pos) return;
    list[k] = (k < m) ? (int)(s_lo + k * s_stride + (long long)(((unsigned long long)k * 2654435761ull) % (unsigned long long)s_stride)) : -1;
}

constexpr int kTauThreads = 128;
__global__ void __launch_bounds__(kTauThreads)
knn_sample_tau_kernel(const float *__restrict__ X, int D, const int *__restrict__ qlist, long long nq, long long s_lo, long long s_stride,
                      int m, int rank, float *__restrict__ tau)
{
    __shared__ __align__(16) float s_pt[32][64];
    __shared__ float s_nrm[32];
    const long long q = (long long)blockIdx.x * kTauThreads + threadIdx.x;
    const long long qrow = (q < nq) ? qlist[q] : 0;
    float4 qv[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int d = 4 * i + e;
            v[e] = (q < nq && d < D) ? X[qrow * D + d] : 0.0f;
        }
        qv[i] = make_float4(v[0], v[1], v[2], v[3]);
    }
    float top[16];
#pragma unroll
    for (int i = 0; i < 16; i++) top[i] = INFINITY;
    for (int k0 = 0; k0 < m; k0 += 32) {
        __syncthreads();
        for (int idx = threadIdx.x; idx < 32 * 64; idx += kTauThreads) {
            const int p = idx >> 6, d = idx & 63;
            // jittered systematic sample: a plain stride would alias with any periodic ordering of the data
            const long long k = k0 + p;
            const long long j = s_lo + k * s_stride + (long long)(((unsigned long long)k * 2654435761ull) % (unsigned long long)s_stride);
            s_pt[p][d] = (k < m && d < D) ? X[j * D + d] : 0.0f;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            float n2 = 0.0f;
            for (int d = 0; d < 64; d++) n2 += s_pt[threadIdx.x][d] * s_pt[threadIdx.x][d];
            s_nrm[threadIdx.x] = (k0 + threadIdx.x < m) ? n2 : INFINITY;
        }
        __syncthreads();
        for (int p = 0; p < 32; p++) {
            const float4 *sp = reinterpret_cast<const float4 *>(s_pt[p]);
            float dot = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float4 a = sp[i];
                dot += qv[i].x * a.x + qv[i].y * a.y + qv[i].z * a.z + qv[i].w * a.w;
            }
            const float key = fmaf(-2.0f, dot, s_nrm[p]);
            if (key < top[15]) {
                top[15] = key;
#pragma unroll
                for (int i = 15; i > 0; i--) {
                    const float lo = fminf(top[i - 1], top[i]), hi = fmaxf(top[i - 1], top[i]);
                    top[i - 1] = lo;
                    top[i] = hi;
                }
            }
        }
    }
    if (q < nq) {
        float t = top[0];
#pragma unroll
        for (int i = 1; i < 16; i++) t = (i == rank) ? top[i] : t;
        tau[q] = fminf(t, kTauLimit);
    }
}

// The same for points of any width: the inner dimension is walked in chunks of 64, the dot products with
// the 32 staged sample points are kept in registers across the chunks.
__global__ void __launch_bounds__(kTauThreads)
knn_sample_tau_wide_kernel(const float *__restrict__ X, int D, const int *__restrict__ qlist, long long nq, long long s_lo,
                           long long s_stride, int m, int rank, float *__restrict__ tau)
{
    __shared__ float s_pt[32][65];
    __shared__ float s_nrm[32];
    const long long q = (long long)blockIdx.x * kTauThreads + threadIdx.x;
    const long long qrow = (q < nq) ? qlist[q] : 0;
    float top[16];
#pragma unroll
    for (int i = 0; i < 16; i++) top[i] = INFINITY;
    for (int k0 = 0; k0 < m; k0 += 32) {
        float dot[32];
#pragma unroll
        for (int p = 0; p < 32; p++) dot[p] = 0.0f;
        float n2 = 0.0f;
        for (int d0 = 0; d0 < D; d0 += 64) {
            __syncthreads();
            for (int idx = threadIdx.x; idx < 32 * 64; idx += kTauThreads) {
                const int p = idx >> 6, d = idx & 63;
                const long long k = k0 + p;
                const long long j = s_lo + k * s_stride + (long long)(((unsigned long long)k * 2654435761ull) % (unsigned long long)s_stride);
                s_pt[p][d] = (k < m && d0 + d < D) ? X[j * D + d0 + d] : 0.0f;
            }
            __syncthreads();
            float qv[64];
#pragma unroll
            for (int d = 0; d < 64; d++) qv[d] = (q < nq && d0 + d < D) ? X[qrow * D + d0 + d] : 0.0f;
#pragma unroll
            for (int p = 0; p < 32; p++) {   // fully unrolled: dot[] stays in registers
                float acc = 0.0f;
#pragma unroll
                for (int d = 0; d < 64; d++) acc = fmaf(qv[d], s_pt[p][d], acc);
                dot[p] += acc;
            }
            if (threadIdx.x < 32)
                for (int d = 0; d < 64; d++) n2 = fmaf(s_pt[threadIdx.x][d], s_pt[threadIdx.x][d], n2);
        }
        __syncthreads();
        if (threadIdx.x < 32) s_nrm[threadIdx.x] = (k0 + threadIdx.x < m) ? n2 : INFINITY;
        __syncthreads();
#pragma unroll
        for (int p = 0; p < 32; p++) {
            const float key = fmaf(-2.0f, dot[p], s_nrm[p]);
            if (key < top[15]) {
                top[15] = key;
#pragma unroll
                for (int i = 15; i > 0; i--) {
                    const float lo = fminf(top[i - 1], top[i]), hi = fmaxf(top[i - 1], top[i]);
                    top[i - 1] = lo;
                    top[i] = hi;
                }
            }
        }
    }
    if (q < nq) {
        float t = top[0];
#pragma unroll
        for (int i = 1; i < 16; i++) t = (i == rank) ? top[i] : t;
        tau[q] = fminf(t, kTauLimit);
    }
}

__global__ void knn_tc_collect_failed_kernel(const int *__restrict__ failed, long long nq, const int *__restrict__ qlist, int *__restrict__ list,
                                             int *__restrict__ count)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < nq && failed[q]) list[atomicAdd(count, 1)] = qlist[q];
}


// Exercises mbar_wait's limit: a barrier that expects one arrival and never gets it.  Every thread of the
// block must come back with `false` after limit_ns and the block must exit normally.
__global__ void mbar_wait_selftest_kernel(int *abort_flag, int *gave_up, unsigned long long limit_ns)
{
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const bool ok = mbar_wait(&bar, 0, abort_flag, 128, limit_ns);
    if (!ok) atomicAdd(gave_up, 1);
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(&bar)) : "memory");
}
}  // namespace

// wide points: the inner dimension (D + 1) does not fit the narrow kernel's shared-memory images
static bool tc_wide(int D) { return D + 1 > 64; }
// Operand form of the filter: bf16 pairs (three bf16 products per key, half the tensor-core time of 3xTF32, error
// 3 * 2^-16 of sum |x_ik||2 x_jk|) unless B200TSNE_KNN_FILTER=tf32 asks for the TF32 pairs (error ~2^-20).
static bool tc_bf16()
{
    const char *e = getenv("B200TSNE_KNN_FILTER");
    return !(e && strcmp(e, "tf32") == 0);
}

// nd: database rows the search will scan
// The limit of a kernel's dynamic shared memory is one value per function and device, shared by all threads of the
// process: a call that set it to its own need could lower it between another's call here and its launch.  So every call
// sets the most that any size needs, and launches with its own.
constexpr int kFilterSmemMax = 227 * 1024 - 1024;   // beside the kernels' static 0.1 KB
template <class Kernel> static int allow_smem(Kernel kernel, size_t most)
{
    B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    return 0;
}

bool knn_tc_supported(int64_t nd, int D, int K)
{
    if (K + 32 > kMaxL || D > 8192) return false;
    return nd >= 2048;   // below this whole rows of distances are faster than the set-up of this one (knn_dense.cu)
}

// candidate buffer entries per query in a fixed-threshold pass: 8 L (two halves of 4 L for ~1.5 L expected each)
static int fixed_cap(int K) { return (K + 32 <= 128) ? 1024 : 2048; }
constexpr int kSampleStride = 16;    // the sample pass looks at every 16th database tile
constexpr int kMaxSampleTiles = 128; // first threshold level: at most 16 384 sample points

// Device workspace of launch_knn_tc, carved in this order.
struct TcWorkspace {
    bool wide, bf16;
    size_t image_bytes;        // one tile's image (hi and lo)
    int Dp;
    int sw, nks, n_rest;       // bytes of a swizzled image row (0: core matrices without swizzle), K steps of the narrow kernel
    int whole;                 // full groups of 16 dimensions of a packed image, -1: not packed
    long long tq, td;          // tiles allocated for the query list / the database list
    float *img_q, *img_db;
    double *norms_q;
    float2 *res_q;             // bf16 form: norms of the lo parts and of the leftovers of every query
    float *img_s;              // images of the sample of the first threshold level (two-pass searches)
    int *slist;
    int *qlist, *dblist;
    float *xp;   // database rows in list order (cells only)
    unsigned char *cell_q;     // queries whose distances to the centres are not kept: their cells
    float *dist_q;             // and the distances
    int2 *segs;
    int *nseg;
    uint2 *cand;
    float *tau;
    int *counts, *failed, *flist, *counters;
    size_t bytes;
};

static TcWorkspace tc_carve(void *base, int D, int K, long long nq, long long nd, bool cells_kept)
{
    TcWorkspace w;
    w.wide = tc_wide(D);
    w.bf16 = tc_bf16();
    // one extra inner column carries the norm (two in bf16); wide points are chunked along the inner dimension
    w.sw = w.n_rest = 0;
    w.whole = w.bf16 && !w.wide ? D / 16 : -1;
    if (w.bf16 && !w.wide) {
        // packed K steps of 16 columns in swizzled rows of 32, 64 or 128 bytes; more of them: blocks of 128-byte rows
        w.nks = D / 16;
        w.n_rest = (3 * (D % 16) + 3 + 15) / 16;
        const int steps = 2 * w.nks + w.n_rest;
        w.sw = steps == 1 ? 32 : (steps == 2 ? 64 : 128);
        w.Dp = (steps * 32 + w.sw - 1) / w.sw * w.sw / 4;   // half the columns
    } else if (w.bf16) {
        w.sw = kWideSwizzle;
        w.Dp = (D + 2 + 2 * kWideKC - 1) / (2 * kWideKC) * (2 * kWideKC);
        w.nks = w.Dp / 16;
    } else {
        w.Dp = w.wide ? (D + 1 + kWideKC - 1) / kWideKC * kWideKC : (D + 1 + 7) / 8 * 8;
        w.nks = w.Dp / 8;
    }
    w.image_bytes = (size_t)w.Dp * (w.bf16 ? 512 : 1024);
    w.tq = (nq + TM - 1) / TM + 1;                 // one padding tile: a block may hold two query tiles
    w.td = (nd + TN - 1) / TN + point_cells_count(nd);   // every cell may end in a partly filled tile
    if (w.wide) w.td = (w.td + 1) / 2 * 2;         // the wide kernel takes the database two tiles at a time
    char *p = static_cast<char *>(base);
    auto take = [&](size_t bytes) { char *r = p; p += (bytes + 255) / 256 * 256; return r; };
    w.img_q = reinterpret_cast<float *>(take((size_t)w.tq * w.image_bytes));
    w.img_db = reinterpret_cast<float *>(take((size_t)w.td * w.image_bytes));
    w.norms_q = reinterpret_cast<double *>(take(sizeof(double) * (size_t)w.tq * TM));
    w.res_q = reinterpret_cast<float2 *>(take(sizeof(float2) * (size_t)w.tq * TM));
    w.qlist = reinterpret_cast<int *>(take(sizeof(int) * (size_t)w.tq * TM));
    w.dblist = reinterpret_cast<int *>(take(sizeof(int) * (size_t)w.td * TN));
    w.xp = w.wide ? nullptr : reinterpret_cast<float *>(take(sizeof(float) * (size_t)w.td * TN * D));
    w.img_s = reinterpret_cast<float *>(take((size_t)kMaxSampleTiles * w.image_bytes));
    w.slist = reinterpret_cast<int *>(take(sizeof(int) * (size_t)kMaxSampleTiles * TN));
    w.cell_q = cells_kept ? nullptr : reinterpret_cast<unsigned char *>(take((size_t)nq));
    w.dist_q = cells_kept ? nullptr : reinterpret_cast<float *>(take(sizeof(float) * kMaxCells * (size_t)nq));
    w.segs = reinterpret_cast<int2 *>(take(sizeof(int2) * (size_t)w.tq * kMaxCells));
    w.nseg = reinterpret_cast<int *>(take(sizeof(int) * (size_t)w.tq));
    w.cand = reinterpret_cast<uint2 *>(take(sizeof(uint2) * (size_t)nq * fixed_cap(K)));
    w.tau = reinterpret_cast<float *>(take(sizeof(float) * (size_t)nq));
    w.counts = reinterpret_cast<int *>(take(sizeof(int) * (size_t)nq * 2));
    w.failed = reinterpret_cast<int *>(take(sizeof(int) * (size_t)nq));
    w.flist = reinterpret_cast<int *>(take(sizeof(int) * (size_t)nq));
    w.counters = reinterpret_cast<int *>(take(sizeof(int) * 16));   // [0] wait time-out flag, [1] failed rows, [2] listed rows, [3] max error ratio (float bits), [4], [5] largest relative lo part / leftover of a database row (float bits)
    w.bytes = (size_t)(p - static_cast<char *>(base));
    return w;
}

// B200TSNE_KNN_TIMERS=1: device time of the phases of one search (CUDA events on the launching stream, printed to
// stderr when the search ends; the marks synchronise nothing, the print waits for the stream).
struct PhaseTimer {
    static constexpr int kMax = 12;
    bool on = false;
    cudaStream_t st = nullptr;
    cudaEvent_t ev[kMax] = {};
    const char *name[kMax] = {};
    int n = 0;
    explicit PhaseTimer(cudaStream_t s) : st(s)
    {
        const char *e = getenv("B200TSNE_KNN_TIMERS");
        on = e && atoi(e) != 0;
    }
    void mark(const char *what)
    {
        if (!on || n >= kMax) return;
        if (cudaEventCreate(&ev[n]) != cudaSuccess) { on = false; return; }
        cudaEventRecord(ev[n], st);
        name[n++] = what;
    }
    ~PhaseTimer()
    {
        if (n > 1 && cudaEventSynchronize(ev[n - 1]) == cudaSuccess) {
            fprintf(stderr, "knn phases (ms):");
            for (int i = 1; i < n; i++) {
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, ev[i - 1], ev[i]);
                fprintf(stderr, " %s %.2f", name[i], ms);
            }
            fprintf(stderr, "\n");
        }
        for (int i = 0; i < n; i++) cudaEventDestroy(ev[i]);
    }
};

// Workspace (device, 256-byte aligned) needed by launch_knn_tc for nq queries against nd database rows.
size_t knn_tc_workspace_bytes(int D, int K, int64_t nq, int64_t nd, bool cells_kept) { return tc_carve(nullptr, D, K, nq, nd, cells_kept).bytes; }

// Into how many parts the database tiles of every block of queries are dealt, one block a part.  A block holds a whole SM,
// so `blocks` blocks of equal work take ceil(blocks / SMs) turns: 196 on 148 SMs leave a third of the chip idle, 20 seven
// eighths of it.  One part unless more save 3 %.
// The narrow kernel's epilogue is most of its time, and slots taken in memory make it a third longer (30 011 x 32: 0.47
// against 0.61 ms): its tiles are dealt only where half of the SMs would idle.
// Scans, one part and by this rule: 50 000 x 1 024 13.8 -> 10.7 ms, 60 000 x 784 2.26 -> 1.80, 20 011 x 784 2.13 -> 1.23,
// 8 000 x 512 0.76 -> 0.28, 5 000 x 50 0.21 -> 0.10.
static ScanParts scan_parts(int blocks, int tiles, int share, int limit, int sms)
{
    auto cost = [&](int parts) {   // a part's set-up is about a tenth of a share
        const long long turns = ((long long)blocks * parts + sms - 1) / sms;
        return (double)turns * ((double)((tiles + parts - 1) / parts) + 0.1 * share);
    };
    ScanParts p;
    p.idle = std::max(1, sms / blocks);
    p.share = share;
    const int most = std::min(limit, std::max(p.idle, tiles / share));
    double least = 0.97 * cost(1);
    for (int parts = 2; parts <= most; parts++)
        if (cost(parts) < least) { p.most = parts; least = cost(parts); }
    return p;
}

// X: [N][D] row-major (device).  ids/d2: [(q_hi-q_lo)][K].  n_failed_host receives the number of rows
// whose proof did not close; their global row indices are in failed_list (device, first n entries) and
// the caller recomputes them (knn_search).  Returns after the kernels are queued, except for
// the small synchronous read of the counters.
int launch_knn_tc(const float *X, int64_t N, int D, int K, int64_t q_lo, int64_t q_hi, int64_t db_lo, int64_t db_hi, const PointCells &pc,
                  int32_t *ids, float *d2, void *workspace, int **failed_list, int *n_failed_host, float *err_ratio_host,
                  cudaStream_t st)
{
    (void)N;
    const long long nq = q_hi - q_lo, nd = db_hi - db_lo;
    *n_failed_host = 0;
    if (nq <= 0) return 0;
    const bool cells_kept = pc.dist && q_lo >= pc.lo && q_hi <= pc.lo + pc.n;
    const TcWorkspace w = tc_carve(workspace, D, K, nq, nd, cells_kept);
    const int Dp = w.Dp, cells = pc.cells;
    const bool wide = w.wide;
    const int bf16 = w.bf16 ? 1 : 0;
    const int KC = wide ? (bf16 ? 2 * kWideKC : kWideKC) : Dp;   // inner dimensions per image chunk
    const int L = (K + 32 <= 128) ? 128 : 256;                   // candidates that may be evaluated per query; about 3 L pass a scan
    const int cap = fixed_cap(K);
    uint2 *cand = w.cand;
    float *tau = w.tau;
    int *counts = w.counts, *failed = w.failed, *flist = w.flist, *counters = w.counters;
    B200_CUDA(cudaMemsetAsync(counters, 0, sizeof(int) * 16, st));
    PhaseTimer phases(st);
    phases.mark("start");

    // ---- visiting order of the queries and of the database, operand images ----
    B200_CUDA(cudaMemsetAsync(w.qlist, 0xff, sizeof(int) * (size_t)w.tq * TM, st));    // -1 = padding
    B200_CUDA(cudaMemsetAsync(w.dblist, 0xff, sizeof(int) * (size_t)w.td * TN, st));
    long long nd_pos = nd;   // database list positions in use (an upper bound when the cells are padded)
    const float *q_dist = nullptr;   // the queries' distances to the centres
    if (cells > 1) {
        const unsigned gq = (unsigned)((nq + kCellThreads - 1) / kCellThreads), gd = (unsigned)((nd + kCellThreads - 1) / kCellThreads);
        const unsigned char *cell_q = nullptr;
        if (cells_kept) {
            q_dist = pc.dist + (size_t)(q_lo - pc.lo) * kMaxCells;
            cell_q = pc.cell + (q_lo - pc.lo);
        } else {   // queries that are not database rows, or one batch of very many
            q_dist = w.dist_q;
            cell_q = w.cell_q;
            B200_TRY(point_cells_assign(pc, X, D, q_lo, nq, w.dist_q, nullptr, w.cell_q, st));
        }
        knn_cells_reset_kernel<<<1, kMaxCells, 0, st>>>(pc.tab);
        knn_cells_count_kernel<<<std::min(gd, 592u), kCellThreads, 0, st>>>(pc.cell, pc.own, nd, pc.tab, 1);
        knn_cells_count_kernel<<<std::min(gq, 592u), kCellThreads, 0, st>>>(cell_q, nullptr, nq, pc.tab, 0);
        knn_cells_layout_kernel<<<1, 32, 0, st>>>(cells, pc.tab);
        knn_cells_scatter_kernel<<<gd, kCellThreads, 0, st>>>(pc.cell, db_lo, nd, cells, pc.tab, 1, w.dblist);
        knn_cells_scatter_kernel<<<gq, kCellThreads, 0, st>>>(cell_q, q_lo, nq, cells, pc.tab, 0, w.qlist);
        nd_pos = w.td * TN;
        if (!bf16 && w.xp) knn_gather_rows_kernel<<<(unsigned)((nd_pos * D + 255) / 256), 256, 0, st>>>(X, w.dblist, D, nd_pos, w.xp);
    } else {
        knn_iota_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, st>>>(w.dblist, db_lo, nd);
        knn_iota_kernel<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>(w.qlist, q_lo, nq);
    }
    float *const xp = cells > 1 ? w.xp : nullptr;
    B200_CUDA(cudaGetLastError());
    if (bf16) {
        knn_tc_prepare_bf16_kernel<<<(unsigned)w.tq, 256, 0, st>>>(X, w.qlist, D, Dp, KC, w.sw, w.whole, 0, reinterpret_cast<__nv_bfloat16 *>(w.img_q),
                                                                   w.norms_q, w.res_q, nullptr, nullptr);
        knn_tc_prepare_bf16_kernel<<<(unsigned)w.td, 256, 0, st>>>(X, w.dblist, D, Dp, KC, w.sw, w.whole, 1, reinterpret_cast<__nv_bfloat16 *>(w.img_db),
                                                                   nullptr, nullptr, counters + 4, xp);
    } else {
        knn_tc_prepare_kernel<<<(unsigned)w.tq, 128, 0, st>>>(X, w.qlist, D, Dp, KC, 0, w.img_q, w.norms_q);
        knn_tc_prepare_kernel<<<(unsigned)w.td, 128, 0, st>>>(X, w.dblist, D, Dp, KC, 1, w.img_db, nullptr);
    }
    B200_CUDA(cudaGetLastError());

    phases.mark("cells+images");
    // two query tiles per block when their images and the database stages fit in shared memory
    // (one query tile per block, two blocks per SM: 3 % faster at N = 10^6, D = 50, for twice the L2 traffic; not used)
    const int QH = ((size_t)(2 + kBStages) * w.image_bytes + 1024 <= 227 * 1024) ? 2 : 1;
    const long long q_tiles = (nq + TM - 1) / TM;
    // Segments of the blocks: all database tiles (one shared list) unless the cells prune (per block).
    const int all_tiles = wide ? (int)(w.td / 2) : (int)((cells > 1 ? nd_pos : nd + TN - 1) / TN);   // wide: pairs of tiles
    knn_single_segment_kernel<<<1, 1, 0, st>>>(w.segs, w.nseg, all_tiles);
    B200_CUDA(cudaGetLastError());
    int seg_stride = 0;
    auto prune = [&]() -> int {   // segments from the current thresholds
        if (cells <= 1) return 0;
        const int per_block = wide ? 2 : QH;
        knn_cells_segments_kernel<<<(unsigned)((q_tiles + per_block - 1) / per_block), kCellThreads, 0, st>>>(
            q_dist, q_lo, w.qlist, nq, per_block * TM, tau, w.norms_q, cells, 1e-4f + (float)(D + 2) * 5.97e-8f, wide ? 1 : 0, pc.tab, w.segs, w.nseg);
        B200_CUDA(cudaGetLastError());
        seg_stride = kMaxCells;
        return 0;
    };
    // A database image much larger than L2 is scanned in windows of tiles, one launch per window: the blocks
    // that run at the same time then read the same ~60 MB, which stays in L2.  In one launch the blocks
    // drift apart until each streams its own copy from HBM with only one 56 KB stage in flight, and the
    // scan becomes latency-bound (measured at 10^7 rows: 3.85 s per 2^20 queries against 1.3 s of MMAs).
    const long long db_image_bytes = (long long)w.td * (long long)w.image_bytes;
    int window_tiles = db_image_bytes > (512ll << 20) ? (int)((60ll << 20) / (long long)w.image_bytes) : INT_MAX;
    if (const char *e = getenv("B200TSNE_KNN_WINDOW_TILES")) window_tiles = std::max(1, atoi(e));   // for tests
    int device = 0, sm_count = 0;
    B200_CUDA(cudaGetDevice(&device));
    B200_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
    // One scan of every stride-th tile against tau.  The attribute and the launch of the instantiation that fits the images:
    auto scan = [&](int stride) -> int {
        B200_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * (size_t)nq * 2, st));
        const long long tiles = wide ? w.td / 2 : w.td;
        const long long win = (long long)(wide ? std::max(1, window_tiles / 2) : window_tiles) * stride;
        const size_t smem = wide ? (size_t)kWideStages * 4 * kWideChunkBytes : (size_t)(QH + kBStages) * w.image_bytes;
        const int blocks = (int)((q_tiles + (wide ? 2 : QH) - 1) / (wide ? 2 : QH));
        // a share is worth its block's barriers, TMEM, first loads and last epilogue (6 us) ten times over
        const ScanParts parts = scan_parts(blocks, (int)((std::min(tiles, win) + stride - 1) / stride), wide ? (63 + Dp / KC) / (Dp / KC) : 32,
                                            wide || 2 * blocks <= sm_count ? 16 : 1, sm_count);
        const dim3 grid((unsigned)blocks, (unsigned)parts.most);
        // sparse: about 3 L of nd keys pass; where eight keys with one mostly hold no second, it is stored once behind a
        // search for its place, else there is a test and a store per key.  Both forms, scan in ms (D = 20; 50 is alike):
        //   L = 128 (K <= 96): 40 000 rows 0.56 / 0.56, 65 536 0.78 / 0.87, 131 072 2.08 / 2.58, 10^6 47.7 / 59.5
        //   L = 256:           40 000 rows 0.68 / 0.60, 65 536 0.98 / 0.92, 100 000 1.72 / 1.79, 131 072 2.59 / 2.86, 10^6 58.6 / 76.4
        // so the line is at one key in 128.  As an instantiation of its own the sparse form took 61 to 62 ms at 10^6 x 50, 53 by
        // this flag: the kernel's code is large, and where it comes to lie counts.
        const int sparse = nd >= 128ll * 3 * L;
        auto narrow = parts.most > 1 ? (QH == 1 ? knn_tc_filter_kernel<1, false, true> : knn_tc_filter_kernel<2, false, true>)
                                     : (QH == 1 ? knn_tc_filter_kernel<1, false, false> : knn_tc_filter_kernel<2, false, false>);
        if (wide) B200_TRY(allow_smem(knn_tc_wide_kernel<false>, kFilterSmemMax));
        else B200_TRY(allow_smem(narrow, kFilterSmemMax));
        for (long long lo = 0; lo < tiles; lo += win) {
            const int hi = (int)std::min<long long>(tiles, lo + win);
            if (wide)
                knn_tc_wide_kernel<false><<<grid, tc_threads(2), smem, st>>>(
                    w.img_q, w.img_db, Dp / KC, nq, w.segs, w.nseg, seg_stride, stride, (int)lo, hi, tau, cap, cand, counts,
                    counters + 0, bf16, parts);
            else
                narrow<<<grid, tc_threads(QH), smem, st>>>(
                    w.img_q, w.img_db, Dp, nq, nd_pos, w.segs, w.nseg, seg_stride, stride, (int)lo, hi, tau, cap, cand, counts,
                    counters + 0, bf16, w.sw, w.nks, w.n_rest, parts, sparse, 0, nullptr);
            B200_CUDA(cudaGetLastError());
        }
        return 0;
    };
    // Up to three levels, each fixing the threshold of the next:
    //  A  a rank up to 16 of a sample of up to 16,384 points spread over the database -> tau_A;
    //  B  (large databases) every kSampleStride-th tile against a tau_A that ~300 points of it beat;
    //  C  everything against tau_A, or against the key of rank ~3L/kSampleStride in B: ~3L points beat either.
    // Before each scan the cells are tested against the thresholds it will use; a skipped cell holds no
    // point below them, so the candidate sets (and the sample statistics) are those of a full scan.
    // (the wide kernel strides over units of two tiles: the same 1/kSampleStride of the database)
    const long long n_db_tiles = (nd + TN - 1) / TN;
    const double b_points = wide ? (double)((n_db_tiles / 2 + kSampleStride - 1) / kSampleStride) * kWideUnit
                                 : (double)((n_db_tiles + kSampleStride - 1) / kSampleStride) * TN;
    // Up to ~400k points the sample of level A is large enough (16 N / 3L points, rank ~16) to fix the
    // threshold of level C directly; beyond that level B refines it.  The rank decides how far the number of points that
    // pass strays (3 L times a Beta(16, .) variate: fewer than L or more than 8 L in about one of 10^4 rows).
    const bool direct = nd <= 393216;
    const int m_a = direct ? (int)std::min<long long>(16384, std::max<long long>(32, 16 * nd / (3 * L)))
                           : (int)std::min<long long>(16384, std::max<long long>(2048, (long long)(b_points / 32)));
    const long long a_stride = std::max<long long>(1, nd / m_a);
    const double a_target = direct ? 3.0 * L * m_a / (double)nd : 300.0 * m_a / b_points;
    const int rank_a = std::min(16, std::max(4, (int)(a_target + 0.5))) - 1;
    const int rank_b = std::max(4, (3 * L + kSampleStride - 1) / kSampleStride) - 1;
    if (getenv("B200TSNE_KNN_LEVEL_A") && strcmp(getenv("B200TSNE_KNN_LEVEL_A"), "simt") == 0) {
        if (wide)
            knn_sample_tau_wide_kernel<<<(unsigned)((nq + kTauThreads - 1) / kTauThreads), kTauThreads, 0, st>>>(X, D, w.qlist, nq, db_lo,
                                                                                                         a_stride, m_a, rank_a, tau);
        else
            knn_sample_tau_kernel<<<(unsigned)((nq + kTauThreads - 1) / kTauThreads), kTauThreads, 0, st>>>(X, D, w.qlist, nq, db_lo,
                                                                                                    a_stride, m_a, rank_a, tau);
    } else {
        // the same sample on the tensor cores: its points as a few tile images, every query thread keeping its
        // 16 smallest keys in registers (the keys differ from the fp32 sums of the CUDA-core kernels by the
        // filter's error only, and this threshold has to be roughly right, no more)
        const int ts = wide ? (m_a + kWideUnit - 1) / kWideUnit * 2 : (m_a + TN - 1) / TN;
        knn_sample_list_kernel<<<(unsigned)((ts * TN + 255) / 256), 256, 0, st>>>(w.slist, (long long)ts * TN, m_a, db_lo, a_stride);
        if (bf16)
            knn_tc_prepare_bf16_kernel<<<(unsigned)ts, 256, 0, st>>>(X, w.slist, D, Dp, KC, w.sw, w.whole, 1, reinterpret_cast<__nv_bfloat16 *>(w.img_s),
                                                                     nullptr, nullptr, nullptr, nullptr);
        else
            knn_tc_prepare_kernel<<<(unsigned)ts, 128, 0, st>>>(X, w.slist, D, Dp, KC, 1, w.img_s, nullptr);
        knn_single_segment_kernel<<<1, 1, 0, st>>>(w.segs, w.nseg, wide ? ts / 2 : ts);
        B200_CUDA(cudaGetLastError());
        if (wide) {
            const size_t smem_a = (size_t)kWideStages * 4 * kWideChunkBytes;
            B200_TRY(allow_smem(knn_tc_wide_kernel<true>, kFilterSmemMax));
            knn_tc_wide_kernel<true><<<(unsigned)((q_tiles + 1) / 2), tc_threads(2), smem_a, st>>>(
                w.img_q, w.img_s, Dp / KC, nq, w.segs, w.nseg, 0, 1, 0, ts / 2, nullptr, 0, nullptr, nullptr, counters + 0, bf16,
                ScanParts(), rank_a, tau, (long long)m_a);
        } else {
            const size_t smem_a = (size_t)(1 + kBStages) * w.image_bytes;
            B200_TRY(allow_smem(knn_tc_filter_kernel<1, true, false>, kFilterSmemMax));
            knn_tc_filter_kernel<1, true, false><<<(unsigned)q_tiles, tc_threads(1), smem_a, st>>>(
                w.img_q, w.img_s, Dp, nq, (long long)m_a, w.segs, w.nseg, 0, 1, 0, ts, nullptr, 0, nullptr, nullptr, counters + 0,
                bf16, w.sw, w.nks, w.n_rest, ScanParts(), 0, rank_a, tau);
        }
        B200_CUDA(cudaGetLastError());
        knn_single_segment_kernel<<<1, 1, 0, st>>>(w.segs, w.nseg, all_tiles);   // back to all database tiles
    }
    B200_CUDA(cudaGetLastError());
    phases.mark("level_A");
    B200_TRY(prune());
    if (!direct) {
        // level B: only the key of rank rank_b among the sample's candidates is needed
        B200_TRY(scan(kSampleStride));
        const unsigned sel_grid = (unsigned)((nq + 3) / 4);
        if (cap <= 1024) knn_tc_pick_kernel<32><<<sel_grid, 128, 0, st>>>(cand, cap, counts, nq, rank_b + 1, tau);
        else knn_tc_pick_kernel<64><<<sel_grid, 128, 0, st>>>(cand, cap, counts, nq, rank_b + 1, tau);
        B200_CUDA(cudaGetLastError());
        phases.mark("level_B+pick");
        B200_TRY(prune());
    }
    B200_TRY(scan(1));   // level C
    phases.mark("level_C");
    // Error bound of the filter relative to (|x_i|^2 + d^2 + 1): 3xTF32 drops terms of order 2^-22 |x_i||x_j|,
    // and the fp32 accumulation of D products (not IEEE in the tensor core: take two units in the last place
    // per addition) adds up to 2 D 2^-24 |x_i||x_j| in the worst case.  2^-14 covers both with a wide margin
    // up to D = 256; beyond, the bound grows with D.  The re-rank checks the observed error of every
    // candidate against half of it.
    // bf16 pairs: what the products drop is bounded row by row in the re-rank (see knn_tc_prepare_bf16_kernel), so
    // the scale covers the accumulation only.
    const float err_scale = bf16 ? std::max(1.52587890625e-05f, (float)(D + 8) * 2.384185791015625e-07f)      // max(2^-16, (D + 8) 2^-22)
                                 : std::max(6.103515625e-05f, (float)(D + 8) * 2.384185791015625e-07f);   // max(2^-14, (D + 8) 2^-22)
    // rows are copied 16, 8 or 4 bytes at a time, as their length keeps them aligned
    const size_t x_at = reinterpret_cast<size_t>(X);
    const int vec = (D % 4 == 0 && x_at % 16 == 0) ? 4 : ((D % 2 == 0 && x_at % 8 == 0) ? 2 : 1);
    auto rerank = L == 128 ? (vec == 4 ? knn_tc_rerank_kernel<4, 4> : (vec == 2 ? knn_tc_rerank_kernel<2, 4> : knn_tc_rerank_kernel<1, 4>))
                           : (vec == 4 ? knn_tc_rerank_kernel<4, 8> : (vec == 2 ? knn_tc_rerank_kernel<2, 8> : knn_tc_rerank_kernel<1, 8>));
    const size_t rerank_smem = sizeof(float) * kRerankWarps * rerank_floats(D, L);
    B200_TRY(allow_smem(rerank, sizeof(float) * kRerankWarps * rerank_floats_max(L)));
    rerank<<<(unsigned)((nq + kRerankWarps - 1) / kRerankWarps), kRerankWarps * 32, rerank_smem, st>>>(
        X, D, w.qlist, w.dblist, q_lo, nq, cand, cap, counts, tau, K, w.norms_q, err_scale, bf16 ? w.res_q : nullptr,
        reinterpret_cast<const float *>(counters + 4), ids, d2, failed, counters + 1, reinterpret_cast<float *>(counters + 3), xp, kMinusZero2);
    B200_CUDA(cudaGetLastError());
    knn_tc_collect_failed_kernel<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>(failed, nq, w.qlist, flist, counters + 2);
    B200_CUDA(cudaGetLastError());
    phases.mark("rerank");
    int h[4] = {0, 0, 0, 0};
    B200_CUDA(cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, st));
    B200_CUDA(cudaStreamSynchronize(st));
    if (h[0]) { set_error("tensor-core kNN: a wait inside the kernel ran out of time"); return -2; }
    *n_failed_host = h[2];
    *failed_list = flist;
    if (err_ratio_host) memcpy(err_ratio_host, &h[3], sizeof(float));
    return 0;
}


// Runs mbar_wait_selftest_kernel: returns -5 when all 64 threads gave up within the limit (the expected
// outcome), 0 if any of them (wrongly) got through.
int mbar_wait_selftest(int timeout_ms, float *waited_ms, cudaStream_t st)
{
    if (timeout_ms <= 0 || timeout_ms > 2000) { set_error("mbarrier wait self-test: timeout must be 1..2000 ms"); return -1; }
    int *d = nullptr;
    cudaEvent_t a = nullptr, b = nullptr;
    struct Free { int *&d; cudaEvent_t &a, &b; ~Free() { if (d) cudaFree(d); if (a) cudaEventDestroy(a); if (b) cudaEventDestroy(b); } } guard{d, a, b};
    B200_CUDA(cudaMalloc((void **)&d, sizeof(int) * 2));
    B200_CUDA(cudaMemsetAsync(d, 0, sizeof(int) * 2, st));
    B200_CUDA(cudaEventCreate(&a));
    B200_CUDA(cudaEventCreate(&b));
    B200_CUDA(cudaEventRecord(a, st));
    mbar_wait_selftest_kernel<<<1, 64, 0, st>>>(d, d + 1, (unsigned long long)timeout_ms * 1000000ull);
    B200_CUDA(cudaGetLastError());
    B200_CUDA(cudaEventRecord(b, st));
    B200_CUDA(cudaStreamSynchronize(st));
    float ms = 0.0f;
    B200_CUDA(cudaEventElapsedTime(&ms, a, b));
    if (waited_ms) *waited_ms = ms;
    int h[2] = {0, 0};
    B200_CUDA(cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost));
    if (h[0] == 1 && h[1] == 64) { set_error("kNN pipeline: a barrier wait ran out (self-test)"); return -5; }
    return 0;
}

}  // namespace b200
