// Exact kNN by a tensor-core filter and an exact second look.
//
// The k nearest rows of a query are defined by the f32 FMA-chain distances of
// knn.cu's tile kernel; computing all n of them per query is FP32 issue work
// (166 ms for 200k x 30 dims). Here every pair is first scored on the tensor
// cores with an error bound, and only the few points whose score could still
// make them one of the k nearest get the exact chain:
//
//   score s(q, p) = q.p - |p|^2 / 2   (Euclidean; |q - p|^2 = |q|^2 - 2 s),
//                   q.p               (cosine, unit rows),
//
// formed as one bf16 contraction with f32 accumulators in TMEM: a coordinate
// is split into two bf16 pieces (hi, lo; products hi.hi, hi.lo, lo.hi) or, up
// to kFineDim dims, three (six products, f32 accuracy), and -|p|^2 / 2 rides
// along as three more columns against ones. Coordinates are taken relative to
// a mean of sampled rows, which changes no difference and keeps norms small.
//
//   1. k_filter<.., 1> over a sample of the point tiles: per query the largest
//      score in each of 64 groups of points. The (k + 1)-th largest of these
//      maxima belongs to k + 1 different points, so with the error bound it
//      gives a distance that at least k points other than the query keep to.
//   2. k_filter_threshold turns it into the least score a true neighbour can
//      have (bounds below).
//   3. k_filter<.., 2> over all tiles: indices of points at or above it, about
//      kHitTarget per query.
//   4. k_refine: exact chain distances of those, the k best by (distance,
//      index).
//
// The sample keeps step 1 at a fraction of step 3; the group maxima cost one
// three-input maximum per two scores with no branch, step 3 the same and a
// rarely taken branch. What bounds k_filter is the issue of its MMAs: 1.5 us a
// 256 x 256 tile at 30 dims (6 steps of 16 columns, 0.81 us at the tensor
// cores' rate), the same without the epilogue's arithmetic and without the
// staging; two epilogue warps a scheduler instead of four, descriptors formed
// in the loop and one lane issuing took 2.4 us. Against the FP32 tile kernel,
// whole knn_exact calls: 10k x 50 dims, k = 15 1.81 -> 0.71 ms, 200k x 30 dims,
// k = 30 166 -> 15.6 ms (of which the copies of host arrays take about 5).
//
// Ranks (trustworthiness: how many points are better than each of k given
// neighbours of a query) use the same scores. k_rank_bounds turns the
// neighbours' exact distances, sorted, into scores at or above which a point is
// surely better (hi) and below which it surely is not (lo); k_filter<1, 3>
// counts, per query, the points of every zone between them, and lists those
// inside a [lo, hi) interval; k_rank_refine settles these by their exact
// distances and adds up. 10k queries x 100k points x 50 dims, k = 15, whole
// call: 15.1 -> 5.4 ms.
//
// Error bound. With u = |q|, v = |p|: of a dot product the contraction leaves
// out lo.lo and the products with what the pieces leave of a coordinate; as
// norms these are at most rho_l and rho_r of a row's, the largest of the data
// (k_filter_norms), together u v (rho_l^2 + 2 rho_r + rho_r^2). (bf16 rounding
// alone bounds that by 4.7e-5 u v for two pieces; random data have 7e-6, and a
// seventh of the candidates near a threshold.) An MMA step adds 16 products to
// the f32 accumulator, each cut to the largest's last place at worst: 2^-19.8 of
// the magnitudes a step. (Measured against 64-bit sums of the same pieces, 2 to
// 191 dims, on rows of one sign with full mantissas, wide ranges or one large
// coordinate a step: at most 0.08 of that.) Centring and norms: a few 2^-24 of
// (u + v)^2. In all
// |s - s_true| <= kappa (u^2 + v^2) with filter_kappa. The chain distance
// itself is within (dim + 8) 2^-24 of the true one, relatively.
// k_filter_threshold carries both, so no true neighbour is left out; a looser
// threshold only means more candidates.
#include <cuda_bf16.h>

#include <cfloat>

#include "internal.cuh"
#include "knn_filter.cuh"

namespace umapcu {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kTileN = 256;       // points per tile (the MMA's N)
constexpr uint32_t kBlkM = 128;        // queries per accumulator (the MMA's M)
constexpr uint32_t kChunkK = 64;       // bf16 columns per staged chunk: a 128-byte row
constexpr uint32_t kABytes = kBlkM * kChunkK * 2;
constexpr uint32_t kBBytes = kTileN * kChunkK * 2;
constexpr uint32_t kGroups = 64;
constexpr uint32_t kFineDim = 10;      // 6 dim + 3 columns still fit one chunk
constexpr uint32_t kMaxChunks = 9;     // 144 KB of A beside two 32 KB stages of B
constexpr uint32_t kSmemMax = 232448 - 1024;
constexpr uint32_t kHalf = kTileN / 2; // columns of an accumulator an epilogue warp reads
constexpr int kFilterThreads = 576;    // 16 epilogue warps, a producer, an MMA issuer
// Candidates per query the sample is chosen for (fewer lengthen step 1, more
// steps 3 and 4: 73 and 146 are within 3 % of each other at 200k x 30 dims),
// and a query's list length.
constexpr uint32_t kHitTarget = 100, kListCap = 640;

struct Pack {
    uint32_t terms, cols, steps, chunks;
};

Pack pack_of(uint32_t dim)
{
    Pack p;
    p.terms = dim <= kFineDim ? 6 : 3;
    p.cols = p.terms * dim + 3;
    p.steps = (p.cols + 15) / 16;
    p.chunks = (p.cols + kChunkK - 1) / kChunkK;
    return p;
}

// kappa (above) of rows whose left-out parts are rho[0] (second pieces, when
// their product is left out) and rho[1] (what all pieces leave) of their norms.
__device__ __forceinline__ double filter_kappa(const float *rho, uint32_t steps)
{
    const double l = rho[0], r = rho[1];
    return 0.52 * (l * l + 2.0 * r + r * r) + 1.1e-6 * steps + 0x1p-21;
}

// ------------------------------------------------------------ preparation

// Column means of up to 1024 rows spread over the data, eight columns a block:
// any point near the data's centre serves.
__global__ void __launch_bounds__(1024) k_filter_centre(const float *__restrict__ x, uint32_t n, uint32_t dim,
                                                        float *__restrict__ mu)
{
    __shared__ float sh[128][8];
    const uint32_t rows = min(n, 1024u), e = threadIdx.x & 7, g = threadIdx.x >> 3, d = blockIdx.x * 8 + e;
    float acc = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) {
        const uint32_t r = g + 128 * i;
        if (r < rows && d < dim) acc += x[(size_t)((uint64_t)r * n / rows) * dim + d] / (float)rows;
    }
    sh[g][e] = acc;
    __syncthreads();
    for (uint32_t w = 64; w > 0; w >>= 1) {
        if (g < w) sh[g][e] += sh[g + w][e];
        __syncthreads();
    }
    if (g == 0 && d < dim) mu[d] = sh[0][e];
}

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// Piece t of v: what the t pieces before it leave, rounded to bf16.
__device__ __forceinline__ float bf16_piece(float v, uint32_t t)
{
    float p = bf16_round(v);
    for (uint32_t i = 0; i < t; i++) {
        v = v - p;
        p = bf16_round(v);
    }
    return p;
}

// |row - mu|^2 of every point, a warp per row, and into rho the largest shares
// of a row's norm that the contraction leaves out (filter_kappa); *bad set when
// a row is not finite or its norm is beyond what the bound's arithmetic can
// hold.
__global__ void k_filter_norms(const float *__restrict__ x, uint32_t n, uint32_t dim, const float *__restrict__ mu,
                               uint32_t terms, float *__restrict__ norm, float *__restrict__ rho,
                               uint32_t *__restrict__ bad)
{
    // (64 bits: 32 threads a row pass 2^32 from 2^27 rows on)
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t row = (uint32_t)(t >> 5), lane = threadIdx.x & 31;
    if (row >= n) return;
    double acc = 0.0;
    float second = 0.0f, rest = 0.0f;
    for (uint32_t d = lane; d < dim; d += 32) {
        const float f = x[(size_t)row * dim + d] - (mu ? mu[d] : 0.0f);
        acc += (double)f * (double)f;
        float r = f - bf16_round(f);
        const float l = bf16_round(r);
        r = r - l;
        if (terms == 6) r = r - bf16_round(r);
        else second += l * l;
        rest += r * r;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acc += __shfl_down_sync(kFull, acc, o);
        second += __shfl_down_sync(kFull, second, o);
        rest += __shfl_down_sync(kFull, rest, o);
    }
    if (lane != 0) return;
    norm[row] = (float)acc;
    if (!(acc < 1e28)) *bad = 1u;
    if (!(acc > 1e-30)) return;  // (the bound's absolute part covers rows this small)
    // (sums of up to 191 f32 squares: rounded up by 1e-4)
    const float inv = (float)(1.0001 / acc);
    const float a = sqrtf(second * inv), b = sqrtf(rest * inv);
    if (a > rho[0]) atomicMax((int *)&rho[0], __float_as_int(a));  // (stale reads only cost an atomic)
    if (b > rho[1]) atomicMax((int *)&rho[1], __float_as_int(b));
}

// The operands as the shared-memory images the MMA reads: K-major rows of 64
// columns (128 bytes) in the 128-byte swizzle (16-byte unit j of row r stands
// at j ^ (r & 7)), so that a plain bulk copy stages a chunk. Queries: blocks
// of 128 rows, [block][chunk][128 rows]; points: tiles of 256 rows,
// [tile][chunk][256 rows]. A thread writes one 16-byte unit (8 columns).
// Rows past the end are zero, past the points with a score of -1e30.
template <bool QUERY>
__global__ void k_filter_pack(const float *__restrict__ x, uint32_t n, uint32_t dim, const float *__restrict__ mu,
                              const float *__restrict__ norm, const uint32_t *__restrict__ qidx, uint32_t q0,
                              uint32_t rows, uint32_t rows_pad, uint32_t terms, uint32_t chunks, bool euc,
                              uint4 *__restrict__ out)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t units = chunks * 8;
    if (t >= (uint64_t)rows_pad * units) return;
    const uint32_t r = (uint32_t)(t / units), u = (uint32_t)(t % units);
    const bool in = r < rows;
    const uint32_t row = !in ? 0u : QUERY ? (qidx ? qidx[q0 + r] : q0 + r) : r;
    const uint32_t cols = terms * dim;
    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) {
        const uint32_t c = u * 8 + i;
        float f = 0.0f;
        if (c < cols) {
            if (in) {
                const uint32_t term = c / dim, d = c - term * dim;
                // products of pieces, query x point: 00 01 10 (11 02 20)
                const uint32_t piece = ((QUERY ? 0x201100u : 0x021010u) >> (4 * term)) & 15u;
                const float xv = x[(size_t)row * dim + d] - (mu ? mu[d] : 0.0f);
                f = bf16_piece(xv, piece);
            }
        } else if (c < cols + 3) {
            if (QUERY) f = 1.0f;
            else if (!in) f = c == cols ? -1e30f : 0.0f;
            else if (euc) f = -bf16_piece(0.5f * norm[row], c - cols);
        }
        v[i] = __float2bfloat16_rn(f);
    }
    const uint32_t per = QUERY ? kBlkM : kTileN;
    const uint32_t blk = r / per, rr = r % per, chunk = u >> 3, j = u & 7;
    out[(((size_t)blk * chunks + chunk) * per + rr) * 8 + (j ^ (rr & 7))] = *reinterpret_cast<const uint4 *>(v);
}

// ------------------------------------------------------- PTX of the kernel

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t *b, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t *b, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t *b, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false after about two seconds of clock cycles, or when another
// role of the block has given up.
__device__ __forceinline__ bool bar_wait(uint64_t *b, uint32_t parity, volatile uint32_t *stop)
{
    if (bar_try(b, parity)) return true;
    const long long t0 = clock64();
    while (!bar_try(b, parity)) {
        if (*stop) return false;
        if (clock64() - t0 > 4000000000ll) {
            *stop = 1u;
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *b)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}
// K-major, 128-byte swizzle, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t mma_desc(uint32_t addr)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// One lane issues; the whole warp runs the loop around it, which keeps the
// operands in uniform registers.
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *b)
{
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_addr(b))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float (&v)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]),
          "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]),
          "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(addr)
        : "memory");
}
// The loaded registers are named so that no use of them moves before the wait.
template <int N>
__device__ __forceinline__ void tmem_wait(float (&v)[N])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; i++) asm volatile("" : "+f"(v[i]));
}
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// -------------------------------------------------------------- the filter

struct FilterArgs {
    const uint4 *a, *b;      // operand images of the query batch and the points
    uint32_t nq, n_tiles, stride, slices;
    uint32_t chunks, steps, stages;
    // PASS 1
    float *gmax;             // [parts][nq][kGroups]
    // PASS 2
    const float *least;      // [nq]
    uint32_t *list;          // [parts][nq][cap]
    uint32_t *count;         // [parts][nq], may exceed cap
    uint32_t cap;
    // PASS 3 (list, count, cap as above)
    uint32_t k, zone_rows;   // zone_rows = 2^steps - 1 >= k
    const float *hi, *lo;    // [nq][k], descending
    const uint32_t *qidx;    // the query rows, or nullptr: q0 + q
    uint32_t q0;
    uint32_t *zones;         // [nq][32], added to
    uint32_t *bad;           // set when a wait gave up
};

// One block: MB x 128 queries against the tiles slice, slice + slices, ... (of
// every stride-th tile). Warp 16 stages point chunks through a ring of 32 KB
// bulk copies, warp 17 issues the MMAs (128 x 256 x 16), warps 0-7 and 8-15
// read accumulators 0 and 1 (a thread 128 columns of one query's row, in two
// loads of 64, after which the accumulator is free). MB = 2: accumulator b holds query block b, so that one
// is contracted while the other is read and a staged tile serves 256 queries
// (32 bytes of L2 reads a clock where 64 would be needed with one block).
// MB = 1, for operands of more than three chunks, whose A would not leave room
// for the ring: the accumulators alternate between tiles. 512 columns of TMEM
// and more than half the shared memory: one block an SM.
// PASS 3 (MB = 1): per score a search of the query's hi scores (the first two
// levels in registers, the others in shared memory, laid out by row, so that the
// lanes of a warp never meet in a bank), one comparison with a lo score and one
// count of the thread's own zone. The search bounds it. STEPS: of that search,
// 2^STEPS > k. Up to 15 thresholds a tile's counts are kept in packed registers,
// four bits a zone for eight scores, then a byte; with 32 zones that takes more
// shifts than it saves, and each score is an add in shared memory. Whole calls,
// 10k queries of 100k points, all levels and counters in shared memory ->
// levels in registers -> packed counts: k = 15 5.18 -> 5.05 -> 4.87 ms, k = 20
// 5.94 -> 5.70 ms (5.82 with packed counts).
template <int MB, int PASS, int STEPS = 0>
__global__ void __launch_bounds__(kFilterThreads, 1) k_filter(const FilterArgs P)
{
    extern __shared__ uint8_t dyn[];
    __shared__ uint64_t full[8], empty[8], tfull[2], tempty[2], afull, done;
    __shared__ uint32_t tmem_base;
    __shared__ uint32_t stop_word;
    volatile uint32_t *stop = &stop_word;
    uint8_t *sa = reinterpret_cast<uint8_t *>(((uintptr_t)dyn + 1023) & ~(uintptr_t)1023);
    uint8_t *sb = sa + (size_t)MB * P.chunks * kABytes;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t slice = blockIdx.y;
    if constexpr (PASS == 2) {  // a block without a query to be listed has nothing to contract
        const uint32_t q = blockIdx.x * MB * kBlkM + threadIdx.x;
        const bool in = threadIdx.x < MB * kBlkM && q < P.nq;
        if (!__syncthreads_or(in && P.least[q] < __int_as_float(0x7f800000))) {
            constexpr uint32_t kParts = MB == 2 ? 2 : 4;  // of a slice
            for (uint32_t p = 0; in && p < kParts; p++) P.count[(size_t)(slice * kParts + p) * P.nq + q] = 0;
            return;
        }
    }
    const uint32_t sampled = (P.n_tiles + P.stride - 1) / P.stride;
    const uint32_t n_items = sampled > slice ? (sampled - slice + P.slices - 1) / P.slices : 0;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < P.stages; i++) {
            bar_init(&full[i], 1);
            bar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            bar_init(&tfull[i], 1);
            bar_init(&tempty[i], 8);
        }
        bar_init(&afull, 1);
        bar_init(&done, 1);
        stop_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 17) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_base))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const uint32_t C = P.chunks, R = P.stages;

    if (warp == 16) {
        if (lane == 0) {
            const uint8_t *ga = reinterpret_cast<const uint8_t *>(P.a) + (size_t)blockIdx.x * MB * C * kABytes;
            bar_expect(&afull, MB * C * kABytes);
            for (uint32_t i = 0; i < MB * C; i++) bulk_load(sa + (size_t)i * kABytes, ga + (size_t)i * kABytes, kABytes, &afull);
            uint32_t it = 0;
            bool ok = true;
            for (uint32_t i = 0; ok && i < n_items; i++) {
                const uint8_t *gb =
                    reinterpret_cast<const uint8_t *>(P.b) + (size_t)((slice + i * P.slices) * P.stride) * C * kBBytes;
                for (uint32_t c = 0; c < C; c++, it++) {
                    const uint32_t st = it % R;
                    ok = bar_wait(&empty[st], ((it / R) & 1) ^ 1, stop);
                    if (!ok) break;
                    bar_expect(&full[st], kBBytes);
                    bulk_load(sb + (size_t)st * kBBytes, gb + (size_t)c * kBBytes, kBBytes, &full[st]);
                }
            }
            // what is in flight ends before the block does: the copies of the
            // last stages (the MMAs are warp 17's to wait for)
            for (uint32_t b = it > R ? it - R : 0; b < it; b++) {
                uint32_t none = 0;
                bar_wait(&full[b % R], (b / R) & 1, &none);
            }
            uint32_t none = 0;
            bar_wait(&afull, 0, &none);
        }
        __syncwarp();
    } else if (warp == 17) {
        // f32 accumulators, bf16 operands, both K-major, N = 256, M = 128
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kTileN >> 3) << 17) | ((kBlkM >> 4) << 24);
        const uint64_t da0 = mma_desc(smem_addr(sa)), db0 = mma_desc(smem_addr(sb));
        const uint32_t last = P.steps - 4 * (C - 1);  // steps of the last chunk
        // the lanes leave the loop together: a wait given up by one ends it for all
        bool ok = __all_sync(kFull, bar_wait(&afull, 0, stop));
        uint32_t st0 = 0, ph0 = 0;  // ring place of the tile's first chunk
        for (uint32_t i = 0; ok && i < n_items; i++) {
            uint32_t st = st0, ph = ph0;
#pragma unroll
            for (uint32_t m = 0; m < (uint32_t)MB; m++) {
                const uint32_t buf = MB == 2 ? m : i & 1, use = MB == 2 ? i : i >> 1;
                ok = __all_sync(kFull, ok && bar_wait(&tempty[buf], (use & 1) ^ 1, stop));
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                st = st0;
                ph = ph0;
                const uint32_t acc = tmem + buf * kTileN;
                uint64_t da = da0 + (uint64_t)(m * C) * (kABytes >> 4);
                for (uint32_t c = 0; c < C; c++) {
                    ok = __all_sync(kFull, ok && bar_wait(&full[st], ph, stop));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t db = db0 + (uint64_t)st * (kBBytes >> 4);
                    const uint32_t ks = c + 1 < C ? 4u : last;
                    mma_bf16(acc, da, db, idesc, c > 0);
                    if (ks > 1) mma_bf16(acc, da + 2, db + 2, idesc, true);
                    if (ks > 2) mma_bf16(acc, da + 4, db + 4, idesc, true);
                    if (ks > 3) mma_bf16(acc, da + 6, db + 6, idesc, true);
                    if (m + 1 == (uint32_t)MB) mma_commit(&empty[st]);
                    da += kABytes >> 4;
                    if (++st == R) {
                        st = 0;
                        ph ^= 1;
                    }
                }
                if (ok) mma_commit(&tfull[buf]);
            }
            st0 = st;
            ph0 = ph;
        }
        // what was issued ends before TMEM and the staged operands are given
        // back, whoever gave up and when
        mma_commit(&done);
        uint32_t none = 0;
        bar_wait(&done, 0, &none);
    } else {
        // columns 128 half .. of accumulator b, rows 32 quarter ..
        const uint32_t b = warp >> 3, half = (warp >> 2) & 1, quarter = warp & 3;
        const uint32_t uses = MB == 2 ? n_items : (n_items + 1 - b) / 2;
        const uint32_t q = blockIdx.x * MB * kBlkM + (MB == 2 ? b * kBlkM : 0) + quarter * 32 + lane;
        const uint32_t t0 = tmem + ((quarter * 32) << 16) + b * kTileN + half * kHalf;
        bool ok = true;
        if constexpr (PASS == 1) {
            const uint32_t part = MB == 2 ? slice : slice * 2 + b;
            float g[32];
#pragma unroll
            for (int j = 0; j < 32; j++) g[j] = -3e38f;
            for (uint32_t u = 0; ok && u < uses; u++) {
                ok = __all_sync(kFull, bar_wait(&tfull[b], u & 1, stop));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                float v[2][32];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    tmem_ld32(t0 + 64 * h, v[0]);
                    tmem_ld32(t0 + 64 * h + 32, v[1]);
                    tmem_wait(v[0]);
                    tmem_wait(v[1]);
                    if (h == 1) {  // the accumulator is read: the next tile's MMAs may write it
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) bar_arrive(&tempty[b]);
                    }
#pragma unroll
                    for (int j = 0; j < 32; j++) g[j] = max3(g[j], v[0][j], v[1][j]);
                }
            }
            if (q < P.nq) {
                float4 *o = reinterpret_cast<float4 *>(P.gmax + ((size_t)part * P.nq + q) * kGroups + half * 32);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    o[j] = make_float4(g[4 * j], g[4 * j + 1], g[4 * j + 2], g[4 * j + 3]);
            }
        } else if constexpr (PASS == 2) {
            const uint32_t part = (MB == 2 ? slice : slice * 2 + b) * 2 + half;
            const float least = q < P.nq ? P.least[q] : __int_as_float(0x7f800000);
            uint32_t *list = P.list + ((size_t)part * P.nq + (q < P.nq ? q : 0)) * P.cap;
            uint32_t count = 0;
            for (uint32_t u = 0; ok && u < uses; u++) {
                ok = __all_sync(kFull, bar_wait(&tfull[b], u & 1, stop));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t item = MB == 2 ? u : 2 * u + b;
                const uint32_t p0 = (slice + item * P.slices) * P.stride * kTileN + half * kHalf;
                constexpr int kS = (int)kHalf / 32;
                uint32_t hit[kS];
                float v[2][32];
                tmem_ld32(t0, v[0]);
                tmem_ld32(t0 + 32, v[1]);
#pragma unroll
                for (int h = 0; h < kS; h++) {
                    float(&w)[32] = v[h & 1];
                    if (h == 0 || h == 2) {
                        tmem_wait(v[0]);
                        tmem_wait(v[1]);
                    }
                    if (h == 2) {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) bar_arrive(&tempty[b]);
                    }
                    float m[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        m[e] = max3(w[8 * e], w[8 * e + 1], w[8 * e + 2]);
                        m[e] = max3(m[e], w[8 * e + 3], w[8 * e + 4]);
                        m[e] = max3(m[e], w[8 * e + 5], w[8 * e + 6]);
                        m[e] = fmaxf(m[e], w[8 * e + 7]);
                    }
                    hit[h] = 0;
                    if (fmaxf(max3(m[0], m[1], m[2]), m[3]) >= least) {
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (m[e] >= least) {
#pragma unroll
                                for (int j = 0; j < 8; j++) hit[h] |= w[8 * e + j] >= least ? 1u << (8 * e + j) : 0u;
                            }
                    }
                    if (h < 2) tmem_ld32(t0 + 64 + 32 * h, w);
                }
#pragma unroll
                for (int h = 0; h < kS; h++)
                    while (hit[h]) {
                        if (count < P.cap) list[count] = p0 + 32 * h + (uint32_t)__ffs(hit[h]) - 1u;
                        count++;
                        hit[h] &= hit[h] - 1u;
                    }
            }
            if (q < P.nq) P.count[(size_t)part * P.nq + q] = count;
        } else {
            const uint32_t part = (slice * 2 + b) * 2 + half;
            float *tables = reinterpret_cast<float *>(sb + (size_t)R * kBBytes);
            float *hi = tables + quarter * 32 + lane;         // [zone_rows][128]
            float *lo = hi + (size_t)P.zone_rows * kBlkM;     // [k + 1][128]: row m of threshold m - 1, row 0 infinite
            uint32_t *zone = reinterpret_cast<uint32_t *>(tables + (size_t)(P.zone_rows + P.k + 1) * kBlkM) + threadIdx.x;
            const bool in = q < P.nq;
            if (b == 0 && half == 0) {
                for (uint32_t m = 0; m < P.zone_rows; m++)
                    hi[m * kBlkM] = in && m < P.k ? P.hi[(size_t)q * P.k + m] : __int_as_float(0xff800000);
                lo[0] = __int_as_float(0x7f800000);
                for (uint32_t m = 0; m < P.k; m++)
                    lo[(m + 1) * kBlkM] = in ? P.lo[(size_t)q * P.k + m] : __int_as_float(0x7f800000);
            }
            for (uint32_t m = 0; m <= P.k; m++) zone[m * 512] = 0;
            asm volatile("bar.sync 1, 512;" ::: "memory");  // the epilogue warps
            // the search's first two levels stay in registers
            constexpr int kTop = STEPS > 1 ? 1 << (STEPS - 1) : 2;
            const float h1 = hi[(kTop - 1) * kBlkM], h2a = hi[(kTop / 2 - 1) * kBlkM], h2b = hi[(kTop + kTop / 2 - 1) * kBlkM];
            const uint32_t self = !in ? ~0u : P.qidx ? P.qidx[P.q0 + q] : P.q0 + q;
            uint32_t *list = P.list + ((size_t)part * P.nq + (in ? q : 0)) * P.cap;
            uint32_t count = 0;
            for (uint32_t u = 0; ok && u < uses; u++) {
                ok = __all_sync(kFull, bar_wait(&tfull[b], u & 1, stop));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t p0 = (slice + (2 * u + b) * P.slices) * P.stride * kTileN + half * kHalf;
                uint64_t even = 0, odd = 0;  // STEPS = 4: the tile's counts, a byte a zone (at most 128)
                for (int h = 0; h < (int)kHalf / 32; h++) {
                    float w[32];
                    tmem_ld32(t0 + 32 * h, w);
                    tmem_wait(w);
                    if (h + 1 == (int)kHalf / 32) {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) bar_arrive(&tempty[b]);
                    }
                    const uint32_t pc = p0 + 32 * h;
                    if (self - pc < 32u) {  // the query itself counts for nothing
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (self - pc == (uint32_t)j) w[j] = __int_as_float(0xff800000);
                    }
                    uint32_t open = 0;
#pragma unroll
                    for (int j0 = 0; j0 < 32; j0 += 8) {
                        // m: thresholds with hi above the score, which is
                        // surely better than the later ones. Eight searches
                        // side by side, and only then the counters: a store
                        // between them would hold back the next one's loads
                        uint32_t m[8];
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const bool far = w[j0 + j] < h1;
                            m[j] = (far ? kTop : 0) + (w[j0 + j] < (far ? h2b : h2a) ? kTop / 2 : 0);
                        }
#pragma unroll
                        for (int st = kTop / 4; st > 0; st >>= 1)
#pragma unroll
                            for (int j = 0; j < 8; j++)
                                if (w[j0 + j] < hi[(m[j] + st - 1) * kBlkM]) m[j] += st;
                        // unsettled unless surely worse than the last of these
                        uint32_t un = 0;
#pragma unroll
                        for (int j = 0; j < 8; j++) un |= w[j0 + j] >= lo[m[j] * kBlkM] ? 1u << j : 0u;
                        open |= un << j0;
                        if constexpr (STEPS == 4) {
                            uint64_t eight = 0;  // four bits a zone; a shift by 64 counts nothing
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                uint64_t one;
                                asm("shl.b64 %0, %1, %2;" : "=l"(one) : "l"(1ull), "r"((un >> j) & 1u ? 64u : 4u * m[j]));
                                eight += one;
                            }
                            even += eight & 0x0f0f0f0f0f0f0f0full;
                            odd += (eight >> 4) & 0x0f0f0f0f0f0f0f0full;
                        } else {
#pragma unroll
                            for (int j = 0; j < 8; j++)
                                if (!((un >> j) & 1u)) atomicAdd(&zone[m[j] * 512], 1u);
                        }
                    }
                    while (open) {
                        if (count < P.cap) list[count] = pc + (uint32_t)__ffs(open) - 1u;
                        count++;
                        open &= open - 1u;
                    }
                }
                if constexpr (STEPS == 4) {
#pragma unroll
                    for (uint32_t m = 0; m < 15; m++)
                        if (m < P.k) zone[m * 512] += (uint32_t)((m & 1u ? odd : even) >> (8 * (m / 2))) & 0xffu;
                }
            }
            if (in) {
                P.count[(size_t)part * P.nq + q] = count;
                for (uint32_t m = 0; m < P.k; m++)
                    if (zone[m * 512]) atomicAdd(&P.zones[(size_t)q * 32 + m], zone[m * 512]);
            }
        }
        if (!ok && lane == 0) *P.bad = 1u;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x == 0 && stop_word) *P.bad = 1u;
    if (warp == 17) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// The least score a true neighbour of each query can have; a warp per query.
// v, the (k + 1)-th largest group maximum, stands for k + 1 different points,
// at least k of them not the query itself.
// Euclidean: such a point has distance D <= u^2 - 2 (v - E), where E =
// kappa (u^2 + w^2) + 1e-30 and w bounds its norm (w <= u + sqrt(D), solved
// with the bound's own share of D); a true neighbour's distance is then at
// most D (1 + 4 gamma), gamma = (dim + 8) 2^-24 covering the chain's rounding
// on both sides, its norm at most u + sqrt of that, its score at least (u^2 -
// D (1 + 4 gamma)) / 2 less the bound. Cosine: scores are the dot products of
// unit rows, E = 2.1 kappa, the chain's rounding dim 2^-24 on both sides and
// that of 1 - dot.
// A query with every group's maximum at or above that least score (some 300
// points of the sample are, in 64 groups) has more candidates than its lists
// hold or pay for: give_up (knn_filter) sends it on without listing any. The
// points of tight clusters far apart or of equal rows all are such: 200k x 30
// dims 163.6 -> 151.4 ms (151.1 by the tile kernel alone).
__global__ void k_filter_threshold(const float *__restrict__ gmax, uint32_t parts, uint32_t nq, uint32_t k,
                                   const float *__restrict__ norm, const uint32_t *__restrict__ qidx, uint32_t q0,
                                   uint32_t dim, bool euc, const float *__restrict__ rho, uint32_t steps, bool give_up,
                                   float *__restrict__ least)
{
    const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (q >= nq) return;  // warp-uniform
    float v0 = -3e38f, v1 = -3e38f;
    for (uint32_t p = 0; p < parts; p++) {
        const float2 f = __ldcs(reinterpret_cast<const float2 *>(gmax + ((size_t)p * nq + q) * kGroups) + lane);
        v0 = fmaxf(v0, f.x);
        v1 = fmaxf(v1, f.y);
    }
    // unsigned integers in the floats' order
    uint32_t o0 = __float_as_uint(v0), o1 = __float_as_uint(v1);
    o0 = (o0 & 0x80000000u) ? ~o0 : o0 | 0x80000000u;
    o1 = (o1 & 0x80000000u) ? ~o1 : o1 | 0x80000000u;
    uint32_t top = 0;
    for (uint32_t r = 0; r <= k; r++) {
        const uint32_t mine = max(o0, o1);
        top = __reduce_max_sync(kFull, mine);
        const unsigned who = __ballot_sync(kFull, mine == top);
        if ((int)lane == __ffs(who) - 1) {
            if (o0 == top) o0 = 0;
            else o1 = 0;
        }
    }
    const double kappa = filter_kappa(rho, steps);
    const double s = (double)__uint_as_float((top & 0x80000000u) ? top ^ 0x80000000u : ~top);
    double g;
    if (euc) {
        const double u2 = (double)norm[qidx ? qidx[q0 + q] : q0 + q], u = sqrt(u2), tiny = 1e-30;
        const double d0 = fmax(u2 - 2.0 * s, 0.0);
        const double w = (u + sqrt(d0 + 2.0 * kappa * u2 + tiny)) / (1.0 - sqrt(2.0 * kappa));
        const double d1 = (d0 + 2.0 * (kappa * (u2 + w * w) + tiny)) * (1.0 + 4.0 * (dim + 8) * 0x1p-24);
        const double w1 = u + sqrt(d1);
        g = 0.5 * (u2 - d1) - kappa * (u2 + w1 * w1) - 2.0 * tiny;
    } else {
        g = s - 2.0 * 2.1 * kappa - (2.0 * dim + 16.0) * 0x1p-24 - 0x1p-22;
    }
    const float l = __double2float_rd(g);
    const bool all = __all_sync(kFull, v0 >= l && v1 >= l);
    if (lane == 0) least[q] = give_up && all ? __int_as_float(0x7f800000) : l;
}

// The candidates listed for query q, all parts together.
__device__ __forceinline__ uint32_t listed(const uint32_t *__restrict__ count, uint32_t parts, uint32_t nq, uint32_t q,
                                           uint32_t lane)
{
    uint32_t c = 0;
    for (uint32_t p = lane; p < parts; p += 32) c += min(count[(size_t)p * nq + q], 1u << 20);
    return __reduce_add_sync(kFull, c);
}

__device__ __forceinline__ bool better(float d, uint32_t i, float td, uint32_t ti)
{
    return d < td || (d == td && i < ti);
}

// The chain distances (knn.cu) of a query's row xq to the 32 candidate rows
// `mine`, one per lane, the first `rows` of them wanted: rows staged through
// the warp's shared memory 32 dims at a time (coalesced; a lane reading its own
// candidate's row would touch 32 lines a load).
template <bool EUC>
__device__ __forceinline__ float chain_distance(const float *__restrict__ x, uint32_t dim, const float *__restrict__ xq,
                                                uint32_t mine, uint32_t rows, float (&S)[32][33], uint32_t lane)
{
    float acc = 0.0f;
    for (uint32_t d0 = 0; d0 < dim; d0 += 32) {
        const uint32_t w = min(32u, dim - d0);
        __syncwarp();
        if (w > 16) {
#pragma unroll 8
            for (uint32_t r = 0; r < rows; r++) {
                const uint32_t id = __shfl_sync(kFull, mine, r);
                if (lane < w) S[r][lane] = __ldg(x + (size_t)id * dim + d0 + lane);
            }
        } else {  // two rows a step
            for (uint32_t r = 0; r < rows; r += 2) {
                const uint32_t id = __shfl_sync(kFull, mine, (r + (lane >> 4)) & 31u);
                const uint32_t e = lane & 15;
                if (e < w) S[r + (lane >> 4)][e] = __ldg(x + (size_t)id * dim + d0 + e);
            }
        }
        __syncwarp();
        for (uint32_t d = 0; d < w; d++) {
            const float a = __ldg(xq + d0 + d), v = S[lane][d];
            if (EUC) {
                const float df = a - v;
                acc = __fmaf_rn(df, df, acc);
            } else {
                acc = __fmaf_rn(a, v, acc);
            }
        }
    }
    return EUC ? acc : 1.0f - acc;
}

// The exact second look, a warp per query: 32 candidates at a time, their
// chain distances, and insertion into the warp's sorted list (lane l holds
// entry l). A query whose lists overflowed or hold more than a quarter of the
// points (row by row that costs more than the tile kernel's pass over all;
// metrics of 3000 equal rows, whole call: 1.39 -> 0.71 ms, 0.64 by the tile
// kernel alone), or any query when *bad, goes to left.
constexpr int kRefineWarps = 4;
template <bool EUC>
__global__ void __launch_bounds__(kRefineWarps * 32) k_refine(const float *__restrict__ x, uint32_t n, uint32_t dim, uint32_t k,
                                                              const uint32_t *__restrict__ qidx, uint32_t q0,
                                                              uint32_t nq, const uint32_t *__restrict__ list,
                                                              const uint32_t *__restrict__ count, uint32_t parts,
                                                              uint32_t cap, const uint32_t *__restrict__ bad,
                                                              uint32_t *__restrict__ out_idx,
                                                              float *__restrict__ out_dist,
                                                              uint32_t *__restrict__ left, uint32_t *__restrict__ n_left)
{
    __shared__ float sh[kRefineWarps][32][33];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t q = blockIdx.x * kRefineWarps + warp;
    if (q >= nq) return;  // warp-uniform
    const uint32_t self = qidx ? qidx[q0 + q] : q0 + q;
    bool over = *bad != 0 || (n / 4 < parts * cap && listed(count, parts, nq, q, lane) > n / 4);
    float ld = __int_as_float(0x7f800000);
    uint32_t li = ~0u;
    for (uint32_t p = 0; !over && p < parts; p++) {
        const uint32_t c = count[(size_t)p * nq + q];
        if (c > cap) {
            over = true;
            break;
        }
        const uint32_t *L = list + ((size_t)p * nq + q) * cap;
        for (uint32_t b = 0; b < c; b += 32) {
            bool live = b + lane < c;
            uint32_t mine = live ? L[b + lane] : self;
            if (mine >= n) {  // the last tile's padding, listed only under a threshold that excludes nothing
                live = false;
                mine = self;
            }
            const float dist =
                chain_distance<EUC>(x, dim, x + (size_t)self * dim, mine, min(32u, c - b), sh[warp], lane);
            float td = __shfl_sync(kFull, ld, k - 1);
            uint32_t ti = __shfl_sync(kFull, li, k - 1);
            unsigned pend = __ballot_sync(kFull, live && mine != self && better(dist, mine, td, ti));
            while (pend) {
                const int src = __ffs(pend) - 1;
                pend &= pend - 1;
                const float cd = __shfl_sync(kFull, dist, src);
                const uint32_t ci = __shfl_sync(kFull, mine, src);
                const uint32_t pos = __popc(__ballot_sync(kFull, better(ld, li, cd, ci)));
                const float ud = __shfl_up_sync(kFull, ld, 1);
                const uint32_t ui = __shfl_up_sync(kFull, li, 1);
                if (lane < k) {
                    if (lane > pos) {
                        ld = ud;
                        li = ui;
                    } else if (lane == pos) {
                        ld = cd;
                        li = ci;
                    }
                }
            }
        }
    }
    if (!over && __shfl_sync(kFull, li, k - 1) == ~0u) over = true;  // fewer than k: never with a true bound
    if (over) {
        if (lane == 0) left[atomicAdd(n_left, 1u)] = q0 + q;
    } else if (lane < k) {
        out_idx[(size_t)(q0 + q) * k + lane] = li;
        out_dist[(size_t)(q0 + q) * k + lane] = ld;
    }
}

// Ranks: the sorted thresholds of every query, a warp each, and their scores.
// A point is better than a threshold T only at a chain distance of at most T,
// so (gamma as above) surely when its true distance D is below T (1 - 2 gamma)
// and surely not above T (1 + 2 gamma). Its score lies within kappa (u^2 +
// v^2) of (u^2 - D) / 2 with a norm v of at most u + sqrt(D): with
// f(D) = (u^2 - D) / 2 + kappa (u^2 + (u + sqrt D)^2), which falls in D from
// D0 = (2 kappa u / (1 - 2 kappa))^2 on, no point at or beyond T (1 - 2 gamma)
// scores more than hi = f(max(D0, T (1 - 2 gamma))), and none up to T (1 + 2
// gamma) less than lo, the same with -kappa. Cosine: scores are dot products,
// the threshold's 1 - T, the bound as in k_filter_threshold. A threshold that
// is no number goes to *bad.
__global__ void k_rank_bounds(const float *__restrict__ thr_d, const uint32_t *__restrict__ thr_j, uint32_t nq, uint32_t k,
                              const float *__restrict__ norm, const uint32_t *__restrict__ qidx, uint32_t q0, uint32_t dim,
                              bool euc, const float *__restrict__ rho, uint32_t steps, float *__restrict__ hi,
                              float *__restrict__ lo,
                              uint32_t *__restrict__ given, uint32_t *__restrict__ bad)
{
    const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (q >= nq) return;  // warp-uniform
    const size_t at = (size_t)(q0 + q) * k;
    const float td = lane < k ? thr_d[at + lane] : 0.0f;
    const uint32_t tj = lane < k ? thr_j[at + lane] : 0u;
    if (lane < k && !(td <= FLT_MAX)) *bad = 1u;
    uint32_t place = 0;  // a repeated neighbour keeps the order of the lanes
    for (uint32_t m = 0; m < k; m++) {
        const float od = __shfl_sync(kFull, td, m);
        const uint32_t oj = __shfl_sync(kFull, tj, m);
        place += (better(od, oj, td, tj) || (od == td && oj == tj && m < lane)) ? 1u : 0u;
    }
    if (lane >= k || place >= k) return;
    const double kappa = filter_kappa(rho, steps);
    double up, down;
    if (euc) {
        const double u2 = (double)norm[qidx ? qidx[q0 + q] : q0 + q], u = sqrt(u2), tiny = 1e-30;
        const double gamma = (dim + 8) * 0x1p-24, t1 = (double)td * (1.0 - 2.0 * gamma), t2 = (double)td * (1.0 + 2.0 * gamma);
        const double r0 = 2.0 * kappa * u / (1.0 - 2.0 * kappa), r1 = fmax(r0, sqrt(fmax(t1, 0.0))), r2 = sqrt(fmax(t2, 0.0));
        up = 0.5 * (u2 - r1 * r1) + kappa * (u2 + (u + r1) * (u + r1)) + tiny;
        down = 0.5 * (u2 - r2 * r2) - kappa * (u2 + (u + r2) * (u + r2)) - tiny;
    } else {
        const double e = 2.1 * kappa + (dim + 16.0) * 0x1p-24 + 0x1p-22;
        up = 1.0 - (double)td + e;
        down = 1.0 - (double)td - e;
    }
    const size_t o = (size_t)q * k + place;
    hi[o] = __double2float_ru(up);
    lo[o] = __double2float_rd(down);
    given[o] = lane;
}

// The listed points of every query, settled by their chain distances against
// all its thresholds (lane m holds the m-th of the sorted ones), plus the zone
// counts: a point of zone z is better than the thresholds from z on.
template <bool EUC>
__global__ void __launch_bounds__(kRefineWarps * 32)
    k_rank_refine(const float *__restrict__ x, uint32_t n, uint32_t dim, uint32_t k, const uint32_t *__restrict__ qidx,
                  uint32_t q0, uint32_t nq, const float *__restrict__ thr_d, const uint32_t *__restrict__ thr_j,
                  const uint32_t *__restrict__ given, const uint32_t *__restrict__ zones, const uint32_t *__restrict__ list,
                  const uint32_t *__restrict__ count, uint32_t parts, uint32_t cap, const uint32_t *__restrict__ bad,
                  uint32_t *__restrict__ counts, uint32_t *__restrict__ left, uint32_t *__restrict__ n_left)
{
    __shared__ float sh[kRefineWarps][32][33];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t q = blockIdx.x * kRefineWarps + warp;
    if (q >= nq) return;  // warp-uniform
    const uint32_t self = qidx ? qidx[q0 + q] : q0 + q;
    bool over = *bad != 0 || (n / 4 < parts * cap && listed(count, parts, nq, q, lane) > n / 4);
    const size_t at = (size_t)(q0 + q) * k;
    uint32_t c_m = 0, g = 0, tj = 0;
    float td = 0.0f;
    if (!over && lane < k) {
        c_m = zones[(size_t)q * 32 + lane];
        g = given[(size_t)q * k + lane];
        td = thr_d[at + g];
        tj = thr_j[at + g];
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, c_m, off);
        if ((int)lane >= off) c_m += u;
    }
    for (uint32_t p = 0; !over && p < parts; p++) {
        const uint32_t c = count[(size_t)p * nq + q];
        if (c > cap) {
            over = true;
            break;
        }
        const uint32_t *L = list + ((size_t)p * nq + q) * cap;
        for (uint32_t b = 0; b < c; b += 32) {
            const uint32_t rows = min(32u, c - b);
            uint32_t mine = lane < rows ? L[b + lane] : self;
            if (mine >= n) mine = self;
            const float dist = chain_distance<EUC>(x, dim, x + (size_t)self * dim, mine, rows, sh[warp], lane);
            for (uint32_t r = 0; r < rows; r++) {
                const float d = __shfl_sync(kFull, dist, r);
                const uint32_t i = __shfl_sync(kFull, mine, r);
                c_m += (i != self && better(d, i, td, tj)) ? 1u : 0u;
            }
        }
    }
    if (over) {
        if (lane == 0) left[atomicAdd(n_left, 1u)] = q0 + q;
    } else if (lane < k) {
        counts[at + g] = c_m;
    }
}

template <int MB, int PASS, int STEPS = 0>
void launch_filter(const FilterArgs &P, uint32_t blocks, size_t smem, cudaStream_t s)
{
    // the most of any call: the attribute is the function's, shared by all threads
    check_cuda(cudaFuncSetAttribute(k_filter<MB, PASS, STEPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax),
               "filter shared memory");
    k_filter<MB, PASS, STEPS><<<dim3(blocks, P.slices), kFilterThreads, smem, s>>>(P);
    check_launch("k_filter");
}

// The points' operand image, norms and centre, and room for a batch's queries.
struct Packed {
    Pack pk;
    DevBuf<float> mu, norm, rho;
    DevBuf<uint4> a, b;
    DevBuf<uint32_t> bad;
    const float *centre = nullptr;
    uint32_t n_tiles = 0;
    void alloc(const KnnFilterArgs &A, uint32_t batch, cudaStream_t s)
    {
        pk = pack_of(A.dim);
        n_tiles = ceil_div(A.n, kTileN);
        mu.alloc(A.dim, s);
        norm.alloc(A.n, s);
        rho.alloc(2, s);
        b.alloc((size_t)n_tiles * pk.chunks * (kBBytes / 16), s);
        a.alloc((size_t)(batch / kBlkM) * pk.chunks * (kABytes / 16), s);
        bad.alloc(1, s);
    }
    void points(const KnnFilterArgs &A, cudaStream_t s)
    {
        check_cuda(cudaMemsetAsync(bad.p, 0, sizeof(uint32_t), s), "memset");
        check_cuda(cudaMemsetAsync(rho.p, 0, 2 * sizeof(float), s), "memset");
        if (A.euc) {
            k_filter_centre<<<ceil_div(A.dim, 8), 1024, 0, s>>>(A.x, A.n, A.dim, mu.p);
            centre = mu.p;
        }
        k_filter_norms<<<ceil_div((uint64_t)A.n * 32, 256), 256, 0, s>>>(A.x, A.n, A.dim, centre, pk.terms, norm.p,
                                                                                rho.p, bad.p);
        k_filter_pack<false><<<ceil_div((uint64_t)n_tiles * kTileN * pk.chunks * 8, 256), 256, 0, s>>>(
            A.x, A.n, A.dim, centre, norm.p, nullptr, 0, A.n, n_tiles * kTileN, pk.terms, pk.chunks, A.euc, b.p);
        check_launch("filter packing");
    }
    void queries(const KnnFilterArgs &A, uint32_t q0, uint32_t nq, uint32_t rows, cudaStream_t s)
    {
        k_filter_pack<true><<<ceil_div((uint64_t)rows * pk.chunks * 8, 256), 256, 0, s>>>(
            A.x, A.n, A.dim, centre, norm.p, A.qidx, q0, nq, rows, pk.terms, pk.chunks, A.euc, a.p);
        check_launch("filter packing");
    }
};

// Slices of the points for `blocks` query blocks: fewest rounds of blocks over
// the SMs, a block costing about six tiles besides its own.
uint32_t slices_of(uint32_t blocks, uint32_t tiles)
{
    const uint32_t sms = (uint32_t)device_sm_count();
    uint32_t best = 1;
    uint64_t cost = ~0ull;
    for (uint32_t S = 1; S <= 16 && S <= tiles; S++) {
        const uint64_t c = (uint64_t)ceil_div((uint64_t)blocks * S, sms) * (ceil_div(tiles, S) + 6);
        if (c < cost) {
            cost = c;
            best = S;
        }
    }
    return best;
}

// The most (blocks x slices) of any batch.
uint32_t most_items(uint32_t nq, uint32_t batch, uint32_t rows, uint32_t tiles)
{
    uint32_t most = 1;
    for (uint32_t q0 = 0; q0 < nq; q0 += batch) {
        const uint32_t blocks = ceil_div(std::min(batch, nq - q0), rows);
        most = std::max(most, slices_of(blocks, tiles) * blocks);
    }
    return most;
}

// Shared memory of k_filter<1, 3> behind A and the ring: hi, lo, zone counters.
uint32_t rank_steps(uint32_t k) { return k < 16 ? 4 : 5; }
size_t rank_smem(uint32_t k)
{
    return sizeof(float) * kBlkM * (((size_t)1 << rank_steps(k)) - 1 + k + 1) + sizeof(uint32_t) * 512 * (k + 1);
}
uint32_t rank_stages(uint32_t chunks, uint32_t k)
{
    const size_t fixed = 2048 + (size_t)chunks * kABytes + rank_smem(k);
    return fixed >= kSmemMax ? 0u : (uint32_t)std::min<size_t>(5, (kSmemMax - fixed) / kBBytes);
}

}  // namespace

// The filter prepares all points for whatever number of queries, so it takes
// searches of at least kFilterPairs pairs whose queries are enough to pay for
// that: (500 + 10 dim) sqrt(3 / k) up to 12 000 points, fewer beyond (a tile
// kernel of few queries keeps its SMs busy the longer, the filter's few blocks
// do not), but from 160 + n / 4000 on. (The preparation of n points and the
// tile kernel's work per query are both linear in n; a longer list costs the
// tile kernel more, and lists of one or two so little that it keeps several times
// the queries and pairs.) Below kFilterPoints points the sample is too small for
// its groups, and beyond 191 dims the operands no longer fit beside the ring.
// us, k_knn_tile and the filter, queries chosen from n points on the device:
//   10k x 50, k = 3     256 queries 134, 180   1000 178, 189    2000 265, 205
//   100k x 190, k = 15  256 980, 1241          1000 2430, 1247
//   1M x 50, k = 3      64 633, 1777           256 1689, 1751   512 3099, 1816
// relative to the tile kernel, 2 dims, k = 1: 2600 points 0.77, 4000 0.95, 7000
// 1.46, 2000 queries of 12 000 1.00, of 50 000 1.28; k = 2: 2600 0.99, 4000 1.23;
// and whole calls over all points, k = 15: 2048 points x 2 / 50 / 190 dims 472,
// 306; 514, 354; 628, 569; 4096 points 646, 338; 753, 435; 1120, 786.
bool knn_filter_takes(uint32_t n, uint32_t dim, uint32_t nq, uint32_t k)
{
    constexpr uint32_t kFilterPoints = 2048;
    constexpr uint64_t kFilterPairs = 4u << 20;
    const uint64_t pairs = kFilterPairs * (k < 3 ? 4 - k : 1);
    if (n < kFilterPoints || n >= (1u << 30) || (uint64_t)n * nq < pairs || k + 1 >= kGroups) return false;
    if (dim > 3u * kChunkK || pack_of(dim).chunks > kMaxChunks) return false;
    const double list = std::sqrt(3.0 / k);
    const double few = k == 1 ? 2600.0 + 10.0 * dim : k == 2 ? 1000.0 + 10.0 * dim : list * (500.0 + 10.0 * dim);
    return nq >= few * std::min(1.0, std::sqrt(12000.0 / n)) && nq >= list * std::min(512.0, 160.0 + n / 4000.0);
}

bool knn_filter(const KnnFilterArgs &A, uint32_t *left, uint32_t *n_left, cudaStream_t s)
{
    const Pack pk = pack_of(A.dim);
    const uint32_t C = pk.chunks, MB = C <= 3 ? 2 : 1;
    const uint32_t n_tiles = ceil_div(A.n, kTileN), sms = (uint32_t)device_sm_count();
    const uint32_t stages = std::min<uint32_t>(5, (kSmemMax - 2048 - MB * C * kABytes) / kBBytes);
    const size_t smem = (size_t)MB * C * kABytes + (size_t)stages * kBBytes + 1024;
    // every stride-th tile: the sample's (k + 1)-th group maximum is about its
    // r-th best point, r = -G ln(1 - (k + 1) / G), so about r * stride
    // points of all reach it
    const double r = -(double)kGroups * std::log(1.0 - (double)(A.k + 1) / kGroups);
    const uint32_t stride = std::max(1u, std::min((uint32_t)(kHitTarget / r), n_tiles / 4));
    const bool give_up = 320 * stride >= std::min(A.n / 4, kListCap);
    // queries in batches of at most two waves of blocks (four with one block of
    // queries each): bounds the scratch
    const uint32_t rows = MB * kBlkM, batch = std::min<uint32_t>(ceil_div(A.nq, rows), (MB == 2 ? 2 : 4) * sms) * rows;
    const uint32_t sampled = ceil_div(n_tiles, stride);
    const uint32_t most1 = most_items(A.nq, batch, rows, sampled), most2 = most_items(A.nq, batch, rows, n_tiles);
    const uint32_t per = MB == 2 ? 1 : 2;  // accumulators of a slice
    Packed K;
    DevBuf<float> gmax, least;
    DevBuf<uint32_t> list, count;
    try {
        K.alloc(A, batch, s);
        gmax.alloc((size_t)most1 * per * rows * kGroups, s);
        least.alloc(batch, s);
        // a part's list (a slice's, of one half of the columns) holds its
        // share of kListCap and 64 more
        list.alloc((size_t)most2 * per * 2 * rows * 64 + (size_t)batch * kListCap, s);
        count.alloc((size_t)most2 * per * 2 * rows, s);
    } catch (const Error &e) {
        if (e.status != UMAPCU_CUDA_ALLOC) throw;
        return false;
    }
    K.points(A, s);
    for (uint32_t q0 = 0; q0 < A.nq; q0 += batch) {
        const uint32_t nq = std::min(batch, A.nq - q0), blocks = ceil_div(nq, rows);
        K.queries(A, q0, nq, blocks * rows, s);
        FilterArgs P{};
        P.a = K.a.p;
        P.b = K.b.p;
        P.nq = nq;
        P.n_tiles = n_tiles;
        P.chunks = C;
        P.steps = pk.steps;
        P.stages = stages;
        P.bad = K.bad.p;
        P.stride = stride;
        P.slices = slices_of(blocks, sampled);
        P.gmax = gmax.p;
        if (MB == 2) launch_filter<2, 1>(P, blocks, smem, s);
        else launch_filter<1, 1>(P, blocks, smem, s);
        k_filter_threshold<<<ceil_div((uint64_t)nq * 32, 256), 256, 0, s>>>(
            gmax.p, P.slices * per, nq, A.k, K.norm.p, A.qidx, q0, A.dim, A.euc, K.rho.p, pk.steps, give_up, least.p);
        check_launch("k_filter_threshold");
        P.stride = 1;
        P.slices = slices_of(blocks, n_tiles);
        P.least = least.p;
        P.list = list.p;
        P.count = count.p;
        const uint32_t parts = P.slices * per * 2;
        P.cap = kListCap / parts + 64;
        if (MB == 2) launch_filter<2, 2>(P, blocks, smem, s);
        else launch_filter<1, 2>(P, blocks, smem, s);
        const unsigned rg = ceil_div(nq, kRefineWarps);
        if (A.euc)
            k_refine<true><<<rg, kRefineWarps * 32, 0, s>>>(A.x, A.n, A.dim, A.k, A.qidx, q0, nq, list.p, count.p, parts,
                                                            P.cap, K.bad.p, A.out_idx, A.out_dist, left, n_left);
        else
            k_refine<false><<<rg, kRefineWarps * 32, 0, s>>>(A.x, A.n, A.dim, A.k, A.qidx, q0, nq, list.p, count.p, parts,
                                                             P.cap, K.bad.p, A.out_idx, A.out_dist, left, n_left);
        check_launch("k_refine");
    }
    return true;
}

bool rank_filter_takes(uint32_t n, uint32_t dim, uint32_t nq, uint32_t k)
{
    return knn_filter_takes(n, dim, nq, k) && k < 32 && rank_stages(pack_of(dim).chunks, k) >= 2;
}

bool rank_filter(const KnnFilterArgs &A, const float *thr_d, const uint32_t *thr_j, uint32_t *counts, uint32_t *left,
                 uint32_t *n_left, cudaStream_t s)
{
    const Pack pk = pack_of(A.dim);
    const uint32_t C = pk.chunks, n_tiles = ceil_div(A.n, kTileN), stages = rank_stages(C, A.k);
    const size_t smem = (size_t)C * kABytes + (size_t)stages * kBBytes + rank_smem(A.k) + 1024;
    // at most 16 384 queries at a time: a query's lists hold 4096 points and 64
    // more a part
    constexpr uint32_t kRankCap = 4096;
    const uint32_t batch = std::min<uint32_t>(ceil_div(A.nq, kBlkM), 128) * kBlkM;
    const uint32_t most = most_items(A.nq, batch, kBlkM, n_tiles);
    Packed K;
    DevBuf<float> hi, lo;
    DevBuf<uint32_t> given, zones, list, count;
    try {
        K.alloc(A, batch, s);
        hi.alloc((size_t)batch * A.k, s);
        lo.alloc((size_t)batch * A.k, s);
        given.alloc((size_t)batch * A.k, s);
        zones.alloc((size_t)batch * 32, s);
        list.alloc((size_t)most * 4 * kBlkM * 64 + (size_t)batch * kRankCap, s);
        count.alloc((size_t)most * 4 * kBlkM, s);
    } catch (const Error &e) {
        if (e.status != UMAPCU_CUDA_ALLOC) throw;
        return false;
    }
    K.points(A, s);
    for (uint32_t q0 = 0; q0 < A.nq; q0 += batch) {
        const uint32_t nq = std::min(batch, A.nq - q0), blocks = ceil_div(nq, kBlkM);
        K.queries(A, q0, nq, blocks * kBlkM, s);
        k_rank_bounds<<<ceil_div((uint64_t)nq * 32, 256), 256, 0, s>>>(thr_d, thr_j, nq, A.k, K.norm.p, A.qidx, q0, A.dim,
                                                                       A.euc, K.rho.p, pk.steps, hi.p, lo.p, given.p,
                                                                       K.bad.p);
        check_launch("k_rank_bounds");
        check_cuda(cudaMemsetAsync(zones.p, 0, sizeof(uint32_t) * 32 * nq, s), "memset");
        FilterArgs P{};
        P.a = K.a.p;
        P.b = K.b.p;
        P.nq = nq;
        P.n_tiles = n_tiles;
        P.chunks = C;
        P.steps = pk.steps;
        P.stages = stages;
        P.bad = K.bad.p;
        P.stride = 1;
        P.slices = slices_of(blocks, n_tiles);
        P.list = list.p;
        P.count = count.p;
        P.k = A.k;
        P.zone_rows = (1u << rank_steps(A.k)) - 1;
        P.hi = hi.p;
        P.lo = lo.p;
        P.qidx = A.qidx;
        P.q0 = q0;
        P.zones = zones.p;
        const uint32_t parts = P.slices * 4;
        P.cap = kRankCap / parts + 64;
        if (rank_steps(A.k) == 4) launch_filter<1, 3, 4>(P, blocks, smem, s);
        else launch_filter<1, 3, 5>(P, blocks, smem, s);
        const unsigned rg = ceil_div(nq, kRefineWarps);
        if (A.euc)
            k_rank_refine<true><<<rg, kRefineWarps * 32, 0, s>>>(A.x, A.n, A.dim, A.k, A.qidx, q0, nq, thr_d, thr_j, given.p,
                                                                 zones.p, list.p, count.p, parts, P.cap, K.bad.p, counts,
                                                                 left, n_left);
        else
            k_rank_refine<false><<<rg, kRefineWarps * 32, 0, s>>>(A.x, A.n, A.dim, A.k, A.qidx, q0, nq, thr_d, thr_j, given.p,
                                                                  zones.p, list.p, count.p, parts, P.cap, K.bad.p, counts,
                                                                  left, n_left);
        check_launch("k_rank_refine");
    }
    return true;
}

}  // namespace umapcu
