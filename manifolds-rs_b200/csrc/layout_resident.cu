// Small layouts: many epochs in one launch.
//
// A problem of a few hundred 32-node segments is bound by latency, not by
// work: one launch per epoch pays for the launch, for every block reading its
// segment again and for the chain bit words -> active entries -> other
// endpoints -> coordinates each time (8.2 us an epoch at 10k points, k = 15,
// of which the gathers need about one). Here every segment owns a block for
// the whole run, launched cooperatively so that all blocks are resident, and
// the blocks follow one another through the coordinates themselves:
//  * a node's row is one 16-byte word {coordinates, epoch tag}, stored and
//    loaded whole; a gather repeats until the row carries the epoch it needs,
//    so there is no barrier between epochs and a row's way from the node that
//    writes it to the entry that reads it is a store and a load through L2 (a
//    grid-wide counter between epochs -- fence, counter, poll and only then the
//    gathers -- made 4.2 us an epoch at 1k points where this takes 3.7 with the
//    call's 0.45 ms of preparation in it);
//  * rows stand in a ring of kRing epochs; a block overwrites one only when
//    the counter of that epoch shows that all blocks have left it, which they
//    have long done when it is looked at;
//  * positions, moments, row starts and other endpoints of the segment stay
//    in registers and shared memory;
//  * while warp 0 steps the nodes of one epoch, other warps form the batches
//    of the next (bit words, ranks, other endpoints, negatives depend on the
//    schedule and the hash only).
// The batches, their order and every sum are those of k_epoch_split_bits
// (epoch_segment_split_bits), so the result is bit-identical to it. What is
// left is one warp's chain of dependent instructions (gather, terms, segmented
// sum, node sums, Adam): about 4000 cycles an epoch.
// Measured (whole one-shot calls, Adam, k = 15), launches per epoch -> here:
// 500 epochs 1k points 3.68 -> 1.87 ms, 5k 4.24 -> 2.4, 10k 4.78 -> 2.76; 200
// epochs 14k points 2.36 -> 1.68, 18k 2.58 -> 1.80.
#include "epoch_device.cuh"

namespace umapcu {
namespace {

// Seconds-long bound of every wait, in clock cycles.
constexpr long long kWaitLimit = 4000000000ll;
constexpr uint32_t kRing = 8;
// Entries of a segment whose other endpoint and node (as index in the segment
// << 27 | offset in the row) are kept in shared memory (8 bytes each); those of
// a longer segment past them are looked up each time.
constexpr uint32_t kEntries = 1024;

using Word = unsigned __int128;

__device__ __forceinline__ Word load_word(const uint4 *p)
{
    Word v;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint32_t load_counter(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Barrier `id` of THREADS threads (whole warps).
template <int THREADS>
__device__ __forceinline__ void group_sync(uint32_t id)
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}

template <int D>
__device__ __forceinline__ void store_tagged(uint4 *p, const float (&y)[D], uint32_t tag)
{
    Word v = (Word)tag << 96;
#pragma unroll
    for (int d = 0; d < D; d++) v |= (Word)__float_as_uint(y[d]) << (32 * d);
    asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(v) : "memory");
}

template <int D>
__device__ __forceinline__ bool unpack(Word v, uint32_t tag, float (&y)[D])
{
#pragma unroll
    for (int d = 0; d < D; d++) y[d] = __uint_as_float((uint32_t)(v >> (32 * d)));
    return (uint32_t)(v >> 96) == tag;
}

// The rows of an entry once all carry `tag`; gives up, with *stop set, after
// the limit or when *stop is set already.
template <int D, int NR>
__device__ __forceinline__ void gather(const uint4 *slot, uint32_t tag, uint32_t o, BatchRows<D, NR> &R,
                                       volatile bool *stop, uint32_t *status)
{
    long long t0 = 0;
    uint32_t missing = (2u << NR) - 1u;  // rows not there yet: only these are loaded again
    for (;;) {
        Word w[NR + 1];
#pragma unroll
        for (int t = 0; t <= NR; t++)
            if ((missing >> t) & 1u) w[t] = load_word(slot + (t == 0 ? o : R.kk[t - 1]));
#pragma unroll
        for (int t = 0; t <= NR; t++)
            if ((missing >> t) & 1u) {
                if (unpack<D>(w[t], tag, t == 0 ? R.yo : R.yk[t - 1])) missing &= ~(1u << t);
            }
        if (!missing || *stop) return;
        const long long now = clock64();
        if (!t0) t0 = now;
        if (now - t0 > kWaitLimit) {
            atomicCAS(status, 0u, (uint32_t)UMAPCU_TIMEOUT);
            *stop = true;
            return;
        }
    }
}

// *status set to UMAPCU_CAPACITY when a segment has more bit words than a
// block holds.
__global__ void k_resident_fits(const uint32_t *__restrict__ offsets, uint32_t n, uint32_t *__restrict__ status)
{
    const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) * 32u;
    if (b >= n) return;
    const uint32_t lo = offsets[b], hi = offsets[min(b + 32u, n)];
    if (hi > lo && ((hi - 1) >> 5) - (lo >> 5) + 1 > kSplitWords) *status = (uint32_t)UMAPCU_CAPACITY;
}

// NG groups of G warps take the epochs in turn (a group forms its next epoch's
// batches while another group's epoch runs), warp 0 steps the nodes after each.
template <int D, int NG, int G, int MIN_BLOCKS>
__global__ void __launch_bounds__(32 * (NG * G + 1), MIN_BLOCKS)
    k_layout_resident(const EpochArgs A, const float4 *__restrict__ scal, uint32_t first, uint32_t count, uint64_t words,
                      uint4 *ring, uint32_t *counter, uint32_t *status)
{
    constexpr int NR = 5;
    constexpr uint32_t kThreads = 32 * (NG * G + 1), kRound = 32 * G;
    struct Seg {
        uint32_t beg[33];
        float ys[32][D];
    };
    __shared__ Seg S;
    __shared__ float part[NG][G][32][D];
    __shared__ unsigned has_w[NG][G];
    __shared__ uint32_t words_of[NG][kSplitWords], before[NG][G][kSplitWords], active_of[NG];
    __shared__ uint2 entries[kEntries];
    __shared__ volatile bool stop;
    if (*status) return;  // an earlier span gave up
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t node0 = blockIdx.x * 32u, node = node0 + lane;
    const uint32_t n = A.n;
    const bool valid = node < n;
    uint32_t sbeg = A.offsets[node0], send = A.offsets[min(node0 + 32u, n)];
#ifdef UMAPCU_CHECKED
    if (!checked_ok(sbeg <= send && send <= A.n_entries, A.err)) sbeg = send = 0;
#endif
    const uint32_t w0 = sbeg >> 5, nw = send > sbeg ? ((send - 1) >> 5) - w0 + 1 : 0;
    float ys[D], m[D], v[D];
#pragma unroll
    for (int d = 0; d < D; d++) ys[d] = m[d] = v[d] = 0.0f;
    if (warp == 0) {
        load_segment<D, false, kShared>(A, S, node0, lane, ys);
        if (valid) {
            load_row<D, kShared>(A.m, node, m);
            load_row<D, kShared>(A.v, node, v);
            store_tagged<D>(ring + node, ys, 1u);
        }
    }
    if (threadIdx.x == 0) stop = false;
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < min(send - sbeg, kEntries); t += kThreads) {
        const uint32_t at = local_node(S.beg, sbeg + t);
        entries[t] = make_uint2(__ldcs(A.other + sbeg + t), (at << kRecNodeShift) | (sbeg + t - S.beg[at]));
    }
    __syncthreads();

    if (warp == 0) {
        for (uint32_t i = 0; i < count; i++) {
            const uint32_t grp = i % NG;
            const float4 sc = scal[i];
            // blocks that have left the epoch whose ring slot this step reuses
            uint32_t left = 0;
            if (i >= kRing - 1 && lane == 0) left = load_counter(counter + (i + 1 - kRing));
            float g[D];
#pragma unroll
            for (int d = 0; d < D; d++) g[d] = 0.0f;
            bool act = false;
            for (uint32_t r0 = 0;; r0 += kRound) {
                group_sync<32 * G + 32>(1 + NG + grp);
                const uint32_t total = active_of[grp];
                const int batches = (int)min((uint32_t)G, (total - r0 + 31u) / 32u);
#pragma unroll 4
                for (int w = 0; w < batches; w++) {
                    if ((has_w[grp][w] >> lane) & 1u) {
                        act = true;
#pragma unroll
                        for (int d = 0; d < D; d++) g[d] += part[grp][w][lane][d];
                    }
                }
                if (r0 + kRound >= total) break;
                group_sync<32 * G + 32>(1 + NG + grp);
            }
            // all of this block's reads of the epoch's rows are done
            if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter + i) : "memory");
            if (act) {
                if (A.optimiser == UMAPCU_OPT_SGD) {
#pragma unroll
                    for (int d = 0; d < D; d++) ys[d] = ys[d] + sc.z * g[d];
                } else {
#pragma unroll
                    for (int d = 0; d < D; d++)
                        ys[d] = adam_coord(g[d], m[d], v[d], ys[d], sc.x, sc.y, A.omb1, A.omb2);
                }
            }
            if (i + 1 == count) break;
            if (i >= kRing - 1) {
                if (lane == 0 && left != gridDim.x) {
                    const long long t0 = clock64();
                    while (!stop && load_counter(counter + (i + 1 - kRing)) != gridDim.x) {
                        if (clock64() - t0 > kWaitLimit) {
                            atomicCAS(status, 0u, (uint32_t)UMAPCU_TIMEOUT);
                            stop = true;
                        }
                    }
                }
                __syncwarp();
            }
            if (valid) store_tagged<D>(ring + (size_t)((i + 1) % kRing) * n + node, ys, i + 2);
#pragma unroll
            for (int d = 0; d < D; d++) S.ys[lane][d] = ys[d];
            group_sync<32 * G + 32>(1 + 2 * NG + (i + 1) % NG);
        }
        if (valid) {
            store_row<D>((count & 1) ? A.y_next : const_cast<float *>(A.y_cur), node, ys);
            if (A.optimiser != UMAPCU_OPT_SGD) {
                store_row<D>(A.m, node, m);
                store_row<D>(A.v, node, v);
            }
        }
        return;
    }

    const uint32_t grp = (uint32_t)(warp - 1) / G, mine = (uint32_t)(warp - 1) % G, gt = mine * 32u + lane;
    uint32_t(&wm)[kSplitWords] = words_of[grp];
    uint32_t(&pre)[kSplitWords] = before[grp][mine];
    uint32_t o = 0, j = 0, el = 0;
    BatchRows<D, NR> R;
    // The active entry of rank r and its negatives in epoch first + i.
    auto entry = [&](uint32_t r, uint32_t i) {
        uint32_t lo = 0, hi = nw;  // last word with pre <= r
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (pre[mid] <= r) lo = mid;
            else hi = mid;
        }
        const uint32_t p = (w0 + lo) * 32u + select_bit(wm[lo], r - pre[lo]);
        if (p - sbeg < kEntries) {
            const uint2 e = entries[p - sbeg];
            o = e.x;
            j = e.y >> kRecNodeShift;
            el = e.y & kRecOffsetMask;
        } else {
            o = __ldg(A.other + p);
            j = local_node(S.beg, p);
            el = p - S.beg[j];
        }
        if (!checked_ok(o < n, A.err)) o = node0;
#pragma unroll
        for (int t = 0; t < NR; t++)
            R.kk[t] = fastmod_u32(hash_neg_raw(A.seed32, node0 + j, first + i, el, (uint32_t)t), A.fastmod_M, n);
    };
    // epoch words, loaded an epoch of the group ahead and masked when used
    auto load = [&](uint32_t i, uint32_t t) { return __ldcs(A.bits + (uint64_t)(first + i) * words + w0 + t); };
    auto masked = [&](uint32_t x, uint32_t t) {
        const uint32_t wi = w0 + t;
        if (wi * 32u < sbeg) x &= ~0u << (sbeg - wi * 32u);
        if (wi * 32u + 32u > send) x &= (send - wi * 32u >= 32u) ? ~0u : ((1u << (send - wi * 32u)) - 1u);
        return x;
    };
    uint32_t ahead = 0;
    if (gt < nw && grp < count) ahead = load(grp, gt);
    for (uint32_t i = grp; i < count; i += NG) {
        if (gt < nw) wm[gt] = masked(ahead, gt);
        for (uint32_t u = gt + kRound; u < nw; u += kRound) wm[u] = masked(load(i, u), u);
        group_sync<32 * G>(1 + grp);
        if (gt < nw && i + NG < count) ahead = load(i + NG, gt);
        // the counts of active entries before each word, a copy per warp
        uint32_t total = 0;
        for (uint32_t t0 = 0; t0 < nw; t0 += 32) {
            const uint32_t t = t0 + lane;
            const uint32_t c = t < nw ? __popc(wm[t]) : 0u;
            uint32_t x = c;
#pragma unroll
            for (int f = 1; f < 32; f <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, x, f);
                if (lane >= f) x += y;
            }
            if (t < nw) pre[t] = total + x - c;
            total += __shfl_sync(kFull, x, 31);
        }
        __syncwarp();
        if (32u * mine + lane < total) entry(32u * mine + lane, i);
        // gathers start when this block has stepped its own nodes: before that
        // they would only load L2 (10k points with gathers started at once: 10 ms)
        if (i) group_sync<32 * G + 32>(1 + 2 * NG + grp);
        for (uint32_t r0 = 0;; r0 += kRound) {
            const uint32_t rb = r0 + 32u * mine;
            if (rb < total) {  // warp-uniform
                const bool live = rb + lane < total;
                if (r0 && live) entry(rb + lane, i);
                if (live) gather<D, NR>(ring + (size_t)(i % kRing) * n, i + 1, o, R, &stop, status);
                __syncwarp();
                float gd[D];
                bool ad = false;
                // (the rows came after warp 0 had read the group's last sums)
                const unsigned has = process_batch<D, false, NR, kShared, kU, true, true, true>(
                    A, S, live, 0u, o, j, el, node0, lane, gd, ad, nullptr, part[grp][mine], &R);
                if (lane == 0) has_w[grp][mine] = has;
            }
            if (r0 == 0 && gt == 0) active_of[grp] = total;
            group_sync<32 * G + 32>(1 + NG + grp);
            if (r0 + kRound >= total) break;
            group_sync<32 * G + 32>(1 + NG + grp);
        }
    }
}

template <int D, int NG, int G, int MIN_BLOCKS>
bool try_launch(const EpochArgs &A, const float4 *scal, uint32_t first, uint32_t count, uint64_t words, uint4 *ring,
                uint32_t *counter, uint32_t *status, cudaStream_t s)
{
    const auto kernel = k_layout_resident<D, NG, G, MIN_BLOCKS>;
    const uint32_t nseg = ceil_div(A.n, 32), threads = 32 * (NG * G + 1);
    int per_sm = 0;
    check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0), "occupancy");
    if ((uint64_t)per_sm * device_sm_count() < nseg) return false;
    check_cuda(cudaMemsetAsync(counter, 0, sizeof(uint32_t) * count, s), "memset counter");
    check_cuda(cudaMemsetAsync(ring, 0, resident_ring_bytes(A.n), s), "memset ring");  // no row carries a tag yet
    EpochArgs a = A;
    void *args[] = {&a, &scal, &first, &count, &words, &ring, &counter, &status};
    const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(nseg), dim3(threads), args, 0, s);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        cudaGetLastError();
        return false;
    }
    check_cuda(e, "k_layout_resident");
    return true;
}

// The form by the blocks an SM has to hold. Up to two: two groups, so that a
// group's batches are formed during the other's epoch (1k points 2.06 -> 1.87
// ms). Three or four: registers leave nine or seven warps, and a group of half
// of them would need a second round of batches in most epochs (10k points 3.8
// ms with two groups of four, 2.76 with one of nine). Eight blocks of three
// warps are slower than launches (25k points 3.36 ms, launches 3.25).
template <int D>
bool launch_form(const EpochArgs &A, const float4 *scal, uint32_t first, uint32_t count, uint64_t words, uint4 *ring,
                 uint32_t *counter, uint32_t *status, cudaStream_t s)
{
    const uint32_t nseg = ceil_div(A.n, 32), sms = (uint32_t)device_sm_count();
    if (nseg <= sms && try_launch<D, 2, 8, 1>(A, scal, first, count, words, ring, counter, status, s)) return true;
    if (nseg <= 2 * sms && try_launch<D, 2, 7, 2>(A, scal, first, count, words, ring, counter, status, s)) return true;
    if (nseg <= 3 * sms && try_launch<D, 1, 9, 3>(A, scal, first, count, words, ring, counter, status, s)) return true;
    return try_launch<D, 1, 7, 4>(A, scal, first, count, words, ring, counter, status, s);
}

}  // namespace

size_t resident_ring_bytes(uint32_t n) { return (size_t)kRing * n * sizeof(uint4); }

bool resident_takes(uint32_t n, uint32_t n_dim)
{
    return (n_dim == 2 || n_dim == 3) && ceil_div(n, 32) <= kResidentSegments;
}

void launch_resident_fits(const uint32_t *offsets, uint32_t n, uint32_t *status, cudaStream_t s)
{
    k_resident_fits<<<ceil_div(ceil_div(n, 32), 256), 256, 0, s>>>(offsets, n, status);
    check_launch("k_resident_fits");
}

bool launch_layout_resident(const EpochArgs &A, uint32_t n_dim, const float4 *scal, uint32_t first, uint32_t count,
                            uint64_t words, uint4 *ring, uint32_t *counter, uint32_t *status, cudaStream_t s)
{
    return n_dim == 2 ? launch_form<2>(A, scal, first, count, words, ring, counter, status, s)
                      : launch_form<3>(A, scal, first, count, words, ring, counter, status, s);
}

}  // namespace umapcu
