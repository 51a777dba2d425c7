// Tensor-core candidate filter of the exact kNN search (knn_filter.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace umapcu {

struct KnnFilterArgs {
    const float *x;         // [n, dim] points (cosine: unit rows)
    uint32_t n, dim, k;
    bool euc;
    const uint32_t *qidx;   // [nq] query rows, nullptr: query q is row q
    uint32_t nq;
    uint32_t *out_idx;      // [nq][k]
    float *out_dist;
};

// Whether the filter takes a search of this size (the rule's reasons stand at
// its definition).
bool knn_filter_takes(uint32_t n, uint32_t dim, uint32_t nq, uint32_t k);

// The k nearest of every query, bit for bit what the tile kernel finds.
// Queries the filter could not settle (more candidates than its lists hold,
// non-finite or huge data) are appended to left [nq] with *n_left counting
// them, both on the device; their outputs are not written. false: not enough
// device memory for its scratch, nothing was done.
bool knn_filter(const KnnFilterArgs &A, uint32_t *left, uint32_t *n_left, cudaStream_t s);

// The same for ranks: counts [nq][k] = points strictly before each threshold
// (thr_d, thr_j) [nq][k] of the query by (distance, index), itself excluded
// (A.out_idx and A.out_dist are not used). Counts of queries in left are not
// written.
bool rank_filter_takes(uint32_t n, uint32_t dim, uint32_t nq, uint32_t k);
bool rank_filter(const KnnFilterArgs &A, const float *thr_d, const uint32_t *thr_j, uint32_t *counts, uint32_t *left,
                 uint32_t *n_left, cudaStream_t s);

}  // namespace umapcu
