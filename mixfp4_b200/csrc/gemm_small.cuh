// Entry of the tensor-core kernel for a few dozen tokens (gemm_small.cu).
#pragma once

#include "common.cuh"

namespace mixfp4 {

constexpr int kSmallMaxTokens = 128;
constexpr int kSmallMaxGrouped = 64;     // several weights in one launch: beyond it one chain per tile would be longer than apart

struct SmallPlan {
    int cluster, nclusters;        // CTAs per cluster, clusters
    int flush;                     // units after which a piece's accumulators are flushed, 0: never (17 tokens and more)
};
// clusters[c] (c = 1..8): how many clusters of c CTAs run at once.
SmallPlan plan_small(int ntiles, int units, int np, int64_t chain_limit, const int* clusters);
// gemm.cu: products in one accumulator of the 128-row tiles (which cut K over up to eight CTAs) for these sizes.
int64_t gemm_tile_chain(int64_t m, int64_t n, int64_t k);

// y_i = x * W_i^T for up to three stream-layout (or kernel-layout) weights that share x, 1 <= m <= 128 (64 for several weights); x with 16-byte aligned rows
// (else MIXFP4_E_ALIGN).  The segments' pointers and alignment are checked by the caller.  dependent: launch as
// a programmatic dependent of the kernel before (only x may come from it).  chain_limit: products that one tensor-core
// accumulator may sum, a multiple of 128 (up to 16 rows of x it is 256 at most).  wait_ns: limit of the bounded waits (the
// kernel before, whose end a dependent launch waits for, does not count).
int gemm_small(const void* x, int64_t m, int64_t ldx, int64_t k, const mixfp4_gemv_segment* segments, int count,
               bool stream_layout, int out_dtype, int64_t chain_limit, uint64_t wait_ns, bool dependent, int* status,
               cudaStream_t st);

}  // namespace mixfp4
