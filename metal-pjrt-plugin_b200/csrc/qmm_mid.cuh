// The quantised matmul for 9 to 32 rows of x (qmm_mid.cu), as seen by qmm.cu.
#pragma once
#include "tp.cuh"

namespace b200 {
// Enqueues it (the parameters have passed b200_qmm_validate, 9 <= M <= 32).  B200_RESOURCE_EXHAUSTED: nothing was enqueued,
// the caller's scratch is too small or the pool has none.
b200_status QmmMidRun(b200_context* ctx, cudaStream_t stream, const b200_qmm_params* p, const QmmCaller& caller);
// Floats of scratch it takes for M rows (0: one slice of K, or no plan).
size_t QmmMidScratchFloats(const b200_context* ctx, int bits, int group, int64_t M, int64_t N, int64_t K);
// Rows of a tile, slices of K and batch blocks that it would use.
b200_status QmmMidPlan(const b200_qmm_params* p, int sm_count, int max_smem, int* rows, int* slices, int* mb);
}  // namespace b200
