// b200_qmm for more than 32 rows of x (qmm_many.cu), as seen by qmm.cu.
#pragma once
#include "common.cuh"

namespace b200 {
// The tensor-core GEMM on weights widened on their way in, or on panels of dequantised ones.  The parameters have passed
// b200_qmm_validate.
b200_status QmmManyRows(b200_context* ctx, cudaStream_t stream, const b200_qmm_params* p);
}  // namespace b200
