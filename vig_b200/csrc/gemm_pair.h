// GEMMs on pairs of CTAs (gemm_pair.cu, gemm_pair_norm.cu), for the dispatch of the entry points.  Arguments checked by the caller; K % 64 == 0.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vig {

int pair_swiglu_launch(const void* x, int64_t ldx, const void* w, void* out, int64_t ldo, int64_t M, int K, int I, int dtype, int32_t* status, cudaStream_t stream);
// x W^T + bias (may be null); N % 8 == 0
int pair_linear_launch(const void* x, int64_t ldx, const void* w, const void* bias, void* out, int64_t ldo, int64_t M, int K, int N, int dtype, int32_t* status, cudaStream_t stream);
// rows of 256, 384 or 768 values
int pair_norm_launch(const void* x, int64_t ldx, const void* w, const void* residual, const void* norm_w, void* out_r, void* out_h, int64_t M, int K, int N, float eps,
                     int dtype, int32_t* status, cudaStream_t stream);
// tiles of 256 rows that the GPU works on at a time
int pair_norm_clusters(int N, int dtype);

}  // namespace vig
