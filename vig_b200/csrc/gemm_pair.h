// GEMMs on pairs of CTAs (gemm_pair.cu), for the dispatch of the entry points.  Arguments checked by the caller; K % 64 == 0.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vig {

int pair_swiglu_launch(const void* x, int64_t ldx, const void* w, void* out, int64_t ldo, int64_t M, int K, int I, int dtype, int32_t* status, cudaStream_t stream);

}  // namespace vig
