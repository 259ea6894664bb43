// out[M, N] = x W^T + bias on pairs of CTAs (gemm_pair.cu): the stacked input projection of a block (bf16 / fp16).  One GEMM produces
// [q | k | v | output-gate logits | gate logits] per token (qkv_proj, g_proj and the folded gk_proj of GatedLinearAttention,
// classification/models/vig.py:283-290 and 431-439).
#include "tc_common.cuh"
#include "gemm_pair.h"

using namespace vig;

static bool lb_shape(int64_t M, int K, int N, int dtype) {
    return (dtype == VIG_DTYPE_BF16 || dtype == VIG_DTYPE_F16) && M > 0 && K > 0 && N > 0 && K % 64 == 0 && N % 8 == 0 && M < (1ll << 31);
}

static int lb_launch(const void* x, int64_t ldx, const void* w, const void* bias, void* out, int64_t ldo, int64_t M, int K, int N, int dtype, int32_t* status, void* stream) {
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(bias)) & 15) return VIG_ERR_ALIGN;
    if (ldx < K || ldo < N || (ldx * 2) % 16 || (ldo * 2) % 16) return VIG_ERR_ARG;
    return pair_linear_launch(x, ldx, w, bias, out, ldo, M, K, N, dtype, status, (cudaStream_t)stream);
}

// K a multiple of 64 up to 192, N a multiple of 8, and enough rows to give every SM 256 of them.
extern "C" int vig_linear_bias_supported(int64_t M, int K, int N, int dtype) {
    return lb_shape(M, K, N, dtype) && K <= 192 && M >= 256 * (int64_t)device_sms() && tc::encode_fn() != nullptr;
}

extern "C" int vig_linear_bias_fwd(const void* x, int64_t ldx, const void* w, const void* bias, void* out, int64_t ldo,
                                   int64_t M, int K, int N, int dtype, int32_t* status_dev, void* stream) {
    if (!x || !w || !out) return VIG_ERR_NULL;
    if (M == 0) return VIG_OK;
    if (!vig_linear_bias_supported(M, K, N, dtype) || (N + 191) / 192 > device_sms()) return VIG_ERR_SHAPE;
    return lb_launch(x, ldx, w, bias, out, ldo, M, K, N, dtype, status_dev, stream);
}

// Against the library's GEMM by how many rounds the tiles of 256 x 256 make on the pairs; us here / there, rounds: 25088 x 384 x 2304 (11.9) 43.5 / 46.2, x 1536 (7.9) 32.0 / 33.0,
// 262144 x 192 x 1152 (69) 148 / 154 - 180, 262144 x 192 x 768 (42) 95 / 135, 50176 x 192 x 768 (7.9) 23.4 / 25.7, 32768 x 384 x 2304 (15.6) 55.5 / 61,
// but 12544 x 384 x 1536 (4.0) 21.0 / 19.6, 12544 x 192 x 768 (2.0) 12.8 / 11.9.  The library's tiles are smaller and its epilogue shorter where there are few of
// them; behind that, x and W of a tile come in once for two SMs.  At K = 768 the power cap decides: 131072 x 768 x 4608 750 / 880 by itself, but ViG-B forwards
// of 131072 and 50000 tokens took 0.2 - 0.7 % longer with it.
extern "C" int vig_linear_pair_preferred(int64_t M, int K, int N, int dtype) {
    return lb_shape(M, K, N, dtype) && K <= 384 && (M + 255) / 256 * ((N + 255) / 256) >= 7 * (int64_t)(device_sms() / 2) && tc::encode_fn() != nullptr;
}

extern "C" int vig_linear_pair_fwd(const void* x, int64_t ldx, const void* w, const void* bias, void* out, int64_t ldo,
                                   int64_t M, int K, int N, int dtype, int32_t* status_dev, void* stream) {
    if (!x || !w || !out) return VIG_ERR_NULL;
    if (M == 0) return VIG_OK;
    if (!lb_shape(M, K, N, dtype)) return VIG_ERR_SHAPE;
    if (!tc::encode_fn()) return VIG_ERR_DEVICE;
    return lb_launch(x, ldx, w, bias, out, ldo, M, K, N, dtype, status_dev, stream);
}
