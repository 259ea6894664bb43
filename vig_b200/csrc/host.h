// Host side of the package in C++: torch tensors in, calls of the C ABI (include/vig_b200.h) out.  The kernels' library is
// opened by path (the one the ctypes binding uses), so both bindings share one copy of it.
#pragma once
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cmath>
#include "../../include/vig_b200.h"

namespace vig_host {

using at::Tensor;
namespace py = pybind11;

#define VIG_HOST_API(X)                                                                                                     \
    X(vig_strerror) X(vig_bigla_fwd) X(vig_bigla_workspace_bytes) X(vig_bigla_bwd_full) X(vig_bigla_bwd_full_workspace_bytes) \
    X(vig_dwconv3x3_fwd) X(vig_gate_inject_fwd) X(vig_add_rmsnorm_fwd) X(vig_layernorm_act_fwd) X(vig_layernorm_act_add_fwd)  \
    X(vig_layernorm_act_add_rmsnorm_fwd) X(vig_linear_swiglu_fwd) X(vig_linear_swiglu_preferred) X(vig_linear_add_rmsnorm_fwd) X(vig_linear_add_rmsnorm_preferred) \
    X(vig_stem_fold_fwd) X(vig_stem_unfold_fwd) X(vig_stem_conv_ln_fwd)                   \
    X(vig_stem_conv_ln_supported) X(vig_swiglu_fwd) X(vig_add_layernorm_fwd) X(vig_chain_launches) X(vig_token_mean_fwd) X(vig_embed_conv_ln_fwd) X(vig_linear_pair_preferred) X(vig_linear_pair_fwd) X(vig_conv_proj_preferred) X(vig_conv_proj_fwd) X(vig_block_tail_preferred) X(vig_block_tail_fwd)
struct Api {
#define X(name) decltype(&::name) name = nullptr;
    VIG_HOST_API(X)
#undef X
};
extern Api api;

inline void ok(int status, const char* what) {
    if (status != 0) throw std::runtime_error(std::string(what) + " failed with status " + std::to_string(status) + ": " + api.vig_strerror(status));
}
inline int dtype_code(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return VIG_DTYPE_F32;
        case at::kBFloat16: return VIG_DTYPE_BF16;
        case at::kHalf: return VIG_DTYPE_F16;
        default: return -1;
    }
}
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline void* stream() { return at::cuda::getCurrentCUDAStream().stream(); }
// the device's error word, registered by the Python layer; NULL before that
int32_t* status_ptr(int device);
bool status_known(int device);

struct S3 {                                   // (b, h, l) element strides of a [B,H,L,d] view
    int64_t s[3];
    explicit S3(const Tensor& t) { if (t.defined()) { s[0] = t.stride(0); s[1] = t.stride(1); s[2] = t.stride(2); } }
};

// bi_gla on checked tensors; undefined tensors = absent.  The workspace comes from the caching allocator on every call: it is
// ordered with the stream's other work and given back at once.
void bi_gla_into(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gf, const Tensor& gb, const Tensor& o, double scale, double out_scale,
                 double norm, double clamp, const Tensor& init_f, const Tensor& init_b, const Tensor& final_f, const Tensor& final_b, int dir_mask, int impl);

void bind_model(py::module_& m);

}  // namespace vig_host
