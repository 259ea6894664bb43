// Shared helpers for the vig_b200 kernels: dtype traits, 16-byte vector access, parameter block.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <atomic>
#include "../../include/vig_b200.h"

namespace vig {

template <typename T> struct DType;
template <> struct DType<float> {
    static constexpr int VEC = 4;
    __device__ static float to_f(float x) { return x; }
    __device__ static float from_f(float x) { return x; }
};
template <> struct DType<__nv_bfloat16> {
    static constexpr int VEC = 8;
    __device__ static float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
    __device__ static __nv_bfloat16 from_f(float x) { return __float2bfloat16_rn(x); }
};
template <> struct DType<__half> {
    static constexpr int VEC = 8;
    __device__ static float to_f(__half x) { return __half2float(x); }
    __device__ static __half from_f(float x) { return __float2half_rn(x); }
};

// 16-byte vector of T, loaded / stored with one instruction, unpacked to fp32.
template <typename T> struct alignas(16) Vec16 {
    static constexpr int N = DType<T>::VEC;
    T e[N];
    __device__ void load(const T* p) { *reinterpret_cast<uint4*>(e) = *reinterpret_cast<const uint4*>(p); }
    __device__ void load_nc(const T* p) { *reinterpret_cast<uint4*>(e) = __ldg(reinterpret_cast<const uint4*>(p)); }
    __device__ void store(T* p) const { *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(e); }
    __device__ void to_float(float* f) const {
#pragma unroll
        for (int i = 0; i < N; ++i) f[i] = DType<T>::to_f(e[i]);
    }
    __device__ void from_float(const float* f) {
#pragma unroll
        for (int i = 0; i < N; ++i) e[i] = DType<T>::from_f(f[i]);
    }
};

__device__ __forceinline__ float log_sigmoid(float x) {
    // min(x,0) - log1p(exp(-|x|)), the numerically stable form torch uses
    return fminf(x, 0.f) - log1pf(__expf(-fabsf(x)));
}

__device__ __forceinline__ float sigmoidf_(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
// Sigmoid for kernels whose result is rounded to a 16-bit type: one MUFU (tanh.approx, ~2^-11 relative) instead of two
// (exp + reciprocal) -- these kernels are bound by the quarter-rate MUFU pipe, not by DRAM.  fp32 keeps the exact form.
template <typename T> __device__ __forceinline__ float sigmoid_t(float x) {
    if (sizeof(T) == 4) return sigmoidf_(x);
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
    return fmaf(0.5f, t, 0.5f);
}

// Scan of states over chunks, four neighbouring values of one key channel: in place, local states become the states that
// enter each chunk.  slot(i): index of the i-th chunk in scan order; the loads of 8 to 16 chunks are in flight ahead of the
// dependent chain (with 4, long scans took 1.4 to 1.7 times as long: few threads, each waiting).  Returns the state after the last chunk; gsum: summed log-gates of the channel.
template <typename Slot, typename Decay>
__device__ __forceinline__ float4 scan_states(float4* ws, const float* decay, int per, int e, int dk, int d, int nchunk, float4 S, float& gsum, Slot slot, Decay factor) {
    constexpr int PF = 8;
    float4 u[2][PF];
    float g[2][PF];
    auto fetch = [&](int c0, int b) {
#pragma unroll
        for (int i = 0; i < PF; ++i) {
            if (c0 + i < nchunk) {
                const size_t s = slot(c0 + i);
                u[b][i] = __ldcg(ws + s * per + e);
                g[b][i] = __ldcg(decay + s * dk + d);
            }
        }
    };
    auto run = [&](int c0, int b) {
#pragma unroll
        for (int i = 0; i < PF; ++i) {
            if (c0 + i < nchunk) {
                __stcg(ws + slot(c0 + i) * per + e, S);
                const float a = factor(g[b][i]);
                gsum += g[b][i];
                S.x = fmaf(S.x, a, u[b][i].x); S.y = fmaf(S.y, a, u[b][i].y); S.z = fmaf(S.z, a, u[b][i].z); S.w = fmaf(S.w, a, u[b][i].w);
            }
        }
    };
    fetch(0, 0);
    for (int c0 = 0; c0 < nchunk; c0 += 2 * PF) {
        if (c0 + PF < nchunk) fetch(c0 + PF, 1);
        run(c0, 0);
        if (c0 + PF >= nchunk) break;
        if (c0 + 2 * PF < nchunk) fetch(c0 + 2 * PF, 0);
        run(c0 + PF, 1);
    }
    return S;
}

// SMs of the current device (1 where there is none to ask)
inline int device_sms() {
    static std::atomic<int> known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    int n = known[dev].load(std::memory_order_relaxed);
    if (!n) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 1;
        known[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// GELU in its erf form.  16-bit results: erf by Abramowitz & Stegun 7.1.26 (|error| <= 1.5e-7), one exponential and one
// reciprocal; fp32 keeps erff.
template <typename T> __device__ __forceinline__ float gelu_t(float x) {
    const float z = x * 0.70710678118654752f;
    if (sizeof(T) == 4) return 0.5f * x * (1.f + erff(z));
    const float az = fabsf(z), t = __fdividef(1.f, fmaf(0.3275911f, az, 1.f));
    const float poly = t * fmaf(t, fmaf(t, fmaf(t, fmaf(t, 1.061405429f, -1.453152027f), 1.421413741f), -0.284496736f), 0.254829592f);
    const float q = poly * __expf(-az * az);                     // 1 - erf(|z|)
    return 0.5f * x * (z < 0.f ? q : 2.f - q);
}

// Programmatic dependent launch.  A kernel that calls pdl_wait() before it touches what an earlier kernel wrote may be launched
// while that kernel still runs (launch_chained); pdl_launch() lets the next kernel of the stream do the same.  Both do nothing
// in an ordinary launch.  A kernel allocates tensor memory only after pdl_wait(): earlier it could hold what a kernel it
// waits for still has to allocate.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What an earlier kernel writes is not read through the non-coherent path by one that may have begun before that write.
__device__ __forceinline__ uint2 ld_coherent(const void* p) {
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// Whether this thread's launches may be chained: set around a model's forward, whose kernels read weights -- which none of them
// writes -- before pdl_wait().
extern thread_local int chain_launches;

template <typename... K, typename... A>
inline cudaError_t launch_overlapped(bool overlap, void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, K(args)...);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <typename... K, typename... A>
inline cudaError_t launch_chained(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    return launch_overlapped(chain_launches != 0, kernel, grid, block, smem, stream, std::forward<A>(args)...);
}

// A later launch of one call, behind a first one in the ordinary way: the call's inputs were complete before that one began, so
// they may be read before pdl_wait(), and only what the call itself wrote has to be waited for.
template <typename... K, typename... A>
inline cudaError_t launch_next(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    return launch_overlapped(true, kernel, grid, block, smem, stream, std::forward<A>(args)...);
}

// Parameter block of the bi-GLA launchers (host fills it from the C ABI arguments).
struct BiglaParams {
    const void *q, *k, *v, *gf, *gb;
    void* o;
    int64_t sq[3], sk[3], sv[3], sgf[3], sgb[3], so[3];  // element strides of (b, h, l)
    int B, H, L, dk, dv, dtype;
    float qscale;       // scale * out_scale, folded into q
    float gate_norm;    // > 0: gates are raw logits, g = logsigmoid(x) / gate_norm
    float clamp_min;    // NaN = no clamp
    const float *init_f, *init_b;
    float *final_f, *final_b, *logdecay_f, *logdecay_b;
    int dir_mask;
    float* ws_state;    // [B*H][nchunk][2][dk*dv]
    float* ws_decay;    // [B*H][nchunk][2][dk]
    int nchunk;
    int32_t* status;
    // single-launch tensor-core path: work tickets, per-(b,h) arrival counters, per-CTA scratch for operand tiles
    uint32_t* ticket;
    uint32_t* group_cnt;
    uint8_t* qscratch;
    int nseg;
};

__device__ __forceinline__ float gate_transform(float x, float gate_norm, float clamp_min) {
    float g = gate_norm > 0.f ? log_sigmoid(x) / gate_norm : x;
    if (clamp_min == clamp_min) g = fmaxf(g, clamp_min);
    return g;
}

int bigla_simt_launch(const BiglaParams& p, cudaStream_t stream);
size_t bigla_simt_workspace(int B, int H, int L, int dk, int dv);
// mma.sync form, both directions of a segment in one sweep (short and medium sequences, dv = 32, fp32)
bool bigla_seg_supported(const BiglaParams& p);
bool bigla_seg_preferred(const BiglaParams& p);
int bigla_seg_launch(const BiglaParams& p, size_t ws_bytes, cudaStream_t stream);
size_t bigla_seg_workspace(int B, int H, int L, int dk, int dv, int dtype);   // with which small calls run in their finest segments; bigla_simt_workspace is enough
// scan over p.nchunk per-chunk (or per-segment) local states in the workspace, in place (phase B)
int bigla_scan_launch(const BiglaParams& p, cudaStream_t stream);
int bigla_tc_launch(const BiglaParams& p, void* ws, size_t ws_bytes, bool allow_fused, cudaStream_t stream);
size_t bigla_tc_workspace(int B, int H, int L, int dk, int dv, bool split_only);
size_t bigla_tc_min_workspace(const BiglaParams& p);   // what this very call uses (0 for one segment with an output)
bool bigla_tc_supported(const BiglaParams& p);
bool bigla_tc_prefers_single(int L);
// warp-specialised wavefront form (large batches): one persistent CTA per SM, state hand-off between segments
bool bigla_wave_supported(const BiglaParams& p);
bool bigla_wave_preferred(const BiglaParams& p);
size_t bigla_wave_workspace(int B, int H, int L, int dk, int dv);
int bigla_wave_launch(const BiglaParams& p, void* ws, size_t ws_bytes, cudaStream_t stream);
// TMA-fed depthwise conv: launches and returns a status, or VIG_DWCONV_NOT_TAKEN when the shape is left to the other forms
constexpr int VIG_DWCONV_NOT_TAKEN = -1000;
int dwconv_tma_try(const void* x, const void* wt, const void* bias, void* y, int B, int h, int w, int C, int act, int dtype,
                   int32_t* status, cudaStream_t stream);

}  // namespace vig
