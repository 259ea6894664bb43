// First convolution of the hierarchical model's patch embedding (3 channels, 3 x 3, stride 2, padding 1) with its bias, the
// LayerNorm over its channels and GELU, from the image as it is (NCHW) to channels-last rows (classification/models/vig_h.py,
// patch embedding "v2"); bf16 / fp16, 32, 48 or 64 channels.
//
// The library takes four passes: a copy to channels-last, a convolution without tensor cores for want of channels, a bias add
// and the norm (28 + 87 + 45 + 65 us for 64 images of 224 x 224, 48 channels).  Here a warp forms 16 output pixels as one
// m16n8k16 tile row with K = 27 padded to 32: a lane's eight taps are the same for every pixel, so it reads its values
// straight from the image (each is read 2.25 times, from L1), the weights stay in registers, and the norm needs two
// shuffles.  Bound by instruction issue of the norm and GELU (about 15 instructions a value); 15 us of traffic.
#include "mma_common.cuh"

namespace vig {
namespace {

using tc::Pack2;

template <typename T> __device__ __forceinline__ void mma_e(float* c, const uint32_t* a, const uint32_t* b);
template <> __device__ __forceinline__ void mma_e<__nv_bfloat16>(float* c, const uint32_t* a, const uint32_t* b) { mm::mma16816(c, a, b); }
template <> __device__ __forceinline__ void mma_e<__half>(float* c, const uint32_t* a, const uint32_t* b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <typename T, int O>
__global__ void __launch_bounds__(256, 2) embed_conv_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ conv_bias,
                                                            const T* __restrict__ ln_w, const T* __restrict__ ln_b, T* __restrict__ y, int64_t pixels, int H,
                                                            int W, int OH, int OW, float eps, int gelu) {
    constexpr int NT = O / 8;
    const int lane = threadIdx.x & 31, t = lane & 3, g = lane >> 2;
    // my taps: k = 16 ks + 8 hf + 2 t + e  <->  (channel, row, column) of the 3 x 3 x 3 window; taps past 27 read tap 0 with weight 0
    int off[8];
    uint32_t dyx = 0;                                                    // two bits each: row and column of tap i
    uint32_t wr[2][NT][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        int k = 16 * (i >> 2) + 8 * ((i >> 1) & 1) + 2 * t + (i & 1);
        if (k >= 27) k = 0;
        const int dy = k % 9 / 3, dx = k % 3;
        off[i] = (k / 9) * H * W + (dy - 1) * W + dx - 1;
        dyx |= (uint32_t)(dy * 4 + dx) << (4 * i);
    }
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int k = 16 * ks + 8 * hf + 2 * t;
                const T* row = w + (n * 8 + g) * 27;
                wr[ks][n][hf] = Pack2<T>::pack(k < 27 ? DType<T>::to_f(row[k]) : 0.f, k + 1 < 27 ? DType<T>::to_f(row[k + 1]) : 0.f);
            }
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32), tiles = (pixels + 15) / 16;
    for (int64_t tile = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); tile < tiles; tile += warps) {
        uint16_t v[2][8];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t px = (uint32_t)min(tile * 16 + g + 8 * r, pixels - 1), line = px / (uint32_t)OW;
            const int ox = (int)(px - line * OW), oy = (int)(line % (uint32_t)OH);
            const uint16_t* at = reinterpret_cast<const uint16_t*>(x) + ((int64_t)(line / (uint32_t)OH) * 3 * H + 2 * oy) * W + 2 * ox;
            // rows 2 oy - 1 .. 2 oy + 1 and columns 2 ox - 1 .. 2 ox + 1: which of the three lie inside
            const uint32_t ok_y = (oy > 0 ? 1u : 0u) | 2u | (2 * oy + 1 < H ? 4u : 0u), ok_x = (ox > 0 ? 1u : 0u) | 2u | (2 * ox + 1 < W ? 4u : 0u);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t dy = dyx >> (4 * i + 2) & 3u, dx = dyx >> (4 * i) & 3u;
                v[r][i] = (ok_y >> dy & ok_x >> dx & 1u) ? __ldg(at + off[i]) : (uint16_t)0;
            }
        }
        float c[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) c[n][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t a[4];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                for (int r = 0; r < 2; ++r) a[2 * hf + r] = (uint32_t)v[r][4 * ks + 2 * hf] | (uint32_t)v[r][4 * ks + 2 * hf + 1] << 16;
#pragma unroll
            for (int n = 0; n < NT; ++n) mma_e<T>(c[n], a, wr[ks][n]);
        }
        float sum[2] = {0.f, 0.f}, ss[2] = {0.f, 0.f};
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const float2 b = conv_bias ? Pack2<T>::unpack(__ldg(reinterpret_cast<const uint32_t*>(conv_bias + n * 8 + 2 * t))) : make_float2(0.f, 0.f);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                // the convolution's result and its sum with the bias are each rounded, as the separate passes round them
                const float2 f = Pack2<T>::unpack(Pack2<T>::pack(c[n][2 * r], c[n][2 * r + 1]));
                const float2 s = Pack2<T>::unpack(Pack2<T>::pack(f.x + b.x, f.y + b.y));
                c[n][2 * r] = s.x; c[n][2 * r + 1] = s.y;
                sum[r] += s.x + s.y;
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
            sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
            sum[r] *= 1.f / O;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) { c[n][2 * r + e] -= sum[r]; ss[r] = fmaf(c[n][2 * r + e], c[n][2 * r + e], ss[r]); }
            ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], 1);
            ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], 2);
            ss[r] = rsqrtf(ss[r] * (1.f / O) + eps);
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const float2 wf = Pack2<T>::unpack(__ldg(reinterpret_cast<const uint32_t*>(ln_w + n * 8 + 2 * t)));
            const float2 bf = Pack2<T>::unpack(__ldg(reinterpret_cast<const uint32_t*>(ln_b + n * 8 + 2 * t)));
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                uint32_t o = Pack2<T>::pack(c[n][2 * r] * ss[r] * wf.x + bf.x, c[n][2 * r + 1] * ss[r] * wf.y + bf.y);
                if (gelu) { const float2 f = Pack2<T>::unpack(o); o = Pack2<T>::pack(gelu_t<T>(f.x), gelu_t<T>(f.y)); }
                const int64_t px = tile * 16 + g + 8 * r;
                if (px < pixels) *reinterpret_cast<uint32_t*>(y + px * O + n * 8 + 2 * t) = o;
            }
        }
    }
}

template <typename T> int launch(const void* x, const void* w, const void* cb, const void* lw, const void* lb, void* y, int B, int H, int W, int O, float eps, int gelu,
                                 cudaStream_t s) {
    const int OH = (H + 1) / 2, OW = (W + 1) / 2;
    const int64_t pixels = (int64_t)B * OH * OW, blocks = (pixels + 127) / 128;
    const int64_t most = device_sms() * 8;
    const int grid = (int)(blocks < most ? blocks : most);
#define VIG_EC(OO) case OO: embed_conv_kernel<T, OO><<<grid, 256, 0, s>>>((const T*)x, (const T*)w, (const T*)cb, (const T*)lw, (const T*)lb, (T*)y, pixels, H, W, OH, OW, eps, gelu); break;
    switch (O) { VIG_EC(32) VIG_EC(48) VIG_EC(64) default: return VIG_ERR_SHAPE; }
#undef VIG_EC
    return (int)cudaGetLastError();
}

}  // namespace
}  // namespace vig

using namespace vig;

extern "C" int vig_embed_conv_ln_fwd(const void* x, const void* w, const void* conv_bias, const void* ln_w, const void* ln_b, void* y, int B, int H, int W, int O,
                                     float eps, int act_gelu, int dtype, void* stream) {
    if (!x || !w || !ln_w || !ln_b || !y) return VIG_ERR_NULL;
    if (dtype != VIG_DTYPE_BF16 && dtype != VIG_DTYPE_F16) return VIG_ERR_DTYPE;
    if (B < 0 || H <= 0 || W <= 0 || !(O == 32 || O == 48 || O == 64) || (int64_t)B * ((H + 1) / 2) * ((W + 1) / 2) >= (1ll << 31) - 16 || 3ll * H * W >= (1ll << 31)) return VIG_ERR_SHAPE;
    if (B == 0) return VIG_OK;
    for (const void* p : {conv_bias, ln_w, ln_b, (const void*)y})
        if (reinterpret_cast<uintptr_t>(p) & 3) return VIG_ERR_ALIGN;
    cudaStream_t s = (cudaStream_t)stream;
    return dtype == VIG_DTYPE_BF16 ? launch<__nv_bfloat16>(x, w, conv_bias, ln_w, ln_b, y, B, H, W, O, eps, act_gelu, s)
                                   : launch<__half>(x, w, conv_bias, ln_w, ln_b, y, B, H, W, O, eps, act_gelu, s);
}
