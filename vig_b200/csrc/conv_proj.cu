// Depthwise 3x3 convolution (+ bias, SiLU) and the stacked input projection of a block in one launch, for calls of few tokens (bf16 / fp16;
// classification/models/vig.py:427-433).
//
// As two launches these are 3 + 3 us around a microsecond of work, one behind the other: each waits for the launch before it, fetches
// its operands and writes a result that the next one reads.  Here a CTA has 16 tokens and C columns of the projection: its [C x C] slice of the
// weight and the taps are on their way into shared memory before it waits for the preceding launch; then it convolves its tokens (every column
// slice does: 9 loads a value from L2), keeps them as the A operand and multiplies on mma.sync.  The first slice writes the convolved tokens for
// the gating injection.  Bound: latency, three L2 round trips; with many tokens, the convolutions repeated by each slice.
// ViG-T of one 224 x 224 image: 277 -> 249 us a forward, 128 x 128: 237 -> 215.  With half the columns a CTA 257 and 212, with 32 tokens 262 - 267; with
// integer divisions and bounds asked by every thread 255.
//
// Roundings are those of the two kernels: the convolution in the same order of sums, rounded to the type; products summed in fp32, the
// bias added, rounded once.
#include "mma_common.cuh"

namespace vig {
namespace {

using namespace tc;

constexpr int CP_TOKENS = 16;

struct CpParams {
    const void *x, *taps, *conv_b, *w, *bias;
    void *xs, *z;
    int M, h, wd, N, act;
};

// 16 tokens and C columns a CTA; 16 x C / 8 threads: eight channels of a token each, two n tiles of 8 columns a warp
template <typename T, int C>
__global__ void __launch_bounds__(2 * C) conv_proj_kernel(const __grid_constant__ CpParams p) {
    constexpr uint32_t P = C * 2 + 16;                       // row pitch of both operands: the 8 rows of an ldmatrix in 8 different bank groups
    constexpr int TM = CP_TOKENS, THREADS = 2 * C, CG = C / 8, NS = 2;
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t *W = smem, *A = smem + C * P, *taps = A + TM * P;
    int2* tok = reinterpret_cast<int2*>(taps + 9 * C * 2);   // per token: first value of its row, and which of the 3 x 3 lie in the image
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = blockIdx.x * TM, n0 = blockIdx.y * C;
    auto copy16 = [](void* dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); };
    if (tid < 9 * CG) copy16(taps + tid * 16, reinterpret_cast<const uint4*>(p.taps) + tid);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int k = 0; k < C * CG / THREADS; ++k) {
        const int r = (tid + k * THREADS) / CG, v = tid % CG;
        copy16(W + r * P + v * 16, reinterpret_cast<const T*>(p.w) + (int64_t)(n0 + r) * C + v * 8);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid < TM) {
        const int t = row0 + tid, at = t % (p.h * p.wd), ty = at / p.wd, tx = at % p.wd;
        int mask = 0;
        for (int j = 0; j < 9; ++j) {
            const int y = ty + j / 3 - 1, x = tx + j % 3 - 1;
            if (t < p.M && y >= 0 && y < p.h && x >= 0 && x < p.wd) mask |= 1 << j;
        }
        tok[tid] = make_int2(t, mask);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                         // taps and tokens
    pdl_wait();
    pdl_launch();
    // ---- convolution
    const int cg = tid % CG, r = tid / CG;
    const int2 tk = tok[r];
    const T* at = reinterpret_cast<const T*>(p.x) + (int64_t)tk.x * C + cg * 8;
    uint4 in[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        in[j] = make_uint4(0u, 0u, 0u, 0u);
        if (tk.y >> j & 1)                                   // not through the non-coherent path: the launch before may still have been writing when this one began
            asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(in[j].x), "=r"(in[j].y), "=r"(in[j].z), "=r"(in[j].w)
                         : "l"(at + ((j / 3 - 1) * p.wd + j % 3 - 1) * C));
    }
    auto f2 = [](uint32_t u) { const float2 f = Pack2<T>::unpack(u); return f2_make(f.x, f.y); };
    const uint4 cb = p.conv_b ? __ldg(reinterpret_cast<const uint4*>(p.conv_b) + cg) : make_uint4(0u, 0u, 0u, 0u);
    F2 s[4] = {f2(cb.x), f2(cb.y), f2(cb.z), f2(cb.w)};
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        const uint4 t = *reinterpret_cast<const uint4*>(taps + j * C * 2 + cg * 16);
        s[0] = f2_fma(f2(in[j].x), f2(t.x), s[0]); s[1] = f2_fma(f2(in[j].y), f2(t.y), s[1]);
        s[2] = f2_fma(f2(in[j].z), f2(t.z), s[2]); s[3] = f2_fma(f2(in[j].w), f2(t.w), s[3]);
    }
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float lo = f2_lo(s[e]), hi = f2_hi(s[e]);
        if (p.act) { lo *= sigmoid_t<T>(lo); hi *= sigmoid_t<T>(hi); }
        o[e] = Pack2<T>::pack(lo, hi);
    }
    *reinterpret_cast<uint4*>(A + r * P + cg * 16) = make_uint4(o[0], o[1], o[2], o[3]);
    if (blockIdx.y == 0 && row0 + r < p.M) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.xs) + (int64_t)(row0 + r) * C + cg * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // ---- projection
    float acc[NS][4];
#pragma unroll
    for (int j = 0; j < NS; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
    const uint32_t a = smem_u32(A) + mm::frag_rows<P>(lane), b = smem_u32(W) + (warp * NS * 8 + (lane & 7)) * P + (lane >> 3) * 16;
#pragma unroll
    for (int ks = 0; ks < C / 16; ks += 2) {
        uint32_t fa[2][4], fb[NS][4];                        // two k steps: a B fragment's four matrices are 32 values of 8 columns
        mm::ldsm4(a + ks * 32, fa[0]); mm::ldsm4(a + ks * 32 + 32, fa[1]);
#pragma unroll
        for (int j = 0; j < NS; ++j) mm::ldsm4(b + j * 8 * P + ks * 32, fb[j]);
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int j = 0; j < NS; ++j) mm::mma_t<T>(acc[j], fa[k], fb[j] + 2 * k);
    }
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        const int col = n0 + (warp * NS + j) * 8 + 2 * (lane & 3);
        const float2 bv = p.bias ? mm::load2_coherent(reinterpret_cast<const T*>(p.bias) + col) : make_float2(0.f, 0.f);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int row = row0 + (lane >> 2) + 8 * hf;
            if (row < p.M) *reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(p.z) + (int64_t)row * p.N + col) = Pack2<T>::pack(acc[j][2 * hf] + bv.x, acc[j][2 * hf + 1] + bv.y);
        }
    }
}

template <typename T, int C> int cp_launch(const CpParams& p, cudaStream_t st) {
    auto k = conv_proj_kernel<T, C>;
    constexpr size_t smem = (size_t)(C + CP_TOKENS) * (C * 2 + 16) + 9 * C * 2 + CP_TOKENS * 8;
    const cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(k), (int)smem);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_chained(k, dim3((unsigned)((p.M + CP_TOKENS - 1) / CP_TOKENS), (unsigned)(p.N / C)), dim3(2 * C), smem, st, p);
}

}  // namespace
}  // namespace vig

using namespace vig;

extern "C" int vig_conv_proj_supported(int64_t M, int C, int N, int dtype) {
    return (dtype == VIG_DTYPE_BF16 || dtype == VIG_DTYPE_F16) && M > 0 && M < (1 << 22) && (C == 96 || C == 192) && N > 0 && N % C == 0 && N / C < 65536;
}

// As long as every CTA has an SM of its own.  Whole forwards in us, one launch / two: ViG-T (768 columns) 64 tokens 215 / 237, 196 tokens 249 / 277, 392
// tokens (100 CTAs) 273 / 279, 784 tokens (1152 columns, 294 CTAs) 340 / 337, 2508 tokens 549 / 478.  Width 96 (the hierarchical model's first stage, images
// of up to about 96 x 96; 384 columns): the two blocks of the stage 61.7 / 65.9 at 576 tokens (144 CTAs), 54.9 / 60.2 at 512.  By themselves, one behind the
// other: width 96 256 tokens 3.2 / 5.6, 576 3.4 / 5.9; width 192, 768 columns, 576 5.0 / 5.9, 1024 (256 CTAs) 6.9 / 6.2.  Width 384 was slower (196 tokens, a
// forward 404 / 392) and is not built.
extern "C" int vig_conv_proj_preferred(int64_t M, int C, int N, int dtype) {
    return vig_conv_proj_supported(M, C, N, dtype) && (M + CP_TOKENS - 1) / CP_TOKENS * (N / C) <= device_sms();
}

extern "C" int vig_conv_proj_fwd(const void* x, const void* taps, const void* conv_bias, const void* w, const void* bias, void* xs, void* z, int B, int h, int wd, int C, int N,
                                 int act_silu, int dtype, void* stream) {
    if (!x || !taps || !w || !xs || !z) return VIG_ERR_NULL;
    if (B < 0 || h <= 0 || wd <= 0) return VIG_ERR_SHAPE;
    if (B == 0) return VIG_OK;
    if (!vig_conv_proj_supported((int64_t)B * h * wd, C, N, dtype)) return VIG_ERR_SHAPE;
    for (const void* a : {x, taps, conv_bias, w, bias, (const void*)xs, (const void*)z})
        if (reinterpret_cast<uintptr_t>(a) & 15) return VIG_ERR_ALIGN;
    const CpParams p{x, taps, conv_bias, w, bias, xs, z, (int)((int64_t)B * h * wd), h, wd, N, act_silu};
    cudaStream_t st = (cudaStream_t)stream;
    if (C == 96) return dtype == VIG_DTYPE_BF16 ? cp_launch<__nv_bfloat16, 96>(p, st) : cp_launch<__half, 96>(p, st);
    return dtype == VIG_DTYPE_BF16 ? cp_launch<__nv_bfloat16, 192>(p, st) : cp_launch<__half, 192>(p, st);
}
