// Bi-directional gated linear attention, chunked on the tensor cores at full operand precision (mma.sync, operands split
// into bf16 terms; see mma_common.cuh): the forward of fp32 calls, and of 16-bit calls whose head sizes the tcgen05 kernels
// do not take (dv = 32: the hierarchical model's heads).  Same three phases as the token-by-token form (bigla_simt.cu):
// chunk states, scan over chunks, outputs; chunks of 64 tokens, per direction
//   o_i += mask(Qt Kt^T) V + Qt (2^r S),  Qt = c q 2^(G-r),  Kt = k 2^(r-G)
// with G the cumulative log-gate in scan order, r its value at the chunk's middle, S the state entering the chunk.
//
// Why: token by token, a 64 x 64 head costs two shared-memory loads per multiply-add and 64 dependent steps a chunk (127 us
// for 2 x 3 x 196 tokens in fp32, 2.7 ms for a 64 x 3 x 3136 fp16 call of the first hierarchical stage); as products it is
// a few hundred MMAs.  A chunk whose |G - r| leaves the factorisation's range is evaluated token by token in place.
#include "mma_common.cuh"

namespace vig {
namespace {

using namespace mm;

template <int DK, int DV, typename T> struct FwdStatesSmem {
    static constexpr uint32_t V = 0, K = V + Terms<T>::RAW * C * Pitch<DV>::B, SUM = K + Terms<T>::SC * C * Pitch<DK>::B, BYTES = SUM + 2 * NT * 4;
};

template <int DK, int DV, typename T>
__global__ void __launch_bounds__(NT) fwd_states_mma_kernel(const __grid_constant__ BiglaParams p) {
    using CL = ColLay<DK>;
    using SM = FwdStatesSmem<DK, DV, T>;
    constexpr int RAW = Terms<T>::RAW, SC = Terms<T>::SC;
    constexpr int MT = DK / 16, WN = 4 / MT, NC = DV / WN, NTL = NC / 8;      // warps: MT row tiles x WN column groups
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t sb = tc::smem_u32(smem);
    float* gsum = reinterpret_cast<float*>(smem + SM::SUM);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H;
    const int64_t t0 = (int64_t)c * C;
    const int n = min(C, p.L - (int)t0);
    const int pr = threadIdx.x % CL::PAIRS, r0 = (threadIdx.x / CL::PAIRS) * CL::RPG;
    load_raw<T, DV, RAW>(smem + SM::V, head_ptr<T>(p.v, p.sv, b, h, t0), p.sv[2], n);
    const T* kp = head_ptr<T>(p.k, p.sk, b, h, t0);
    for (int dir = gridDim.z == 1 ? 0 : blockIdx.z; dir < 2; dir += gridDim.z == 1 ? 1 : 2) {
        if (!(p.dir_mask & (1 << dir))) continue;
        const size_t slot = ((size_t)bh * p.nchunk + c) * 2 + dir;
        float2 G[CL::RPG], ref, tot;
        cum_gates<DK, T>(G, ref, tot, gsum, dir ? head_ptr<T>(p.gb, p.sgb, b, h, t0) : head_ptr<T>(p.gf, p.sgf, b, h, t0),
                         dir ? p.sgb[2] : p.sgf[2], n, dir, p.gate_norm, p.clamp_min);
        if (r0 == 0) *reinterpret_cast<float2*>(p.ws_decay + slot * DK + 2 * pr) = make_float2(tot.x * tc::LN2, tot.y * tc::LN2);
#pragma unroll
        for (int r = 0; r < CL::RPG; ++r) {
            float2 k = make_float2(0.f, 0.f);
            if (r0 + r < n) k = load2<T>(kp + (r0 + r) * p.sk[2] + 2 * pr);
            uint32_t t[SC];
            split2<SC>(k.x * ex2_t<T>(tot.x - G[r].x), k.y * ex2_t<T>(tot.y - G[r].y), t);
#pragma unroll
            for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(smem + SM::K + i * C * Pitch<DK>::B + (r0 + r) * Pitch<DK>::B + pr * 4) = t[i];
        }
        __syncthreads();
        const int mt = warp % MT, wn = warp / MT;
        float acc[NTL][4];
#pragma unroll
        for (int i = 0; i < NTL; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
        state_mma<DK, DV, SC, RAW, NTL>(acc, sb + SM::K + mt * 32, sb + SM::V + wn * NC * 2, lane);
        float* out = p.ws_state + slot * DK * DV + (mt * 16 + (lane >> 2)) * DV + wn * NC + 2 * (lane & 3);
#pragma unroll
        for (int i = 0; i < NTL; ++i) {
            *reinterpret_cast<float2*>(out + i * 8) = make_float2(acc[i][0], acc[i][1]);
            *reinterpret_cast<float2*>(out + 8 * DV + i * 8) = make_float2(acc[i][2], acc[i][3]);
        }
        __syncthreads();
    }
}

template <int DK, int DV, typename T> struct FwdOutSmem {
    static constexpr uint32_t V = 0, K = V + Terms<T>::RAW * C * Pitch<DV>::B, Q = K + Terms<T>::SC * C * Pitch<DK>::B,
                              S = Q + Terms<T>::SC * C * Pitch<DK>::B, SUM = S + Terms<T>::SC * DK * Pitch<DV>::B, SCL = SUM + 2 * NT * 4,
                              BYTES = SCL + DK * 4;
    static_assert(SUM >= C * DV * 4, "the exact form keeps its outputs in the operand tiles");
};

// One chunk token by token (any gates), outputs of both directions summed in shared memory: thread j < DV owns column j.
template <int DK, int DV, typename T> __device__ __noinline__ void exact_chunk(const BiglaParams& p, float* so, int bh, int c, int use_ws) {
    const int b = bh / p.H, h = bh % p.H, j = threadIdx.x;
    const int64_t t0 = (int64_t)c * C;
    const int n = min(C, p.L - (int)t0);
    if (j >= DV) return;
    for (int i = 0; i < n; ++i) so[i * DV + j] = 0.f;
    for (int dir = 0; dir < 2; ++dir) {
        if (!(p.dir_mask & (1 << dir))) continue;
        const float* init = dir ? p.init_b : p.init_f;
        const float* Sin = use_ws ? p.ws_state + (((size_t)bh * p.nchunk + c) * 2 + dir) * DK * DV : init ? init + (size_t)bh * DK * DV : nullptr;
        float st[DK];
        for (int d = 0; d < DK; ++d) st[d] = Sin ? Sin[d * DV + j] : 0.f;
        for (int ii = 0; ii < n; ++ii) {
            const int i = dir ? n - 1 - ii : ii;
            const T* g = (dir ? head_ptr<T>(p.gb, p.sgb, b, h, t0 + i) : head_ptr<T>(p.gf, p.sgf, b, h, t0 + i));
            const T *q = head_ptr<T>(p.q, p.sq, b, h, t0 + i), *k = head_ptr<T>(p.k, p.sk, b, h, t0 + i);
            const float v = DType<T>::to_f(head_ptr<T>(p.v, p.sv, b, h, t0 + i)[j]);
            float acc = 0.f;
            for (int d = 0; d < DK; ++d) {
                st[d] = fmaf(st[d], __expf(gate_transform(DType<T>::to_f(g[d]), p.gate_norm, p.clamp_min)), DType<T>::to_f(k[d]) * v);
                acc = fmaf(p.qscale * DType<T>::to_f(q[d]), st[d], acc);
            }
            so[i * DV + j] += acc;
        }
    }
    for (int i = 0; i < n; ++i)
        (reinterpret_cast<T*>(p.o) + b * p.so[0] + h * p.so[1] + (t0 + i) * p.so[2])[j] = DType<T>::from_f(so[i * DV + j]);
}

template <int DK, int DV, typename T>
__global__ void __launch_bounds__(NT) fwd_out_mma_kernel(const __grid_constant__ BiglaParams p, int use_ws) {
    using CL = ColLay<DK>;
    using SM = FwdOutSmem<DK, DV, T>;
    constexpr int RAW = Terms<T>::RAW, SC = Terms<T>::SC;
    constexpr uint32_t PK = Pitch<DK>::B, PV = Pitch<DV>::B;
    constexpr uint32_t TK = C * PK, TV = C * PV, TS = DK * PV;          // bytes from one term's tile to the next
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t sb = tc::smem_u32(smem);
    float* gsum = reinterpret_cast<float*>(smem + SM::SUM);
    float* scl = reinterpret_cast<float*>(smem + SM::SCL);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H;
    const int64_t t0 = (int64_t)c * C;
    const int n = min(C, p.L - (int)t0);
    const int pr = threadIdx.x % CL::PAIRS, gr = threadIdx.x / CL::PAIRS, r0 = gr * CL::RPG;
    const T* qp = head_ptr<T>(p.q, p.sq, b, h, t0);
    const T* kp = head_ptr<T>(p.k, p.sk, b, h, t0);
    load_raw<T, DV, RAW>(smem + SM::V, head_ptr<T>(p.v, p.sv, b, h, t0), p.sv[2], n);
    const uint32_t aQ = sb + SM::Q + 16 * w * PK + frag_rows<PK>(lane), bK = sb + SM::K + frag_cols<PK>(lane);
    const uint32_t tV = sb + SM::V + frag_rows<PV>(lane), tS = sb + SM::S + frag_rows<PV>(lane);
    float o[DV / 8][4];
#pragma unroll
    for (int i = 0; i < DV / 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] = 0.f;
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
        if (!(p.dir_mask & (1 << dir))) continue;
        const float* init = dir ? p.init_b : p.init_f;
        const float* Sin = use_ws ? p.ws_state + (((size_t)bh * p.nchunk + c) * 2 + dir) * DK * DV : init ? init + (size_t)bh * DK * DV : nullptr;
        {
            float2 G[CL::RPG], ref, tot;
            cum_gates<DK, T>(G, ref, tot, gsum, dir ? head_ptr<T>(p.gb, p.sgb, b, h, t0) : head_ptr<T>(p.gf, p.sgf, b, h, t0),
                             dir ? p.sgb[2] : p.sgf[2], n, dir, p.gate_norm, p.clamp_min);
            const float lim = range_limit<T>();
            bool fine = fabsf(ref.x) <= lim && fabsf(ref.y) <= lim;
            if (gr == 0) *reinterpret_cast<float2*>(scl + 2 * pr) = make_float2(ex2_t<T>(ref.x), ex2_t<T>(ref.y));
#pragma unroll
            for (int r = 0; r < CL::RPG; ++r) {
                float2 q = make_float2(0.f, 0.f), k = q;
                if (r0 + r < n) { q = load2<T>(qp + (r0 + r) * p.sq[2] + 2 * pr); k = load2<T>(kp + (r0 + r) * p.sk[2] + 2 * pr); }
                const float x = G[r].x - ref.x, y = G[r].y - ref.y;
                fine = fine && fabsf(x) <= lim && fabsf(y) <= lim;
                uint32_t t[SC];
                split2<SC>(p.qscale * q.x * ex2_t<T>(x), p.qscale * q.y * ex2_t<T>(y), t);
#pragma unroll
                for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(smem + SM::Q + i * TK + (r0 + r) * PK + pr * 4) = t[i];
                split2<SC>(k.x * ex2_t<T>(-x), k.y * ex2_t<T>(-y), t);
#pragma unroll
                for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(smem + SM::K + i * TK + (r0 + r) * PK + pr * 4) = t[i];
            }
            if (__syncthreads_or(!fine)) {
                exact_chunk<DK, DV, T>(p, reinterpret_cast<float*>(smem), bh, c, use_ws);
                return;
            }
        }
        if (Sin) {
            load_state<DK, DV, SC>(smem + SM::S, Sin, scl, nullptr, nullptr);
            __syncthreads();
        }
#pragma unroll 1
        for (int jb = dir ? w : 0; jb < (dir ? C / 16 : w + 1); ++jb) {  // 16-token blocks scanned at or before mine
            float pb[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            uint32_t ap[SC][4];
            block_nt<DK, SC, SC>(pb, aQ, TK, bK + jb * 16 * PK, TK);
            mask_split<SC>(pb, jb == w, lane, [&](int r, int j) { return dir ? j >= r : j <= r; }, ap);
            block_nn<DV, SC, RAW>(o, ap, tV + jb * 16 * PV, TV);
        }
        if (Sin) {
#pragma unroll
            for (int ks = 0; ks < DK / 16; ++ks) {
                uint32_t fa[SC][4];
#pragma unroll
                for (int t = 0; t < SC; ++t) ldsm4(aQ + t * TK + ks * 32, fa[t]);
                block_nn<DV, SC, SC>(o, fa, tS + ks * 16 * PV, TS);
            }
        }
        __syncthreads();                                                // the tiles may be rewritten
    }
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
        const int row = 16 * w + (lane >> 2) + 8 * hf;
        if (row >= n) continue;
        T* out = reinterpret_cast<T*>(p.o) + b * p.so[0] + h * p.so[1] + (t0 + row) * p.so[2] + 2 * (lane & 3);
#pragma unroll
        for (int i = 0; i < DV / 8; ++i) store2<T>(out + 8 * i, o[i][2 * hf], o[i][2 * hf + 1]);
    }
}

template <int DK, int DV, typename T>
int launch_typed(const BiglaParams& p, cudaStream_t stream) {
    const int BH = p.B * p.H;
    constexpr uint32_t smA = FwdStatesSmem<DK, DV, T>::BYTES, smC = FwdOutSmem<DK, DV, T>::BYTES;
    const bool use_ws = p.nchunk > 1 || p.final_f || p.final_b || p.logdecay_f || p.logdecay_b;
    cudaError_t e;
    if (use_ws) {
        auto kA = fwd_states_mma_kernel<DK, DV, T>;
        if ((e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kA), (int)smA)) != cudaSuccess) return (int)e;
        // few chunks: one CTA per direction, so that more of the GPU works; many: one CTA reads k and v once for both
        const int gz = p.dir_mask == 3 && (int64_t)p.nchunk * BH < 148 * 4 ? 2 : 1;
        kA<<<dim3(p.nchunk, BH, gz), NT, smA, stream>>>(p);
        if (int s = bigla_scan_launch(p, stream)) return s;
    }
    if (p.o) {
        auto kC = fwd_out_mma_kernel<DK, DV, T>;
        if ((e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kC), (int)smC)) != cudaSuccess) return (int)e;
        kC<<<dim3(p.nchunk, BH), NT, smC, stream>>>(p, use_ws ? 1 : 0);
    }
    return (int)cudaGetLastError();
}

template <typename T>
int launch_dims(const BiglaParams& p, cudaStream_t stream) {
#define VIG_CASE(DKV, DVV) if (p.dk == DKV && p.dv == DVV) return launch_typed<DKV, DVV, T>(p, stream);
    VIG_CASE(16, 32) VIG_CASE(32, 32)
    if constexpr (sizeof(T) == 4) { VIG_CASE(32, 64) VIG_CASE(64, 64) }      // 16-bit: the tcgen05 kernels' head sizes
#undef VIG_CASE
    return VIG_ERR_SHAPE;
}

}  // namespace

// Rows are read as pairs (fp32, gates, q, k) and 16-byte vectors (16-bit v): base pointers on 16 bytes, strides multiples of
// 16 bytes.  grid.y holds B*H, hence its limit.  Everything else stays with the token-by-token form.
bool bigla_mma_supported(const BiglaParams& p) {
    const bool dims = (p.dk == 16 && p.dv == 32) || (p.dk == 32 && p.dv == 32) || (p.dtype == VIG_DTYPE_F32 && (p.dk == 32 || p.dk == 64) && p.dv == 64);
    if (!dims || (int64_t)p.B * p.H > 65535) return false;
    const int unit = p.dtype == VIG_DTYPE_F32 ? 4 : 8;
    auto ok = [&](const void* base, const int64_t* s) {
        return !base || (!(reinterpret_cast<uintptr_t>(base) & 15) && s[0] % unit == 0 && s[1] % unit == 0 && s[2] % unit == 0);
    };
    auto ok16 = [](const void* x) { return !(reinterpret_cast<uintptr_t>(x) & 15); };
    return ok(p.q, p.sq) && ok(p.k, p.sk) && ok(p.v, p.sv) && ok(p.gf, p.sgf) && ok(p.gb, p.sgb) && ok(p.o, p.so) && ok16(p.init_f) && ok16(p.init_b);
}

int bigla_mma_launch(const BiglaParams& p_in, cudaStream_t stream) {
    BiglaParams p = p_in;
    p.nchunk = (p.L + C - 1) / C;
    switch (p.dtype) {
        case VIG_DTYPE_F32: return launch_dims<float>(p, stream);
        case VIG_DTYPE_BF16: return launch_dims<__nv_bfloat16>(p, stream);
        case VIG_DTYPE_F16: return launch_dims<__half>(p, stream);
    }
    return VIG_ERR_DTYPE;
}

}  // namespace vig
