// r = x W^T + residual,  h = RMSNorm(r) * norm_weight   in one kernel (bf16 / fp16): the output projection of the
// attention branch (or the down projection of the MLP) with the residual add and the next RMSNorm as its epilogue
// (classification/models/vig.py:463 `o_proj`, :497 `down_proj`, :596-606 `attn_norm` / `mlp_norm` with residual and
// prenorm).  The projection output never goes to HBM: instead of (GEMM: write y) + (norm: read y, read residual,
// write r, write h) the kernel reads the residual and writes r and h.
//
// Here: rows of up to 192 values, on single CTAs; longer ones in gemm_pair_norm.cu.
//
// tcgen05 GEMM with full output rows per tile.  A persistent CTA owns tiles of 128 rows; x and W stream through a ring
// of stages [128 x 64 of x | N x 64 of W] (TMA, 128-byte swizzle); the accumulator [128 x N] fp32 lives in tensor
// memory (two buffers: the epilogue of a tile overlaps the MMAs of the next).
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warps 2..9 epilogue.  Every wait is bounded.
// Epilogue: the tile's residual rows arrive by TMA in 128-byte-swizzled boxes (two tile
// buffers); a thread owns half a row (its TMEM lane, two warps per lane quadrant): pass 1 adds the residual with the
// roundings of the unfused path (projection rounded to T, sum rounded to T), writes r in place and keeps it in
// registers, the halves' sums of squares meet in shared memory; a TMA store sends r out; pass 2 writes h over the same
// boxes once that store has read them and a second TMA store sends h out.  (Per-thread row stores, the first version,
// cost 32 sectors per request and made the kernel slower than the two it replaces.)
#include "tc_common.cuh"
#include "gemm_pair.h"

namespace vig {
namespace {

using namespace tc;

constexpr int AN_BK = 64;                      // k elements per stage (128 bytes per row)
constexpr int AN_THREADS = 64 + 256;            // TMA warp, MMA warp, 8 epilogue warps (two per TMEM lane quadrant)
constexpr int AN_A_BYTES = 128 * AN_BK * 2;    // [128 rows x 64 k]

struct AnMaps { CUtensorMap x, w, res, r, h; };

__device__ __forceinline__ void epi_bar_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

template <typename T, int NT>            // NT = N, the row width, a compile-time constant so that a row lives in registers
__global__ void __launch_bounds__(AN_THREADS, 1) linear_add_rmsnorm_kernel(const __grid_constant__ AnMaps maps, bool has_res, const T* __restrict__ norm_w, int M, int KB,
                                                                           int nstage, float eps, int32_t* status) {
    extern __shared__ uint8_t an_smem_raw[];
    uint8_t* smem = an_smem_raw + ((1024u - (smem_u32(an_smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    constexpr int N = NT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage_bytes = AN_A_BYTES + (uint32_t)N * AN_BK * 2;
    constexpr uint32_t E_BYTES = (uint32_t)(NT / 64) * 128 * 128;      // one [128 x N] tile as N/64 swizzled boxes
    const uint32_t off_e = (uint32_t)nstage * stage_bytes;
    const uint32_t off_bar = off_e + 2 * E_BYTES;
    const uint32_t bar_full = sbase + off_bar, bar_empty = bar_full + 8 * 8;          // up to 8 stages
    const uint32_t bar_acc_full = bar_empty + 8 * 8, bar_acc_empty = bar_acc_full + 16;
    const uint32_t bar_res_full = bar_acc_empty + 16, bar_e_free = bar_res_full + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + off_bar + 8 * 24);
    float* ss_part = reinterpret_cast<float*>(smem + off_bar + 8 * 24 + 16);       // [2 column halves][128 rows]
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const Waiter waiter{abort_flag, status};

    if (tid == 0) {
        for (int s = 0; s < nstage; ++s) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_acc_full + 8 * b, 1); mbar_init(bar_acc_empty + 8 * b, 256);
            mbar_init(bar_res_full + 8 * b, 1); mbar_init(bar_e_free + 8 * b, 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int ntiles = (M + 127) / 128;

    if (warp == 0) {
        if (lane == 0) {                          // ---- TMA producer -------------------------------------------
            uint32_t st = 0, phase = 0, t_it = 0;
            for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++t_it) {
                const uint32_t eb = t_it & 1u;        // the tile's residual rows, into the epilogue buffer of this tile
                waiter.wait(bar_e_free + 8 * eb, ((t_it >> 1) & 1u) ^ 1u);
                if (*abort_flag) break;
                if (has_res) {
                    mbar_expect_tx(bar_res_full + 8 * eb, E_BYTES);
                    for (int bx = 0; bx < NT / 64; ++bx)
                        tma_load_2d(sbase + off_e + eb * E_BYTES + bx * 16384, &maps.res, bx * 64, tile * 128, bar_res_full + 8 * eb);
                } else {
                    mbar_arrive_plain(bar_res_full + 8 * eb);
                }
                for (int kb = 0; kb < KB; ++kb) {
                    waiter.wait(bar_empty + 8 * st, phase ^ 1u);
                    if (*abort_flag) break;
                    mbar_expect_tx(bar_full + 8 * st, stage_bytes);
                    const uint32_t dst = sbase + st * stage_bytes;
                    tma_load_2d(dst, &maps.x, kb * AN_BK, tile * 128, bar_full + 8 * st);
                    tma_load_2d(dst + AN_A_BYTES, &maps.w, kb * AN_BK, 0, bar_full + 8 * st);
                    if (++st == (uint32_t)nstage) { st = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {                       // ---- MMA issuer ---------------------------------------------
        // The whole warp walks the loop (uniform control flow keeps the descriptor arithmetic cheap), lane 0 issues;
        // a descriptor's low word advances by adding to its address field (16-byte units).
        constexpr uint32_t IDESC = make_idesc(Pack2<T>::FMT, 0, 0, 128, N);
        uint32_t st = 0, phase = 0, acc_it = 0;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++acc_it) {
            const uint32_t buf = acc_it & 1u;
            waiter.wait(bar_acc_empty + 8 * buf, ((acc_it >> 1) & 1u) ^ 1u);   // the epilogue has drained this buffer
            if (*abort_flag) break;
            tc_fence_after();
            const uint32_t d = tmem + buf * (uint32_t)N;
            for (int kb = 0; kb < KB; ++kb) {
                waiter.wait(bar_full + 8 * st, phase);
                tc_fence_after();
                const uint32_t a_lo = make_desc(sbase + st * stage_bytes), b_lo = make_desc(sbase + st * stage_bytes + AN_A_BYTES);
                if (lane == 0) {
                    tc_mma(d, a_lo, b_lo, IDESC, kb > 0 ? 1u : 0u);
                    tc_mma(d, a_lo + 2, b_lo + 2, IDESC, 1u);
                    tc_mma(d, a_lo + 4, b_lo + 4, IDESC, 1u);
                    tc_mma(d, a_lo + 6, b_lo + 6, IDESC, 1u);
                    tc_commit(bar_empty + 8 * st);                          // the stage is free when these MMAs are done
                }
                __syncwarp();
                if (++st == (uint32_t)nstage) { st = 0; phase ^= 1u; }
            }
            if (lane == 0) tc_commit(bar_acc_full + 8 * buf);
            __syncwarp();
        }
    } else {                                      // ---- epilogue through shared memory and TMA stores ----------------
        // Two threads a row (its TMEM lane).  The residual tile arrives by TMA in 128-byte-swizzled boxes; pass 1 turns
        // it into r in place (and keeps r in registers), a TMA store sends it out; pass 2 writes h over the same boxes
        // once that store has read them, and a second TMA store sends h out.
        constexpr int NH = NT / 2, NV = NH / 8;   // my half of the row: NH columns = NV 16-byte vectors
        const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;
        const int rr_ = 32 * (warp & 3) + lane;   // my row of the tile
        const int chalf = (warp - 2) >> 2;        // warps 2..5 take the first half of the columns, 6..9 the second
        const bool leader = warp == 2 && lane == 0;
        uint32_t acc_it = 0;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++acc_it) {
            const uint32_t eb = acc_it & 1u, par = (acc_it >> 1) & 1u;         // buffers of this tile, uses of them before
            uint8_t* ebuf = smem + off_e + eb * E_BYTES;
            // both waits by the whole warp: a wait by one lane with the others parked at a warp barrier resumes microseconds late
            waiter.wait(bar_res_full + 8 * eb, par);
            waiter.wait(bar_acc_full + 8 * eb, par);
            __syncwarp();                         // (no early exit on an abort: the four warps meet at named barriers below,
            tc_fence_after();                     //  and after an abort every wait returns at once)
            const uint32_t acc = tmem + lane_base + eb * (uint32_t)NT;
            uint4 rr[NV];
            float ss = 0.f;
#pragma unroll
            for (int cc = 0; cc < NH; cc += 32) { // pass 1: r = T(T(acc) + residual), sum of squares
                const int c = chalf * NH + cc;
                float a[32];
                tc_ld32(acc + c, a);
                tc_wait_ld();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int v = c / 8 + j;      // 16-byte vector of the row: box v / 8, chunk v % 8
                    uint4* cell = reinterpret_cast<uint4*>(ebuf + (v / 8) * 16384 + rr_ * 128 + (((v % 8) ^ (rr_ & 7)) << 4));
                    uint4 rv = has_res ? *cell : make_uint4(0u, 0u, 0u, 0u);
                    uint32_t* rw = reinterpret_cast<uint32_t*>(&rv);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        // the unfused path rounds the projection to T before the add, and the sum to T before the norm
                        const float2 y = Pack2<T>::unpack(Pack2<T>::pack(a[8 * j + 2 * e], a[8 * j + 2 * e + 1]));
                        const float2 rf = Pack2<T>::unpack(rw[e]);
                        rw[e] = Pack2<T>::pack(y.x + rf.x, y.y + rf.y);
                        const float2 s2 = Pack2<T>::unpack(rw[e]);
                        ss = fmaf(s2.x, s2.x, ss); ss = fmaf(s2.y, s2.y, ss);
                    }
                    *cell = rv;
                    rr[cc / 8 + j] = rv;
                }
            }
            tc_fence_before();
            mbar_arrive_plain(bar_acc_empty + 8 * eb);        // the accumulator is read
            ss_part[chalf * 128 + rr_] = ss;                  // the other half of my row belongs to another warp
            fence_proxy_async();
            epi_bar_sync();
            ss += ss_part[(chalf ^ 1) * 128 + rr_];
            if (leader) {
                for (int bx = 0; bx < NT / 64; ++bx) tma_store_2d(&maps.r, bx * 64, tile * 128, sbase + off_e + eb * E_BYTES + bx * 16384);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the boxes may be overwritten
            }
            epi_bar_sync();
            const float rstd = rsqrtf(ss / (float)NT + eps);
#pragma unroll
            for (int vv = 0; vv < NV; ++vv) {     // pass 2: h = r * rstd * norm_weight, into the same boxes
                const int v = chalf * NV + vv;
                const uint4 wv = __ldg(reinterpret_cast<const uint4*>(norm_w) + v);
                const uint32_t* rw = reinterpret_cast<const uint32_t*>(&rr[vv]);
                const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 rf = Pack2<T>::unpack(rw[e]), wf = Pack2<T>::unpack(ww[e]);
                    o[e] = Pack2<T>::pack(rf.x * rstd * wf.x, rf.y * rstd * wf.y);
                }
                *reinterpret_cast<uint4*>(ebuf + (v / 8) * 16384 + rr_ * 128 + (((v % 8) ^ (rr_ & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
            fence_proxy_async();
            epi_bar_sync();
            if (leader) {
                for (int bx = 0; bx < NT / 64; ++bx) tma_store_2d(&maps.h, bx * 64, tile * 128, sbase + off_e + eb * E_BYTES + bx * 16384);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                mbar_arrive_plain(bar_e_free + 8 * eb);       // the buffer may take the residual of the tile after next
            }
        }
        if (leader) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // all stores have landed before the CTA exits
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace
}  // namespace vig

using namespace vig;

extern "C" int vig_linear_add_rmsnorm_supported(int64_t M, int K, int N, int dtype) {
    if (dtype != VIG_DTYPE_BF16 && dtype != VIG_DTYPE_F16) return 0;
    if (M <= 0 || K <= 0 || K % AN_BK || !(N == 64 || N == 128 || N == 192 || N == 256 || N == 384 || N == 768)) return 0;
    return tc::encode_fn() != nullptr;
}

// Whether the one kernel is to be taken instead of the library's GEMM and the norm kernel.  Rows of up to 192 values always (17-22 % faster from
// 50000 rows on).  Longer rows go in rounds of 256-row tiles, 74 pairs or 33 clusters of four at a time; a round costs about the same however
// full it is, while the two kernels' time grows with the rows, so the line is how much of its rounds a call fills (tenths).  Measured (us, one kernel / two; f rounds filled):
//   N = 384, K = 384:  f 0.65 13.6 / 13.6, 0.74 13.7 / 14.0, 1.05 20.4 / 19.7, 1.16 20.5 / 21.3, 1.32 21.0 / 25.6, 2.0 32.6 / 37.3  (rows in DRAM bound it: a round that follows is cheap)
//   N = 384, K = 1024: f 0.85 19.5 / 21.5, 1.57 38.4 / 37.4, 1.69 39.3 / 40.3, 2.2 51.8 / 50.2, 2.4 52.5 / 55.4, 3.0 65.9 / 69.7
//   N = 256, K = 256:  f 0.74 10.5 / 9.7, 0.95 10.7 / 11.1, 1.51 15.4 / 15.2, 1.69 15.6 / 17.0, 2.1 20.7 / 20.1, 2.4 21.6 / 23.1
//   N = 256, K = 704:  f 0.95 13.2 / 13.7, 1.51 19.8 / 21.2, 2.1 30.6 / 28.0, 2.4 31.6 / 30.7, 2.5 32.6 / 33.9
//   N = 768, K = 768:  f 0.76 16.3 / 14.6, 1.3 25.5 / 23.2, 1.67 26.8 / 29.1, 2.4 42.9 / 41.9, 2.6 43.8 / 45.9, 3.2 54.4 / 53.2, 3.4 55.0 / 59.4, 4.03 65.7 / 69.7
//   N = 768, K = 2048: f 1.9 54.3 / 52.7, 2.6 75.5 / 73.2, 3.0 78.4 / 80.4, 3.4 97.0 / 97.3, 3.8 100 / 105, 9.1 267 / 252, 15.5 395 / 415
extern "C" int vig_linear_add_rmsnorm_preferred(int64_t M, int K, int N, int dtype) {
    if (!vig_linear_add_rmsnorm_supported(M, K, N, dtype)) return 0;
    if (N <= 192) return 1;
    const int64_t all = pair_norm_clusters(N, dtype), tiles = (M + 255) / 256, rounds = (tiles + all - 1) / all;
    const int64_t tenths = N == 384 && K <= N ? 5 * rounds + 2 : K > (N == 768 ? 768 : 1024) ? 9 * rounds + 2 : N == 768 ? 8 * rounds + (rounds == 1) : 7 * rounds + 2;
    return 10 * tiles >= all * tenths;
}

extern "C" int vig_linear_add_rmsnorm_fwd(const void* x, int64_t ldx, const void* w, const void* residual, const void* norm_weight,
                                          void* out_r, void* out_h, int64_t M, int K, int N, float eps, int dtype,
                                          int32_t* status_dev, void* stream) {
    if (!x || !w || !norm_weight || !out_r || !out_h) return VIG_ERR_NULL;
    if (M == 0) return VIG_OK;
    if (!vig_linear_add_rmsnorm_supported(M, K, N, dtype)) return VIG_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(residual) |
         reinterpret_cast<uintptr_t>(norm_weight) | reinterpret_cast<uintptr_t>(out_r) | reinterpret_cast<uintptr_t>(out_h)) & 15)
        return VIG_ERR_ALIGN;
    if (ldx < K || (ldx * 2) % 16 || M >= (1ll << 31) - 128) return VIG_ERR_ARG;
    if (N > 192) return pair_norm_launch(x, ldx, w, residual, norm_weight, out_r, out_h, M, K, N, eps, dtype, status_dev, (cudaStream_t)stream);
    AnMaps maps;
    if (!tc::make_map_2d(&maps.x, x, M, K, ldx, 128, dtype) || !tc::make_map_2d(&maps.w, w, N, K, K, N, dtype)) return VIG_ERR_DEVICE;
    const int stage_bytes = AN_A_BYTES + N * AN_BK * 2;
    const size_t e_bytes = 2 * (size_t)(N / 64) * 16384;
    int nstage = (int)((227 * 1024 - 4096 - e_bytes) / stage_bytes);     // the ring gets what the two epilogue tiles leave of the 227 KB
    if (nstage > 6) nstage = 6;
    const size_t smem = (size_t)nstage * stage_bytes + e_bytes + 8 * 24 + 16 + 2 * 128 * 4 + 1024;
    if ((residual && !tc::make_map_2d(&maps.res, residual, M, N, N, 128, dtype)) || !tc::make_map_2d(&maps.r, out_r, M, N, N, 128, dtype) ||
                    !tc::make_map_2d(&maps.h, out_h, M, N, N, 128, dtype))
        return VIG_ERR_DEVICE;
    cudaError_t e;
    const int64_t ntiles = (M + 127) / 128;
    const int sms = device_sms(), grid = (int)(ntiles < sms ? ntiles : sms);
#define VIG_AN_LAUNCH(TT, NN)                                                                                                  \
    {                                                                                                                          \
        auto kfn = linear_add_rmsnorm_kernel<TT, NN>;                                                                          \
        if ((e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kfn), (int)smem)) != cudaSuccess) return (int)e; \
        kfn<<<grid, AN_THREADS, smem, (cudaStream_t)stream>>>(maps, residual != nullptr, (const TT*)norm_weight, (int)M, K / AN_BK, nstage, eps, status_dev); \
    }
#define VIG_AN_WIDTHS(TT)                                                                                                      \
    switch (N) {                                                                                                               \
        case 64: VIG_AN_LAUNCH(TT, 64) break;                                                                                  \
        case 128: VIG_AN_LAUNCH(TT, 128) break;                                                                                \
        default: VIG_AN_LAUNCH(TT, 192) break;                                                                                 \
    }
    if (dtype == VIG_DTYPE_BF16) VIG_AN_WIDTHS(__nv_bfloat16) else VIG_AN_WIDTHS(__half)
#undef VIG_AN_WIDTHS
#undef VIG_AN_LAUNCH
    return (int)cudaGetLastError();
}
