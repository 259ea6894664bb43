// r = x W^T + residual,  h = RMSNorm(r) * norm_weight  on pairs of CTAs (tcgen05, cta_group::2): the output projections of a block
// with the residual add and the next RMSNorm as their epilogue (classification/models/vig.py:463 `o_proj`, :497 `down_proj`,
// :596-606), for rows of 256, 384 and 768 values.  The projection never goes to HBM.
//
// A pair owns 256 full rows: its two tensor memories hold 128 x BN accumulators each, BN up to 384 (one buffer; two of 256).  Rows of
// 768 are shared by the two pairs of a cluster of four CTAs, 384 columns each, which tell each other their rows' sums of squares by st.async.
// x and W stream through a ring of k boxes as in gemm_pair.cu; a tile's residual rows come by TMA into a buffer of their own while its products run.
// Roles: warp 0 loads x and W, warp 1 of the even CTA issues the pair's MMAs, warp 2 loads the residual, then epilogue warps of 32 rows x 128
// columns: pass 1 adds the residual with the roundings of the separate kernels (projection rounded to T, sum rounded to T), keeps r in
// registers and sends it out of its own part of the buffer, so that tensor memory is free before the norm; pass 2 sends h the same way.
// Bound: three stages of 40 KB are what shared memory leaves beside the residual, 1000 cycles a box against 770 of its MMAs; behind the last tile
// the two passes and their stores, 9000 cycles; with many tiles the copy rate (4.4 of 6.4 TB/s at N = 384).  Without a difference: x asked into L2 ahead,
// by boxes or by rows, and k boxes started at another place in every tile.  Packed adds and weights in fp32 halved the passes (3900 + 1900 -> 2400 + 1600 cycles).
// Every wait is bounded.
#include "tc_common.cuh"
#include "gemm_pair.h"

namespace vig {
namespace {

using namespace tc;

constexpr int PN_BK = 64;
constexpr int PN_A = 128 * PN_BK * 2;
constexpr int PN_CW = 128;                               // columns of an epilogue warp

template <int BN, int NP> struct NormCfg {               // BN columns a pair, NP pairs a row
    static constexpr int NM = BN > 256 ? 2 : 1;          // MMAs a k step
    static constexpr int WROWS = BN / (2 * NM);          // rows of W a CTA loads for each of them
    static constexpr int STAGE = PN_A + BN / 2 * PN_BK * 2;
    static constexpr int E = 128 * BN * 2;               // the residual rows, then r, then h
    static constexpr int PARTS = BN / PN_CW, EPI_WARPS = 4 * PARTS, THREADS = 96 + 32 * EPI_WARPS;
    static constexpr int NB = 2 * BN <= 512 ? 2 : 1;     // accumulators
    static constexpr int SS = 2 * NP * PARTS * 128 * 4;  // sums of squares: [tile parity][part of the row][row]
    static constexpr int NW = BN * 4;                    // the norm's weights in fp32
    static constexpr int MAX_ST = 8, BARS = 8 * (2 * MAX_ST + 8);
    static constexpr int NST = (227 * 1024 - 1024 - E - SS - NW - BARS - 16) / STAGE < MAX_ST ? (227 * 1024 - 1024 - E - SS - NW - BARS - 16) / STAGE : MAX_ST;
    static constexpr int SMEM = NST * STAGE + E + SS + NW + BARS + 16 + 1024;
    static_assert(NST >= 3, "a ring");
};

struct NormMaps { CUtensorMap x, w, res, r, h; };

template <typename T, int BN, int NP>
__global__ void __cluster_dims__(2 * NP, 1, 1) __launch_bounds__(NormCfg<BN, NP>::THREADS, 1)
gemm_pair_norm_kernel(const __grid_constant__ NormMaps maps, bool has_res, const T* __restrict__ norm_w, int M, int KB, int ntiles, float eps, int32_t* status) {
    using Cfg = NormCfg<BN, NP>;
    constexpr int NST = Cfg::NST, N = BN * NP;
    extern __shared__ uint8_t pn_smem_raw[];
    uint8_t* smem = pn_smem_raw + ((1024u - (smem_u32(pn_smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank(), even = rank & ~1u, half = rank & 1u;
    const int cols0 = (int)(rank >> 1) * BN;             // my pair's columns
    const int first = (int)blockIdx.x / (2 * NP), step = (int)gridDim.x / (2 * NP);
    constexpr uint32_t off_e = NST * Cfg::STAGE, off_ss = off_e + Cfg::E, off_nw = off_ss + Cfg::SS, off_bar = off_nw + Cfg::NW;
    const uint32_t bar_full = sbase + off_bar, bar_empty = bar_full + 8 * Cfg::MAX_ST, bar_acc_full = bar_empty + 8 * Cfg::MAX_ST, bar_acc_empty = bar_acc_full + 16,
                   bar_ss = bar_acc_empty + 16, bar_res = bar_ss + 16, bar_free = bar_res + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + off_bar + Cfg::BARS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const Waiter waiter{abort_flag, status};

    if (tid == 0) {
        for (int s = 0; s < NST; ++s) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_acc_full + 8 * b, 1); mbar_init(bar_acc_empty + 8 * b, 2 * Cfg::EPI_WARPS);
            mbar_init(bar_ss + 8 * b, Cfg::EPI_WARPS);
        }
        mbar_init(bar_res, 1); mbar_init(bar_free, Cfg::EPI_WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < BN; i += Cfg::THREADS) reinterpret_cast<float*>(smem + off_nw)[i] = DType<T>::to_f(norm_w[cols0 + i]);   // a weight: no kernel writes it
    if (tid == 32) { tma_prefetch_map(&maps.x); tma_prefetch_map(&maps.w); tma_prefetch_map(&maps.res); tma_prefetch_map(&maps.r); tma_prefetch_map(&maps.h); }
    pdl_wait();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                      // the barriers of all CTAs exist
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {                                     // ---- x and W: my rows, counted by the pair's even CTA
        uint32_t st = 0, phase = 0;
        for (int tile = first; tile < ntiles; tile += step) {
            for (int kb = 0; kb < KB; ++kb) {
                waiter.wait_lite(bar_empty + 8 * st, phase ^ 1u);
                if (*abort_flag) break;
                if (lane == 0) {
                    if (half == 0) mbar_expect_tx(bar_full + 8 * st, 2 * Cfg::STAGE);
                    const uint32_t bar = map_rank(bar_full + 8 * st, even), dst = sbase + st * Cfg::STAGE;
                    tma_load_2d_pair(dst, &maps.x, kb * PN_BK, tile * 256 + 128 * (int)half, bar);
#pragma unroll
                    for (int j = 0; j < Cfg::NM; ++j)
                        tma_load_2d_pair(dst + PN_A + j * Cfg::WROWS * PN_BK * 2, &maps.w, kb * PN_BK, cols0 + (2 * j + (int)half) * Cfg::WROWS, bar);
                }
                __syncwarp();
                if (++st == NST) { st = 0; phase ^= 1u; }
            }
            if (*abort_flag) break;
        }
        for (int s = 0; s < NST; ++s) {                  // no arrival is on its way to this CTA when it ends
            waiter.wait_lite(bar_empty + 8 * st, phase ^ 1u);
            if (++st == NST) { st = 0; phase ^= 1u; }
        }
    } else if (warp == 1) {
        if (half == 0) {                                 // ---- MMA issuer of the pair
            const bool issuer = lane == 0;
            constexpr uint32_t IDESC = make_idesc(Pack2<T>::FMT, 0, 0, 256, BN / Cfg::NM);
            uint32_t st = 0, phase = 0, it = 0, pre = 0;
            const uint32_t lo0 = make_desc(sbase);
            for (int tile = first; tile < ntiles; tile += step, ++it) {
                const uint32_t buf = Cfg::NB == 2 ? it & 1u : 0u, use = Cfg::NB == 2 ? it >> 1 : it;
                waiter.wait_lite(bar_acc_empty + 8 * buf, (use & 1u) ^ 1u);
                if (*abort_flag) break;
                tc_fence_after();
                const uint32_t d = tmem + buf * 256u;
                for (int kb = 0; kb < KB; ++kb) {
                    if (!pre) waiter.wait_lite(bar_full + 8 * st, phase);
                    tc_fence_after();
                    const uint32_t st_next = st + 1 == NST ? 0u : st + 1, ph_next = st + 1 == NST ? phase ^ 1u : phase;
                    const uint32_t a_lo = lo0 + st * (Cfg::STAGE >> 4), b_lo = a_lo + (PN_A >> 4);
#pragma unroll
                    for (uint32_t k4 = 0; k4 < 4; ++k4) {
                        if (k4 == 3) pre = mbar_test_wait(bar_full + 8 * st_next, ph_next);
#pragma unroll
                        for (uint32_t j = 0; j < Cfg::NM; ++j) {
                            if (issuer) tc_mma_pair(d + j * (BN / Cfg::NM), a_lo + 2 * k4, b_lo + 2 * k4 + j * ((Cfg::WROWS * PN_BK * 2) >> 4), IDESC, (kb | k4) > 0 ? 1u : 0u);
                        }
                    }
                    if (issuer) tc_commit_pair(bar_empty + 8 * st, even);
                    st = st_next; phase = ph_next;
                }
                if (issuer) tc_commit_pair(bar_acc_full + 8 * buf, even);
            }
        }
    } else if (warp == 2) {                              // ---- the residual rows of each tile, into the buffer that the tile before has left
        uint32_t it = 0;
        if (has_res)
            for (int tile = first; tile < ntiles; tile += step, ++it) {
                waiter.wait_lite(bar_free, (it & 1u) ^ 1u);
                if (*abort_flag) break;
                if (lane == 0) {
                    mbar_expect_tx(bar_res, Cfg::E);
                    for (int b = 0; b < BN / 64; ++b) tma_load_2d(sbase + off_e + b * 16384, &maps.res, cols0 + b * 64, tile * 256 + 128 * (int)half, bar_res);
                }
                __syncwarp();
            }
    } else {                                             // ---- epilogue
        constexpr int NV = PN_CW / 8;                    // 16-byte vectors of my part of a row
        const int part = (warp - 3) >> 2, quad = warp & 3;
        const int row_in = 32 * quad + lane;             // my row of the CTA's 128
        const uint32_t lane_base = (uint32_t)(32 * quad) << 16;
        uint8_t* mine = smem + off_e + (PN_CW / 64) * part * 16384 + row_in * 128;        // my row in the first of my boxes
        const uint32_t warp_box = sbase + off_e + (PN_CW / 64) * part * 16384 + quad * 4096;
        float* ss_all = reinterpret_cast<float*>(smem + off_ss);
        const int slot = (int)(rank >> 1) * Cfg::PARTS + part;
        const uint32_t drained = map_rank(bar_acc_empty, even);
        const int col = cols0 + PN_CW * part;
        uint32_t it = 0;
        for (int tile = first; tile < ntiles; tile += step, ++it) {
            const uint32_t buf = Cfg::NB == 2 ? it & 1u : 0u, use = Cfg::NB == 2 ? it >> 1 : it, par = it & 1u;
            const int row0 = tile * 256 + 128 * (int)half + 32 * quad;
            if (has_res) waiter.wait_lite(bar_res, it & 1u);
            waiter.wait_lite(bar_acc_full + 8 * buf, use & 1u);
            // (no early exit on an abort: after one every wait returns at once)
            tc_fence_after();
            const uint32_t acc = tmem + lane_base + buf * 256u + PN_CW * part;
            uint4 rr[NV];
            F2 ss2 = f2_make(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < PN_CW; c += 32) {        // pass 1
                float a[32];
                tc_ld32(acc + c, a);
                tc_wait_ld();
                if (c + 32 == PN_CW) { tc_fence_before(); __syncwarp(); if (lane == 0) mbar_arrive_cluster(drained + 8 * buf); }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int v = c / 8 + j;
                    uint4* cell = reinterpret_cast<uint4*>(mine + (v / 8) * 16384 + (((v % 8) ^ (row_in & 7)) << 4));
                    uint4 rv = has_res ? *cell : make_uint4(0u, 0u, 0u, 0u);
                    uint32_t* rw = reinterpret_cast<uint32_t*>(&rv);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        rw[e] = Pack2<T>::add(Pack2<T>::pack(a[8 * j + 2 * e], a[8 * j + 2 * e + 1]), rw[e]);
                        const float2 s = Pack2<T>::unpack(rw[e]);
                        const F2 v2 = f2_make(s.x, s.y);
                        ss2 = f2_fma(v2, v2, ss2);
                    }
                    *cell = rv;
                    rr[v] = rv;
                }
            }
            float ss = f2_lo(ss2) + f2_hi(ss2);
            float* ss_tile = ss_all + par * (NP * Cfg::PARTS * 128);
            ss_tile[slot * 128 + row_in] = ss;
            if constexpr (NP == 2) st_async_f32(map_rank(smem_u32(ss_tile + slot * 128 + row_in), rank ^ 2u), ss, map_rank(bar_ss + 8 * par, rank ^ 2u));
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                // the other pair's sums of this tile are counted as bytes
                if (NP == 2 && warp == 3) mbar_expect_tx(bar_ss + 8 * par, Cfg::EPI_WARPS * 32 * 4); else mbar_arrive_plain(bar_ss + 8 * par);
                if (row0 < M)
                    for (int b = 0; b < PN_CW / 64; ++b) tma_store_2d(&maps.r, col + 64 * b, row0, warp_box + b * 16384);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            waiter.wait_lite(bar_ss + 8 * par, (it >> 1) & 1u);
            ss = 0.f;
#pragma unroll
            for (int i = 0; i < NP * Cfg::PARTS; ++i) ss += ss_tile[i * 128 + row_in];
            const float rstd = rsqrtf(ss / (float)N + eps);
            const F2 rstd2 = f2_make(rstd, rstd);
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // r has left the buffer
            __syncwarp();
#pragma unroll
            for (int v = 0; v < NV; ++v) {               // pass 2
                const float4 *wp = reinterpret_cast<const float4*>(smem + off_nw) + (PN_CW * part) / 4 + 2 * v, w0 = wp[0], w1 = wp[1];
                const F2 ww[4] = {f2_make(w0.x, w0.y), f2_make(w0.z, w0.w), f2_make(w1.x, w1.y), f2_make(w1.z, w1.w)};
                const uint32_t* rw = reinterpret_cast<const uint32_t*>(&rr[v]);
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = Pack2<T>::unpack(rw[e]);
                    const F2 y = f2_mul(f2_mul(f2_make(f.x, f.y), rstd2), ww[e]);
                    o[e] = Pack2<T>::pack(f2_lo(y), f2_hi(y));
                }
                *reinterpret_cast<uint4*>(mine + (v / 8) * 16384 + (((v % 8) ^ (row_in & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                if (row0 < M)
                    for (int b = 0; b < PN_CW / 64; ++b) tma_store_2d(&maps.h, col + 64 * b, row0, warp_box + b * 16384);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                mbar_arrive_plain(bar_free);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                      // no CTA ends while another may still signal it
    if (tid == 0 && *abort_flag && status) atomicOr(status, 1);
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// Clusters at a time: pairs fill the GPU, clusters of four do not have to (33 of them on 148 SMs).
template <typename T, int BN, int NP> int norm_clusters() {
    using Cfg = NormCfg<BN, NP>;
    if (NP == 1) return device_sms() / 2;
    static std::atomic<int> known[64];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return device_sms() / 4;
    if ((n = known[dev & 63].load())) return n;
    auto kfn = gemm_pair_norm_kernel<T, BN, NP>;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(2 * NP); cfg.blockDim = dim3(Cfg::THREADS); cfg.dynamicSmemBytes = Cfg::SMEM;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * NP; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (ensure_smem_attr(reinterpret_cast<const void*>(kfn), Cfg::SMEM) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kfn, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = device_sms() / 4;
    }
    known[dev & 63].store(n);
    return n;
}

template <typename T, int BN, int NP>
int norm_launch(const void* x, int64_t ldx, const void* w, const void* residual, const void* norm_w, void* out_r, void* out_h, int64_t M, int K, float eps,
                int dtype, int32_t* status, cudaStream_t stream) {
    using Cfg = NormCfg<BN, NP>;
    constexpr int N = BN * NP;
    NormMaps maps;
    if (!make_map_2d(&maps.x, x, M, K, ldx, 128, dtype) || !make_map_2d(&maps.w, w, N, K, K, Cfg::WROWS, dtype) ||
        !make_map_2d(&maps.res, residual ? residual : out_r, M, N, N, 128, dtype) || !make_map_2d(&maps.r, out_r, M, N, N, 32, dtype) || !make_map_2d(&maps.h, out_h, M, N, N, 32, dtype))
        return VIG_ERR_DEVICE;
    auto kfn = gemm_pair_norm_kernel<T, BN, NP>;
    const cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(kfn), Cfg::SMEM);
    if (e != cudaSuccess) return (int)e;
    const int64_t ntiles = (M + 255) / 256, all = norm_clusters<T, BN, NP>(), clusters = all < ntiles ? all : ntiles;
    return (int)launch_chained(kfn, dim3((unsigned)(2 * NP * clusters)), dim3(Cfg::THREADS), Cfg::SMEM, stream, maps, residual != nullptr, (const T*)norm_w, (int)M, K / PN_BK,
                               (int)ntiles, eps, status);
}

}  // namespace

int pair_norm_launch(const void* x, int64_t ldx, const void* w, const void* residual, const void* norm_w, void* out_r, void* out_h, int64_t M, int K, int N, float eps,
                     int dtype, int32_t* status, cudaStream_t stream) {
#define VIG_PN(TT) switch (N) {                                                                                                                        \
        case 256: return norm_launch<TT, 256, 1>(x, ldx, w, residual, norm_w, out_r, out_h, M, K, eps, dtype, status, stream);                          \
        case 384: return norm_launch<TT, 384, 1>(x, ldx, w, residual, norm_w, out_r, out_h, M, K, eps, dtype, status, stream);                          \
        case 768: return norm_launch<TT, 384, 2>(x, ldx, w, residual, norm_w, out_r, out_h, M, K, eps, dtype, status, stream);                          \
        default: return VIG_ERR_SHAPE; }
    if (dtype == VIG_DTYPE_BF16) { VIG_PN(__nv_bfloat16) }
    VIG_PN(__half)
#undef VIG_PN
}

int pair_norm_clusters(int N, int dtype) {
    if (N != 768) return device_sms() / 2;
    return dtype == VIG_DTYPE_BF16 ? norm_clusters<__nv_bfloat16, 384, 2>() : norm_clusters<__half, 384, 2>();
}

}  // namespace vig
