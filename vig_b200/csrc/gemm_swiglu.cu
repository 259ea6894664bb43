// out[M, I] = swiglu(x Wg^T, x Wy^T) = silu(x Wg^T) * (x Wy^T), with W = [Wg ; Wy] of shape [2I, K]:
// the gate projection of the SwiGLU MLP and its activation in one kernel, so the [M, 2I] intermediate
// (classification/models/vig.py:494-497: gate_proj -> chunk -> swiglu) never goes to HBM.
//
// Here: the form for K <= 192 and many rows, on single CTAs.  Everything else runs on CTA pairs (gemm_pair.cu).
//
// A persistent CTA owns ONE block of 128 features for the whole launch: its [256 x K] slice of W (gate rows and their y rows, 96 KB)
// is loaded once and stays in shared memory, the x tiles stream through a ring of two [128 x K], the accumulator [128 x 256] is
// double-buffered in tensor memory (tile t+1 is multiplied while tile t is read out).  The CTAs that hold the feature blocks of the
// same row tile have consecutive block indices and run in step, so a tile of x comes from DRAM once and from L2 for the others.
//  * a wait on an already completed mbarrier costs the MMA warp ~200 cycles and a lane-0 branch around the issue another ~200 to
//    reconverge: a tile of x is handed over as a whole, the barriers are asked about ahead of time, and the loops are walked by the
//    whole warp with only the issuing instruction predicated on the lane.
//  * an epilogue warp works through its piece in one dependent chain (TMEM load -> sigmoids -> pack -> store): two sets of eight warps
//    take alternate tiles; a warp packs its piece into a 2 KB box of shared memory and lane 0 sends it out with one TMA store.
// M = 262144, K = 192, I = 512: 93 us before the boxes were swizzled, 90 now, 97 on CTA pairs (the epilogue's traffic slows the MMAs of both);
// 37900 rows 15 / 18, 25088 rows and fewer 25 / 14.
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warps 2..17 epilogue.  Every wait is bounded.
#include "gemm_epilogue.cuh"
#include "gemm_pair.h"

namespace vig {
namespace {

using namespace tc;

constexpr int BK = 64;                         // k elements per stage row (128 bytes)
constexpr int FEAT = 128;                      // features of a CTA
constexpr int A_BOX_BYTES = 128 * BK * 2;      // one [128 rows x 64 k] box
constexpr uint32_t W_BOX = 2 * FEAT * BK * 2;  // one k box of the weight slice: FEAT gate rows + FEAT y rows
constexpr int GS_EPI_WARPS = 16;
constexpr int GS_THREADS = 64 + 32 * GS_EPI_WARPS;
constexpr int OUT_STAGE_BYTES = GS_EPI_WARPS * OUT_BOX_BYTES;
constexpr int NST = 2;                         // x tiles in the ring

struct GsMaps { CUtensorMap x, w, o; };

// grid = row_groups * nblocks CTAs; CTA i holds feature block i % nblocks and walks row tiles i / nblocks, + row_groups, ...
template <typename T>
__global__ void __launch_bounds__(GS_THREADS, 1) linear_swiglu_wide_kernel(const __grid_constant__ GsMaps maps, int M, int I, int KB, int nblocks,
                                                                           int row_groups, int32_t* status) {
    extern __shared__ uint8_t gs_smem_raw[];
    uint8_t* smem = gs_smem_raw + ((1024u - (smem_u32(gs_smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t off_x = (uint32_t)KB * W_BOX;                            // after the weight slice
    const uint32_t off_out = off_x + NST * KB * A_BOX_BYTES;
    const uint32_t off_bar = off_out + OUT_STAGE_BYTES;
    // barriers: weight slice full; x tiles full / empty; accumulator halves full / empty
    const uint32_t bar_w = sbase + off_bar;
    const uint32_t bar_x_full = bar_w + 8, bar_x_empty = bar_x_full + 8 * NST;
    const uint32_t bar_acc_full = bar_x_empty + 8 * NST, bar_acc_empty = bar_acc_full + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + off_bar + 8 * (1 + 2 * NST + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const Waiter waiter{abort_flag, status};

    if (tid == 0) {
        mbar_init(bar_w, 1);
        for (int i = 0; i < NST; ++i) { mbar_init(bar_x_full + 8 * i, 1); mbar_init(bar_x_empty + 8 * i, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(bar_acc_full + 8 * b, 1); mbar_init(bar_acc_empty + 8 * b, GS_EPI_WARPS / 2); }
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
    const int nb = (int)blockIdx.x % nblocks, rg = (int)blockIdx.x / nblocks;
    constexpr uint32_t IDESC = make_idesc(Pack2<T>::FMT, 0, 0, 128, 2 * FEAT);

    if (warp == 0) {
        if (lane == 0) {                          // ---- TMA producer -------------------------------------------
            mbar_expect_tx(bar_w, (uint32_t)KB * W_BOX);
            for (int kb = 0; kb < KB; ++kb) {
                tma_load_2d(sbase + kb * W_BOX, &maps.w, kb * BK, nb * FEAT, bar_w);                           // gate rows
                tma_load_2d(sbase + kb * W_BOX + FEAT * BK * 2, &maps.w, kb * BK, I + nb * FEAT, bar_w);       // matching y rows
            }
        }
        __syncwarp();
        uint32_t st = 0, phase = 0;               // the whole warp waits: a lane that waits while the others are parked at a warp barrier resumes late
        for (int tile = rg; tile < ntiles; tile += row_groups) {
            waiter.wait_lite(bar_x_empty + 8 * st, phase ^ 1u);           // the MMAs of the tile a ring back have read it
            if (*abort_flag) break;
            if (lane == 0) {
                mbar_expect_tx(bar_x_full + 8 * st, KB * A_BOX_BYTES);
                for (int kb = 0; kb < KB; ++kb)
                    tma_load_2d(sbase + off_x + (st * KB + kb) * A_BOX_BYTES, &maps.x, kb * BK, tile * 128, bar_x_full + 8 * st);
            }
            __syncwarp();
            if (++st == NST) { st = 0; phase ^= 1u; }
        }
    } else if (warp == 1) {                       // ---- MMA issuer ---------------------------------------------
        const bool issuer = lane == 0;
        const uint32_t w_lo0 = make_desc(sbase), x_lo0 = make_desc(sbase + off_x);
        waiter.wait_lite(bar_w, 0);
        uint32_t st = 0, phase = 0, it = 0;
        uint32_t pre_x = 0, pre_acc = 0;
        for (int tile = rg; tile < ntiles; tile += row_groups, ++it) {
            const uint32_t buf = it & 1u;
            if (!pre_acc) waiter.wait_lite(bar_acc_empty + 8 * buf, ((it >> 1) & 1u) ^ 1u);   // the epilogue has read this half out
            if (*abort_flag) break;
            tc_fence_after();
            const uint32_t d = tmem + buf * 256u;
            if (!pre_x) waiter.wait_lite(bar_x_full + 8 * st, phase);
            tc_fence_after();
            const uint32_t st_next = st + 1 == NST ? 0u : st + 1, ph_next = st + 1 == NST ? phase ^ 1u : phase;
            for (int kb = 0; kb < KB; ++kb) {
                const uint32_t a_lo = x_lo0 + (st * KB + kb) * (A_BOX_BYTES >> 4);
                const uint32_t b_lo = w_lo0 + (uint32_t)kb * (W_BOX >> 4);
#pragma unroll
                for (uint32_t k4 = 0; k4 < 4; ++k4) {
                    if (kb + 1 == KB && k4 == 3) {       // asked ahead: the next tile of x and the other accumulator
                        pre_x = mbar_test_wait(bar_x_full + 8 * st_next, ph_next);
                        pre_acc = mbar_test_wait(bar_acc_empty + 8 * (buf ^ 1u), (((it + 1) >> 1) & 1u) ^ 1u);
                    }
                    if (issuer) tc_mma(d, a_lo + 2 * k4, b_lo + 2 * k4, IDESC, (kb | k4) > 0 ? 1u : 0u);
                }
            }
            if (issuer) tc_commit(bar_x_empty + 8 * st);
            st = st_next; phase = ph_next;
            if (issuer) tc_commit(bar_acc_full + 8 * buf);
        }
    } else {                                      // ---- epilogue: silu(gate) * y -> out ----------------------------
        // Two sets of eight warps take alternate tiles (set = accumulator half), so a warp has two tile periods for its
        // [32 rows x FEAT / 2 features]: the epilogue of a tile is a chain of latencies (accumulator ready -> TMEM load -> 32 sigmoids
        // -> box -> store, ~3 k cycles) longer than the tile's MMAs, and with all sixteen warps on every tile it set the pace.
        const int ew = warp - 2;                  // 0..15
        const uint32_t set = (uint32_t)ew >> 3;   // tiles of which parity / which accumulator half
        const int fh = (ew >> 2) & 1;             // which half of the block's features, taken as two pieces of 32
        const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;   // a warp reads the TMEM lanes of its quarter
        uint8_t* box = smem + off_out + ew * OUT_BOX_BYTES;
        const uint32_t acc = tmem + lane_base + set * 256u + (FEAT / 2) * fh;
        uint32_t it = 0, uses = 0;
        for (int tile = rg; tile < ntiles; tile += row_groups, ++it) {
            if ((it & 1u) != set) continue;
            waiter.wait_lite(bar_acc_full + 8 * set, uses & 1u);   // by the whole warp
            ++uses;
            if (*abort_flag) break;
            tc_fence_after();
            const int row0 = tile * 128 + 32 * (warp & 3);
            const int col0 = nb * FEAT + (FEAT / 2) * fh;
            float g[32], y[32];
            uint32_t pk[16];
            tc_ld32(acc, g);
            tc_ld32(acc + FEAT, y);
            tc_wait_ld();
            swiglu_pack<T>(g, y, pk);
            tc_ld32(acc + 32, g);
            tc_ld32(acc + FEAT + 32, y);
            tc_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_plain(bar_acc_empty + 8 * set);   // the accumulator is in registers: the MMA warp may refill it
            send_box(box, pk, &maps.o, col0, row0, row0 < M, lane);
            swiglu_pack<T>(g, y, pk);
            send_box(box, pk, &maps.o, col0 + FEAT / 2 - 32, row0, row0 < M, lane);
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the stores have read their boxes
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *abort_flag && status) atomicOr(status, 1);
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace
}  // namespace vig

using namespace vig;

extern "C" int vig_linear_swiglu_supported(int64_t M, int K, int I, int dtype) {
    if (dtype != VIG_DTYPE_BF16 && dtype != VIG_DTYPE_F16) return 0;
    if (M <= 0 || K <= 0 || I <= 0 || K % BK || I % 64) return 0;
    return tc::encode_fn() != nullptr;
}

// Single CTAs: a few row tiles for each CTA of a feature block.
static bool wide_takes(int64_t M, int K, int I, int sms) { return K <= 192 && I % FEAT == 0 && I / FEAT <= sms && (M + 127) / 128 >= 2 * (int64_t)sms; }

// Measured on B200 against cuBLAS + the SwiGLU kernel (us, fused / two kernels): K = 192, I = 512, M = 1000 6.9 / 5.4, 3136 7.0 / 7.2, 25088
// 14 / 26; K = 384, I = 1024, M = 1568 8.0 / 7.7, 3136 10.3 / 11.1, 25088 31 / 65; K = 768, I = 2048, M = 1568 14.4 / 14.1, 3136 19.5 / 23.4,
// 25088 114 / 163; K = 1024, I = 2816, M = 2368 23.6 / 27.6: the fused product needs the more tiles per pair the longer one takes, since
// the library splits small products finer.  Up to K = 192 it is taken at every size: it keeps the projection in fp32.
extern "C" int vig_linear_swiglu_preferred(int64_t M, int K, int I, int dtype) {
    return vig_linear_swiglu_supported(M, K, I, dtype) && (K <= 192 || (M + 255) / 256 * ((I + 127) / 128) * 320 >= (int64_t)(device_sms() / 2) * K);
}

extern "C" int vig_linear_swiglu_fwd(const void* x, int64_t ldx, const void* w, void* out, int64_t ldo,
                                     int64_t M, int K, int I, int dtype, int32_t* status_dev, void* stream) {
    if (!x || !w || !out) return VIG_ERR_NULL;
    if (M == 0) return VIG_OK;
    if (!vig_linear_swiglu_supported(M, K, I, dtype)) return VIG_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) return VIG_ERR_ALIGN;
    if (ldx < K || ldo < I || (ldx * 2) % 16 || (ldo * 2) % 16 || M >= (1ll << 31)) return VIG_ERR_ARG;
    const int sms = device_sms();
    if (!wide_takes(M, K, I, sms)) return pair_swiglu_launch(x, ldx, w, out, ldo, M, K, I, dtype, status_dev, (cudaStream_t)stream);
    const int KB = K / BK;
    GsMaps maps;
    if (!tc::make_map_2d(&maps.x, x, M, K, ldx, 128, dtype) || !tc::make_map_2d(&maps.w, w, 2 * (int64_t)I, K, K, FEAT, dtype) ||
        !tc::make_out_map(&maps.o, out, M, I, ldo, dtype)) return VIG_ERR_DEVICE;
    const int smem = KB * (int)W_BOX + NST * KB * A_BOX_BYTES + OUT_STAGE_BYTES + 8 * (1 + 2 * NST + 4) + 16 + 1024;
    const int nblocks = I / FEAT;
    const int ntiles = (int)((M + 127) / 128);
    int row_groups = sms / nblocks;                            // CTAs per feature block
    if (row_groups > ntiles) row_groups = ntiles;
    auto run = [&](auto kfn) {
        const cudaError_t e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kfn), smem);
        if (e != cudaSuccess) return (int)e;
        kfn<<<row_groups * nblocks, GS_THREADS, smem, (cudaStream_t)stream>>>(maps, (int)M, I, KB, nblocks, row_groups, status_dev);
        return (int)cudaGetLastError();
    };
    return dtype == VIG_DTYPE_BF16 ? run(linear_swiglu_wide_kernel<__nv_bfloat16>) : run(linear_swiglu_wide_kernel<__half>);
}
