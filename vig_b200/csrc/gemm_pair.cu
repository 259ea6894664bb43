// y = x W^T on pairs of CTAs (tcgen05, cta_group::2), with the work that follows the product as its epilogue (bf16 / fp16):
//   SwiGLU:  out[M, I] = silu(x Wg^T) * (x Wy^T), W = [Wg ; Wy] of shape [2I, K]   (classification/models/vig.py:494-497)
//   linear:  out[M, N] = x W^T + bias; an epilogue warp sends its two pieces one behind the other through one box (with a box for each the ring is a
//            stage shorter and W of K = 384 does not fit beside it: 25088 x 384 x 2304 45.6 us against 43.5)
//
// A tile is 256 rows x BN columns of the product and belongs to the two SMs of a cluster: each loads its 128 rows of x and
// its half of the tile's rows of W (TMA, 128-byte swizzle), and its tensor memory holds its 128 rows of the result, two buffers of up to
// 256 columns.  Against one CTA with a 128 x 256 tile that halves what a product brings in from L2.  Two forms:
//   streaming:  k boxes of x and of W go through one ring; tiles go to the pairs column by column, so that x comes from DRAM once.
//   stationary: a pair keeps its columns' whole slice of W for the launch and walks row tiles, x boxes go through the ring.  What SMs
//               fetch from L2 (about 50 bytes a cycle each at most) bounds the streaming form: K = 384, I = 1024, 25088 rows.
// Roles in each CTA: warp 0 TMA producer, warp 1 of the even CTA issues the MMAs of both, warps 2..17 epilogue.  Every wait is bounded.
#include "tc_common.cuh"
#include "gemm_epilogue.cuh"
#include "gemm_pair.h"

namespace vig {
namespace {

using namespace tc;

constexpr int PR_BK = 64;                                // k elements of a box (128-byte rows)
constexpr int PR_A = 128 * PR_BK * 2;                    // one CTA's [128 rows x 64 k] box of x

// GATED: SwiGLU of gate and y columns, half as many output columns; otherwise the columns with a bias
template <bool GATED> struct PairCfg {
    static constexpr int BN = 256;                       // columns of the product in a tile
    static constexpr int B = BN / 2 * PR_BK * 2;         // one CTA's half of a k box of W
    static constexpr int OCOLS = GATED ? BN / 2 : BN, COLS = 32;         // output columns of a tile, of a box
    static constexpr int EPI_WARPS = 16, THREADS = 64 + 32 * EPI_WARPS;
    static constexpr int OUT = EPI_WARPS * OUT_BOX_BYTES;
    static constexpr int MAX_ST = 8;
    static constexpr int BARS = 8 * (2 * MAX_ST + 5);
    static constexpr int RING = 227 * 1024 - 1024 - OUT - BARS - 16;      // what is left for W and the ring
};

struct PairMaps { CUtensorMap x, w, o; };

// stat: stationary form, ``nst`` boxes of x in the ring; otherwise ``nst`` boxes of x and W
template <typename T, bool STAT, bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<GATED>::THREADS, 1)
gemm_pair_kernel(const __grid_constant__ PairMaps maps, const T* bias, int M, int N, int KB, int ntn, int ntm, int nst, int32_t* status) {
    using Cfg = PairCfg<GATED>;
    constexpr int BN = Cfg::BN;
    constexpr int STAGE = PR_A + (STAT ? 0 : Cfg::B);
    extern __shared__ uint8_t pr_smem_raw[];
    uint8_t* smem = pr_smem_raw + ((1024u - (smem_u32(pr_smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    // tiles, counted column by column: mine are first, first + step, ...; in the stationary form all of one column
    const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    const int first = pair, step = pairs, ntiles = ntm * ntn;            // stationary: pairs is a multiple of ntn
    const uint32_t off_ring = STAT ? (uint32_t)KB * Cfg::B : 0u, off_out = off_ring + (uint32_t)nst * STAGE, off_bar = off_out + Cfg::OUT;
    const uint32_t bar_full = sbase + off_bar, bar_empty = bar_full + 8 * Cfg::MAX_ST, bar_acc_full = bar_empty + 8 * Cfg::MAX_ST, bar_acc_empty = bar_acc_full + 16,
                   bar_w = bar_acc_empty + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + off_bar + Cfg::BARS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const Waiter waiter{abort_flag, status};

    if (tid == 0) {
        mbar_init(bar_w, 1);
        for (int s = 0; s < nst; ++s) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(bar_acc_full + 8 * b, 1); mbar_init(bar_acc_empty + 8 * b, 2 * Cfg::EPI_WARPS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid == 32) {
        tma_prefetch_map(&maps.x); tma_prefetch_map(&maps.w); tma_prefetch_map(&maps.o);
    }
    pdl_wait();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                      // the barriers of both CTAs exist
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---- TMA producer: my rows of x, my half of the rows of W; their bytes are counted by the even CTA.  The whole warp walks the loop
        // (a lane that waits while the others are parked at a warp barrier resumes microseconds late).
        uint32_t st = 0, phase = 0;
        if (STAT && lane == 0) {
            const int wrow = pair % ntn * Cfg::OCOLS + (rank ? GATED ? N : BN / 2 : 0);   // the even CTA has the gate rows, the odd one their y rows
            if (rank == 0) mbar_expect_tx(bar_w, 2u * KB * Cfg::B);
            for (int kb = 0; kb < KB; ++kb) tma_load_2d_pair(sbase + kb * Cfg::B, &maps.w, kb * PR_BK, wrow, map_rank(bar_w, 0));
        }
        __syncwarp();
        for (int tile = first; tile < ntiles; tile += step) {
            const int row = (tile / ntn) * 256 + 128 * (int)rank, nb = tile % ntn;
            const int wrow = nb * Cfg::OCOLS + (rank ? GATED ? N : BN / 2 : 0);
            for (int kb = 0; kb < KB; ++kb) {
                waiter.wait_lite(bar_empty + 8 * st, phase ^ 1u);            // the MMAs of a ring ago have read the stage, in both CTAs
                if (*abort_flag) break;
                if (lane == 0) {
                    if (rank == 0) mbar_expect_tx(bar_full + 8 * st, 2 * STAGE);
                    const uint32_t bar = map_rank(bar_full + 8 * st, 0), dst = sbase + off_ring + st * STAGE;
                    tma_load_2d_pair(dst, &maps.x, kb * PR_BK, row, bar);
                    if (!STAT) tma_load_2d_pair(dst + PR_A, &maps.w, kb * PR_BK, wrow, bar);
                }
                __syncwarp();
                if (++st == (uint32_t)nst) { st = 0; phase ^= 1u; }
            }
            if (*abort_flag) break;
        }
        for (int s = 0; s < nst; ++s) {                  // no arrival is on its way to this CTA when it ends
            waiter.wait_lite(bar_empty + 8 * st, phase ^ 1u);
            if (++st == (uint32_t)nst) { st = 0; phase ^= 1u; }
        }
    } else if (warp == 1) {
        if (rank == 0) {                                 // ---- MMA issuer of the pair
            // a wait costs hundreds of cycles even when its phase is long over: the next stage, and the next tile's buffer, are asked about before
            // this stage's MMAs are issued
            const bool issuer = lane == 0;
            constexpr uint32_t IDESC = make_idesc(Pack2<T>::FMT, 0, 0, 256, BN);
            uint32_t st = 0, phase = 0, it = 0, pre = 0, pre_acc = 0;
            const uint32_t lo0 = make_desc(sbase + off_ring), w_lo = make_desc(sbase);
            if (STAT) waiter.wait_lite(bar_w, 0);
            for (int tile = first; tile < ntiles; tile += step, ++it) {
                const uint32_t buf = it & 1u;
                if (!pre_acc) waiter.wait_lite(bar_acc_empty + 8 * buf, ((it >> 1) & 1u) ^ 1u);
                if (*abort_flag) break;
                tc_fence_after();
                const uint32_t d = tmem + buf * 256u;
                for (int kb = 0; kb < KB; ++kb) {
                    if (!pre) waiter.wait_lite(bar_full + 8 * st, phase);
                    tc_fence_after();
                    const uint32_t st_next = st + 1 == (uint32_t)nst ? 0u : st + 1, ph_next = st + 1 == (uint32_t)nst ? phase ^ 1u : phase;
                    const uint32_t a_lo = lo0 + st * (STAGE >> 4), b_lo = STAT ? w_lo + (uint32_t)kb * (Cfg::B >> 4) : a_lo + (PR_A >> 4);
#pragma unroll
                    for (uint32_t k4 = 0; k4 < 4; ++k4) { if (issuer) tc_mma_pair(d, a_lo + 2 * k4, b_lo + 2 * k4, IDESC, (kb | k4) > 0 ? 1u : 0u); }
                    pre = mbar_test_wait(bar_full + 8 * st_next, ph_next);
                    if (kb + 1 == KB) pre_acc = mbar_test_wait(bar_acc_empty + 8 * (buf ^ 1u), (((it + 1) >> 1) & 1u) ^ 1u);
                    if (issuer) tc_commit_pair(bar_empty + 8 * st);
                    st = st_next; phase = ph_next;
                }
                if (issuer) tc_commit_pair(bar_acc_full + 8 * buf);
            }
        }
    } else {                                             // ---- epilogue: a warp has a quarter of the rows and a quarter of the features
        // It reads its whole piece out of tensor memory before it computes, so that the buffer is free 300 cycles after its last MMA.
        // (Two sets of eight warps on alternate tiles with two pieces each held it for 4000; an arrival with release at cluster scope, which
        // waits for the warp's stores, for 2000: K = 192 5000 cycles a tile, 2300 now.)
        const int ew = warp - 2, part = ew >> 2;
        const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;   // a warp reads the TMEM lanes of its quarter
        uint8_t* box = smem + off_out + ew * OUT_BOX_BYTES;
        const uint32_t drained = map_rank(bar_acc_empty, 0);
        constexpr int OCOLS = Cfg::OCOLS, COLS = Cfg::COLS;
        uint32_t it = 0;
        for (int tile = first; tile < ntiles; tile += step, ++it) {
            const uint32_t buf = it & 1u, acc = tmem + lane_base + buf * 256u + COLS * part;
            const int row = (tile / ntn) * 256 + 128 * (int)rank + 32 * (warp & 3), col = (tile % ntn) * OCOLS + COLS * part;
            waiter.wait_lite(bar_acc_full + 8 * buf, (it >> 1) & 1u);    // by the whole warp
            if (*abort_flag) break;
            tc_fence_after();
            float g[64];
            tc_ld32(acc, g);
            tc_ld32(acc + BN / 2, g + 32);
            tc_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(drained + 8 * buf);
            uint32_t pk[16];
            if constexpr (GATED) {
                swiglu_pack<T>(g, g + 32, pk);
                send_box(box, pk, &maps.o, col, row, row < M && col < N, lane);
            } else {
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const int c = col + hf * (BN / 2);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {        // the same addresses for all lanes; N is a multiple of 8
                        const uint4 b = bias && c + 8 * j < N ? __ldg(reinterpret_cast<const uint4*>(bias + c + 8 * j)) : make_uint4(0u, 0u, 0u, 0u);
                        const uint32_t b4[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float2 bv = Pack2<T>::unpack(b4[i]);
                            pk[4 * j + i] = Pack2<T>::pack(g[32 * hf + 8 * j + 2 * i] + bv.x, g[32 * hf + 8 * j + 2 * i + 1] + bv.y);
                        }
                    }
                    send_box(box, pk, &maps.o, c, row, row < M && c < N, lane);
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the stores have read their boxes
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                      // neither CTA ends while the other may still signal it
    if (tid == 0 && *abort_flag && status) atomicOr(status, 1);
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

template <typename T, bool GATED>
int pair_launch(const void* x, int64_t ldx, const void* w, const void* bias, void* out, int64_t ldo, int64_t M, int K, int N, int dtype, int32_t* status, cudaStream_t stream) {
    using Cfg = PairCfg<GATED>;
    constexpr int BN = Cfg::BN;
    PairMaps maps;
    if (!make_map_2d(&maps.x, x, M, K, ldx, 128, dtype) || !make_map_2d(&maps.w, w, (GATED ? 2 : 1) * (int64_t)N, K, K, BN / 2, dtype) ||
        !make_out_map(&maps.o, out, M, N, ldo, dtype)) return VIG_ERR_DEVICE;
    const int ntn = (N + Cfg::OCOLS - 1) / Cfg::OCOLS, KB = K / PR_BK, all = device_sms() / 2;
    const int64_t ntm = (M + 255) / 256;
    if (ntm * ntn > INT32_MAX) return VIG_ERR_SHAPE;
    // Stationary where the slice of W leaves a deep enough ring, (nearly) all pairs have a column and each a tile at least: K = 384, I = 1024,
    // 25088 rows 31 us against 33, K = 192, I = 512, 262144 rows 94 against 102; with a ring of four boxes it would be the slower one.
    const int xst = (Cfg::RING - KB * Cfg::B) / PR_A;
    const bool stat = xst >= 6 && all / ntn * ntn * 16 >= all * 15 && ntm * ntn >= all;
    const int nst = stat ? (xst < Cfg::MAX_ST ? xst : Cfg::MAX_ST) : Cfg::RING / (PR_A + Cfg::B);
    const int smem = (stat ? KB * Cfg::B + nst * PR_A : nst * (PR_A + Cfg::B)) + Cfg::OUT + Cfg::BARS + 16 + 1024;
    const int64_t pairs = stat ? all / ntn * ntn : ntm * ntn < all ? ntm * ntn : all;
    auto kfn = stat ? gemm_pair_kernel<T, true, GATED> : gemm_pair_kernel<T, false, GATED>;
    const cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(kfn), 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_chained(kfn, dim3(2 * (unsigned)pairs), dim3(Cfg::THREADS), smem, stream, maps, (const T*)bias, (int)M, N, KB, ntn, (int)ntm, nst, status);
}

}  // namespace

int pair_swiglu_launch(const void* x, int64_t ldx, const void* w, void* out, int64_t ldo, int64_t M, int K, int I, int dtype, int32_t* status, cudaStream_t stream) {
    if (dtype == VIG_DTYPE_BF16) return pair_launch<__nv_bfloat16, true>(x, ldx, w, nullptr, out, ldo, M, K, I, dtype, status, stream);
    return pair_launch<__half, true>(x, ldx, w, nullptr, out, ldo, M, K, I, dtype, status, stream);
}

int pair_linear_launch(const void* x, int64_t ldx, const void* w, const void* bias, void* out, int64_t ldo, int64_t M, int K, int N, int dtype, int32_t* status, cudaStream_t stream) {
    if (dtype == VIG_DTYPE_BF16) return pair_launch<__nv_bfloat16, false>(x, ldx, w, bias, out, ldo, M, K, N, dtype, status, stream);
    return pair_launch<__half, false>(x, ldx, w, bias, out, ldo, M, K, N, dtype, status, stream);
}

}  // namespace vig
