// The row-local half of a ViG block of width 192 as one kernel (bf16 / fp16): gating injection, output projection + residual
// add + RMSNorm, gate projection + SwiGLU, down projection + residual add + the next RMSNorm (classification/models/vig.py:
// 444-463, 494-497, 596-618), for calls of up to some ten thousand tokens.
//
// As four kernels these cost 2 + 9 + 8 + 9 us and four launches at 196 tokens, 5 + 10 + 12 + 10 at 8192: each is a chain of
// latencies (launch, tensor-memory allocation, first loads, store and reload of its result) around a microsecond of work.
// Everything here depends on one token only, so a CTA takes R = 16, 32 or 64 tokens through all of it with the
// intermediates in shared memory; the three weight matrices (664 KB) stream from L2 through a ring of 24 KB stages in the
// order they are used, and do not wait for the preceding kernel.  Bound: the stream for R = 16 (one CTA draws about 120 B/ns
// from L2: 5.5 us), the mma.sync rate for R = 64 (21 M multiply-adds per CTA at 1024 a cycle: 11 us); R is the smallest that
// keeps the call in one wave of CTAs.  Where 16-token tiles leave most SMs idle, a cluster of 2 or 4 CTAs shares a tile: each does
// the injection and the output projection for itself (72 KB) and its part of the MLP's features, and the first one adds up the
// others' down projections, which they write into its shared memory in fp32.  Large calls run the tcgen05 kernels, whose MMAs are three times faster per SM.
//
// Roundings are those of the separate kernels: injection, projections, sums, norms and activation are each rounded to the type.
#include "mma_common.cuh"

namespace vig {
namespace {

using namespace tc;

constexpr int BT_C = 192, BT_DV = 64, BT_H = 3, BT_IMAX = 512;
constexpr int BT_STAGE = BT_C * 64 * 2;                   // [192 rows x 64 k], 24 KB
constexpr int BT_THREADS = 288;                           // eight warps that compute, one that loads
constexpr uint32_t BT_PA = BT_C * 2 + 16;                 // row pitches: 16 bytes of padding against bank conflicts
constexpr uint32_t BT_PZ = BT_IMAX * 2 + 16;

struct BtMaps { CUtensorMap wo, wg, wd; };
struct BtParams {
    const void *o, *local, *gate, *gn_w, *ln_w, *residual, *n1_w, *n2_w;
    void *out_r, *out_h;
    int64_t ld_gate;
    int M, I, out_act;
    float inj_eps, n1_eps, n2_eps;
    int32_t* status;
};

__device__ __forceinline__ void bt_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

constexpr int BT_CLUSTER = 4;                             // largest cluster of a tile

template <int RB, bool CL> struct BtSmem {
    static constexpr int NST = CL ? 6 : RB == 1 ? 7 : RB == 2 ? 6 : 4;    // what the token tiles (and partial sums) leave of the 227 KB
    static constexpr uint32_t R = 16 * RB, RING = 0, A = RING + NST * BT_STAGE, RES = A + R * BT_PA, Z = RES + R * BT_PA, PART = Z + R * BT_PZ,
                              SUMS = PART + R * 8 * 4,
                              BAR = SUMS + (CL ? (BT_CLUSTER - 1) * R * BT_C * 4 : 0), BYTES = BAR + 2 * NST * 8 + 16 + 1024;
    static_assert(BYTES <= 227 * 1024, "shared memory");
};

// B fragments of NT neighbouring n tiles (rows of a 128-byte-swizzled weight box) for k step ks (16 values)
template <int NT> __device__ __forceinline__ void bt_load_b(uint32_t (*b)[2], uint32_t box, int row0, int ks, int lane) {
#pragma unroll
    for (int n = 0; n + 1 < NT; n += 2) {
        const uint32_t row = row0 + n * 8 + (lane & 7) + (lane >> 4) * 8, ch = ks * 2 + ((lane >> 3) & 1);
        uint32_t r[4];
        mm::ldsm4(box + row * 128 + ((ch ^ (row & 7)) << 4), r);
        b[n][0] = r[0]; b[n][1] = r[1]; b[n + 1][0] = r[2]; b[n + 1][1] = r[3];
    }
    if constexpr (NT & 1) {
        const uint32_t row = row0 + (NT - 1) * 8 + (lane & 7), ch = ks * 2 + ((lane >> 3) & 1);
        mm::ldsm2(box + row * 128 + ((ch ^ (row & 7)) << 4), b[NT - 1]);
    }
}

// RB: blocks of 16 tokens; WR: warp rows (the other 8 / WR warps share the columns); CL: a cluster's CTAs share a tile
template <typename T, int RB, int WR, bool CL>
__global__ void __launch_bounds__(BT_THREADS, 1) block_tail_kernel(const __grid_constant__ BtMaps maps, const __grid_constant__ BtParams p) {
    using SM = BtSmem<RB, CL>;
    constexpr int NST = SM::NST, R = 16 * RB, WC = 8 / WR, MB = RB / WR, NT = BT_C / WC / 8, FT = 64 / WC / 8;   // row blocks, projection n tiles, feature tiles of a warp
    extern __shared__ uint8_t bt_raw[];
    uint8_t* smem = bt_raw + ((1024u - (smem_u32(bt_raw) & 1023u)) & 1023u);
    const uint32_t sb = smem_u32(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full = sb + SM::BAR, empty = full + 8 * NST;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::BAR + 16 * NST);
    const Waiter waiter{abort_flag, p.status};
    const int IB = p.I / 64;                                 // 64-feature chunks of the MLP
    const int share = CL ? (int)cluster_size() : 1, rank = CL ? (int)cluster_rank() : 0;
    const int c0 = rank * IB / share, c1 = (rank + 1) * IB / share;       // mine
    const int64_t row0 = (int64_t)(blockIdx.x / share) * R;
    const int n = (int)min((int64_t)R, p.M - row0);
    if (tid == 0) {
        for (int s = 0; s < NST; ++s) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, 8); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (CL) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");     // every CTA of the cluster runs before its shared memory is written
    if (warp == 8) {                                         // ---- weights, in the order of use: output projection, 64-feature chunks of the gate projection, down projection
        if (lane == 0) {
            const int T1 = BT_C / 64, T2 = T1 + (c1 - c0) * (BT_C / 64), T3 = T2 + c1 - c0;
            for (int t = 0; t < T3; ++t) {
                const int s = t % NST;
                waiter.wait(empty + 8 * s, ((t / NST) & 1) ^ 1);
                if (*abort_flag) break;
                const uint32_t dst = sb + SM::RING + s * BT_STAGE, bar = full + 8 * s;
                if (t >= T1 && t < T2) {
                    const int c = c0 + (t - T1) / (BT_C / 64), kb = (t - T1) % (BT_C / 64);
                    mbar_expect_tx(bar, 2 * 64 * 128);
                    tma_load_2d(dst, &maps.wg, kb * 64, c * 64, bar);                    // gate rows
                    tma_load_2d(dst + 64 * 128, &maps.wg, kb * 64, p.I + c * 64, bar);   // the matching y rows
                } else {
                    mbar_expect_tx(bar, BT_STAGE);
                    tma_load_2d(dst, t < T1 ? &maps.wo : &maps.wd, (t < T1 ? t : c0 + t - T2) * 64, 0, bar);
                }
            }
        }
        if (CL) {                                            // both cluster barriers are for all threads
            asm volatile("barrier.cluster.wait;" ::: "memory");
            asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
            asm volatile("barrier.cluster.wait;" ::: "memory");
        }
        return;
    }
    pdl_wait();
    const int wr = warp / WC, wc = warp % WC;
    uint8_t* At = smem + SM::A;
    uint8_t* Rt = smem + SM::RES;
    // ---- residual rows (asynchronous), gating injection into the A tile
    for (int i = tid; i < R * (BT_C / 8); i += 256) {
        const int r = i / (BT_C / 8), v = i % (BT_C / 8);
        const T* src = reinterpret_cast<const T*>(p.residual) + (row0 + min(r, n - 1)) * BT_C + v * 8;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(Rt + r * BT_PA + v * 16)), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    {
        const int l8 = tid & 7;
        float wg[8], wl[8];
        { Vec16<T> t; t.load_nc(reinterpret_cast<const T*>(p.gn_w) + l8 * 8); t.to_float(wg); t.load_nc(reinterpret_cast<const T*>(p.ln_w) + l8 * 8); t.to_float(wl); }
#pragma unroll
        for (int it = 0; it < (R * BT_H + 31) / 32; ++it) {      // unrolled: all rows' loads in flight at once
            const int g = it * 32 + (tid >> 3);
            if (R * BT_H % 32 && g >= R * BT_H) break;           // whole warps: R = 16 has 48 groups
            const int r = g / BT_H, col = (g % BT_H) * BT_DV + l8 * 8;
            const int64_t row = row0 + min(r, n - 1);
            Vec16<T> ov, lv, gv;
            ov.load(reinterpret_cast<const T*>(p.o) + row * BT_C + col);
            lv.load(reinterpret_cast<const T*>(p.local) + row * BT_C + col);
            gv.load(reinterpret_cast<const T*>(p.gate) + row * p.ld_gate + col);
            float of[8], lf[8], gf[8], so2 = 0.f, sl2 = 0.f;
            ov.to_float(of); lv.to_float(lf); gv.to_float(gf);
#pragma unroll
            for (int i = 0; i < 8; ++i) { so2 = fmaf(of[i], of[i], so2); sl2 = fmaf(lf[i], lf[i], sl2); }
#pragma unroll
            for (int m = 1; m < 8; m <<= 1) { so2 += __shfl_xor_sync(0xffffffffu, so2, m); sl2 += __shfl_xor_sync(0xffffffffu, sl2, m); }
            const float ro = rsqrtf(so2 * (1.f / BT_DV) + p.inj_eps), rl = rsqrtf(sl2 * (1.f / BT_DV) + p.inj_eps);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float gate = sigmoid_t<T>(gf[i]);
                float val = of[i] * ro * wg[i] * gate + lf[i] * rl * wl[i] * (1.f - gate);
                if (p.out_act) val = val * sigmoid_t<T>(val);
                of[i] = val;
            }
            ov.from_float(of);
            *reinterpret_cast<uint4*>(At + r * BT_PA + col * 2) = *reinterpret_cast<const uint4*>(ov.e);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    bt_sync();
    pdl_launch();

    int t = 0;                                               // weight tiles consumed
    const int frow = 16 * MB * wr + (lane >> 2), fcol = 2 * (lane & 3);
    const uint32_t aA = sb + SM::A + 16 * MB * wr * BT_PA + mm::frag_rows<BT_PA>(lane), aZ = sb + SM::Z + 16 * MB * wr * BT_PZ + mm::frag_rows<BT_PZ>(lane);
    float* part = reinterpret_cast<float*>(smem + SM::PART);

    // acc += A W^T over k boxes of 64: A tile at `a` (pitch PA), my NT n tiles of each 192-row weight box
    auto project = [&](float (*acc)[NT][4], uint32_t a, uint32_t pitch, int boxes) {
#pragma unroll 1
        for (int kb = 0; kb < boxes; ++kb, ++t) {
            const int s = t % NST;
            waiter.wait_lite(full + 8 * s, (t / NST) & 1);
            const uint32_t box = sb + SM::RING + s * BT_STAGE;
            uint32_t fa[2][MB][4], fb[2][NT][2];             // fragments of the next k step load during this one's products
            auto fetch = [&](int ks) {
#pragma unroll
                for (int m = 0; m < MB; ++m) mm::ldsm4(a + m * 16 * pitch + kb * 128 + ks * 32, fa[ks & 1][m]);
                bt_load_b<NT>(fb[ks & 1], box, wc * NT * 8, ks, lane);
            };
            fetch(0);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                if (ks < 3) fetch(ks + 1);
#pragma unroll
                for (int m = 0; m < MB; ++m)
#pragma unroll
                    for (int j = 0; j < NT; ++j) mm::mma_t<T>(acc[m][j], fa[ks & 1][m], fb[ks & 1][j]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive_plain(empty + 8 * s);
        }
    };
    // r = T(T(acc) + residual) into the residual tile, h = T(r rstd w) into the A tile
    auto add_norm = [&](float (*acc)[NT][4], const void* w, float eps) {
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float q = 0.f;
                uint8_t* rp = Rt + (frow + 16 * m + 8 * hf) * BT_PA + (wc * NT * 8 + fcol) * 2;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    uint32_t* cell = reinterpret_cast<uint32_t*>(rp + j * 16);
                    const float2 y = Pack2<T>::unpack(Pack2<T>::pack(acc[m][j][2 * hf], acc[m][j][2 * hf + 1])), res = Pack2<T>::unpack(*cell);
                    const uint32_t r = Pack2<T>::pack(y.x + res.x, y.y + res.y);
                    *cell = r;
                    const float2 rf = Pack2<T>::unpack(r);
                    acc[m][j][2 * hf] = rf.x; acc[m][j][2 * hf + 1] = rf.y;
                    q = fmaf(rf.x, rf.x, q); q = fmaf(rf.y, rf.y, q);
                }
                q += __shfl_xor_sync(0xffffffffu, q, 1);
                q += __shfl_xor_sync(0xffffffffu, q, 2);
                if ((lane & 3) == 0) part[(frow + 16 * m + 8 * hf) * 8 + wc] = q;
            }
        bt_sync();                                           // also: every warp has read its A fragments
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int r = frow + 16 * m + 8 * hf;
                float q = 0.f;
#pragma unroll
                for (int c = 0; c < WC; ++c) q += part[r * 8 + c];
                const float rstd = rsqrtf(q / (float)BT_C + eps);
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const int col = wc * NT * 8 + fcol + j * 8;
                    const float2 wf = Pack2<T>::unpack(__ldg(reinterpret_cast<const uint32_t*>(reinterpret_cast<const T*>(w) + col)));
                    *reinterpret_cast<uint32_t*>(At + r * BT_PA + col * 2) = Pack2<T>::pack(acc[m][j][2 * hf] * rstd * wf.x, acc[m][j][2 * hf + 1] * rstd * wf.y);
                }
            }
        bt_sync();
    };
    float acc[MB][NT][4];
    auto zero = [&]() {
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m][j][e] = 0.f;
    };
    zero();
    project(acc, aA, BT_PA, BT_C / 64);
    add_norm(acc, p.n1_w, p.n1_eps);
    {   // ---- gate projection + SwiGLU: the normalised rows stay in registers, 64 features at a time
        uint32_t fa[BT_C / 16][MB][4];
#pragma unroll
        for (int ks = 0; ks < BT_C / 16; ++ks)
#pragma unroll
            for (int m = 0; m < MB; ++m) mm::ldsm4(aA + m * 16 * BT_PA + ks * 32, fa[ks][m]);
#pragma unroll 1
        for (int c = c0; c < c1; ++c) {
            float g[MB][FT][4], y[MB][FT][4];
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int j = 0; j < FT; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) { g[m][j][e] = 0.f; y[m][j][e] = 0.f; }
#pragma unroll
            for (int kb = 0; kb < BT_C / 64; ++kb, ++t) {
                const int s = t % NST;
                waiter.wait_lite(full + 8 * s, (t / NST) & 1);
                const uint32_t box = sb + SM::RING + s * BT_STAGE;
                uint32_t bg[2][FT][2], by[2][FT][2];
                auto fetch = [&](int ks) {
                    bt_load_b<FT>(bg[ks & 1], box, wc * FT * 8, ks, lane);
                    bt_load_b<FT>(by[ks & 1], box + 64 * 128, wc * FT * 8, ks, lane);
                };
                fetch(0);
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    if (ks < 3) fetch(ks + 1);
#pragma unroll
                    for (int m = 0; m < MB; ++m)
#pragma unroll
                        for (int j = 0; j < FT; ++j) {
                            mm::mma_t<T>(g[m][j], fa[kb * 4 + ks][m], bg[ks & 1][j]);
                            mm::mma_t<T>(y[m][j], fa[kb * 4 + ks][m], by[ks & 1][j]);
                        }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive_plain(empty + 8 * s);
            }
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int j = 0; j < FT; ++j)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        float z[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) { const float gv = g[m][j][2 * hf + e]; z[e] = gv * y[m][j][2 * hf + e] * sigmoid_t<T>(gv); }
                        *reinterpret_cast<uint32_t*>(smem + SM::Z + (frow + 16 * m + 8 * hf) * BT_PZ + (c * 64 + wc * FT * 8 + j * 8 + fcol) * 2) = Pack2<T>::pack(z[0], z[1]);
                    }
        }
    }
    bt_sync();
    zero();
    project(acc, aZ + c0 * 128, BT_PZ, c1 - c0);
    if constexpr (CL) {                                      // the others' sums over their features go to the first CTA
        const uint32_t mine = sb + SM::SUMS + (uint32_t)tid * (MB * NT * 16);
        constexpr uint32_t PER = 256 * MB * NT * 16;         // bytes of a CTA's sums
        asm volatile("barrier.cluster.wait;" ::: "memory");
        if (rank) {
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int j = 0; j < NT; ++j)
                    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(map_rank(mine + (rank - 1) * PER, 0) + (m * NT + j) * 16),
                                 "f"(acc[m][j][0]), "f"(acc[m][j][1]), "f"(acc[m][j][2]), "f"(acc[m][j][3]) : "memory");
        }
        cluster_sync();
        if (rank) {                                          // a wait of this CTA that ran out made its sums wrong
            if (tid == 0 && *abort_flag && p.status) atomicOr(p.status, 1);
            return;
        }
        for (int o = 0; o < share - 1; ++o)
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const float4 v = *reinterpret_cast<const float4*>(smem + SM::SUMS + o * PER + tid * (MB * NT * 16) + (m * NT + j) * 16);
                    acc[m][j][0] += v.x; acc[m][j][1] += v.y; acc[m][j][2] += v.z; acc[m][j][3] += v.w;
                }
    }
    add_norm(acc, p.n2_w, p.n2_eps);
    for (int i = tid; i < n * (BT_C / 8); i += 256) {
        const int r = i / (BT_C / 8), v = i % (BT_C / 8);
        reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out_r) + (row0 + r) * BT_C)[v] = *reinterpret_cast<const uint4*>(Rt + r * BT_PA + v * 16);
        reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out_h) + (row0 + r) * BT_C)[v] = *reinterpret_cast<const uint4*>(At + r * BT_PA + v * 16);
    }
    if (tid == 0 && *abort_flag && p.status) atomicOr(p.status, 1);
}

template <typename T, int RB, int WR> int bt_launch(const BtMaps& maps, const BtParams& p, cudaStream_t st) {
    auto k = block_tail_kernel<T, RB, WR, false>;
    const cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(k), (int)BtSmem<RB, false>::BYTES);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_chained(k, dim3((unsigned)((p.M + 16 * RB - 1) / (16 * RB))), dim3(BT_THREADS), BtSmem<RB, false>::BYTES, st, maps, p);
}

// a cluster of ``share`` CTAs a tile of 16 tokens
template <typename T> int bt_launch_shared(const BtMaps& maps, const BtParams& p, int share, cudaStream_t st) {
    auto k = block_tail_kernel<T, 1, 1, true>;
    const cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(k), (int)BtSmem<1, true>::BYTES);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((p.M + 15) / 16 * share)); cfg.blockDim = dim3(BT_THREADS); cfg.dynamicSmemBytes = BtSmem<1, true>::BYTES; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = share; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chain_launches ? 2 : 1;
    const cudaError_t r = cudaLaunchKernelEx(&cfg, k, maps, p);
    return (int)(r != cudaSuccess ? r : cudaGetLastError());
}

template <typename T> int bt_dispatch(const BtMaps& maps, const BtParams& p, cudaStream_t st) {
    // A tile's CTAs: as many as leave the call in one wave (clusters do not fill every group of SMs, hence seven eighths of the GPU) and have a
    // chunk of features each.  Whole forwards of ViG-T in us with 1 / 2 / 4 / 8 of them: 64 tokens 284 / 266 / 256 / 266, 196 tokens 331 / 313 / 297 / 312 (eight
    // start and meet later), 392 tokens 334 / 317 / 302, 588 tokens 339 / 321 / 386 (148 CTAs in fours are two waves), 980 tokens 345 / 336; with six ring
    // stages instead of four, which clusters of four leave room for, 249, 290, 300, 314 and 330.
    const int tiles = (p.M + 15) / 16;
    for (int share = BT_CLUSTER; share >= 2; share /= 2)
        if (tiles * share * 8 <= device_sms() * 7 && p.I / 64 >= share) return bt_launch_shared<T>(maps, p, share, st);
    // the smallest row tile that is one wave of CTAs; beyond that the largest
    if (p.M <= device_sms() * 16) return bt_launch<T, 1, 1>(maps, p, st);
    if (p.M <= device_sms() * 32) return bt_launch<T, 2, 1>(maps, p, st);
    return bt_launch<T, 4, 2>(maps, p, st);
}

}  // namespace
}  // namespace vig

using namespace vig;

extern "C" int vig_block_tail_supported(int64_t M, int H, int dv, int I, int dtype) {
    if (dtype != VIG_DTYPE_BF16 && dtype != VIG_DTYPE_F16) return 0;
    if (M <= 0 || M >= (1ll << 31) - 64 || H != BT_H || dv != BT_DV || I <= 0 || I % 64 || I > BT_IMAX) return 0;
    return tc::encode_fn() != nullptr;
}

// One wave of 64-token tiles; beyond it the tcgen05 kernels win (12544 tokens: 48 us here, 42 as four kernels; 8192: 26, 36).
extern "C" int vig_block_tail_preferred(int64_t M, int H, int dv, int I, int dtype) {
    return vig_block_tail_supported(M, H, dv, I, dtype) && M <= (int64_t)device_sms() * 64;
}

extern "C" int vig_block_tail_fwd(const void* o, const void* local, const void* gate_logits, int64_t ld_gate, const void* w_gnorm, const void* w_lnorm,
                                  float inject_eps, int out_act_swish, const void* w_o, const void* residual, const void* norm_w, float norm_eps,
                                  const void* w_gate, const void* w_down, const void* next_w, float next_eps, void* out_r, void* out_h,
                                  int64_t M, int H, int dv, int I, int dtype, int32_t* status_dev, void* stream) {
    if (!o || !local || !gate_logits || !w_gnorm || !w_lnorm || !w_o || !residual || !norm_w || !w_gate || !w_down || !next_w || !out_r || !out_h) return VIG_ERR_NULL;
    if (M == 0) return VIG_OK;
    if (!vig_block_tail_supported(M, H, dv, I, dtype)) return VIG_ERR_SHAPE;
    for (const void* x : {o, local, gate_logits, w_gnorm, w_lnorm, w_o, residual, norm_w, w_gate, w_down, next_w, (const void*)out_r, (const void*)out_h})
        if (reinterpret_cast<uintptr_t>(x) & 15) return VIG_ERR_ALIGN;
    if (ld_gate < BT_C || ld_gate % 8) return VIG_ERR_ARG;
    BtMaps maps;
    if (!tc::make_map_2d(&maps.wo, w_o, BT_C, BT_C, BT_C, BT_C, dtype) || !tc::make_map_2d(&maps.wg, w_gate, 2 * (int64_t)I, BT_C, BT_C, 64, dtype) ||
        !tc::make_map_2d(&maps.wd, w_down, BT_C, I, I, BT_C, dtype)) return VIG_ERR_DEVICE;
    BtParams p{o, local, gate_logits, w_gnorm, w_lnorm, residual, norm_w, next_w, out_r, out_h, ld_gate, (int)M, I, out_act_swish, inject_eps, norm_eps, next_eps, status_dev};
    return dtype == VIG_DTYPE_BF16 ? bt_dispatch<__nv_bfloat16>(maps, p, (cudaStream_t)stream) : bt_dispatch<__half>(maps, p, (cudaStream_t)stream);
}
