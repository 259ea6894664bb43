// Backward of the bi-directional gated linear attention on the tensor cores: gradients of q, k, v and of both gate tensors
// (finished: cumulative sums and the derivative of the gate transform included).  Replaces, for the merged operator, the
// reference's FusedChunkGLAFunction.backward (flash-linear-attention/fla/ops/gla/chunk_fuse.py:413-518).
//
// Per scan direction, chunks of 64 tokens, in scan order: G_i inclusive cumulative log-gate, r its value at the chunk's
// middle, l its total, S the state entering the chunk, Z the adjoint state entering it from the far side, c = scale:
//   Qt = c q 2^(G-r),  Kt = k 2^(r-G),  P = mask(dO V^T),  A^T = mask(Kt Qt^T)
//   dQ = c 2^(G-r) (P Kt + dO (2^r S)^T)           dK = 2^(r-G) (P^T Qt + V (2^(l-r) Z)^T)
//   dV = A^T dO + Kt (2^(l-r) Z)                   e  = dQ q - dK k
//   dg_t = <S_next, Z> over value columns + sum of e over the chunk's tokens scanned at or after t
// The first term of dg is the gate gradient just past the chunk: d loss / d g_T = <a_T S_{T-1}, D_T> = <S_{T-1}, Z_T>, so no
// sum ever runs over the whole sequence.  Launches: chunk states (U = (k 2^(l-G))^T V and its adjoint; not for a lone chunk); a scan over
// chunks, where there are more than a few (bwd_fold: fewer are summed by the gradients themselves); chunk gradients; and the exact token-by-token
// kernel, to which a chunk is left whose |G - r| exceeds the range set below (it raises its flag), and which returns at once for every other chunk.
#include "bigla_bwd.cuh"
#include "bigla_exact.cuh"

namespace vig {
namespace {

using namespace mm;
static_assert(C == BWD_CHUNK, "both forms share the workspace");

// ---- chunk states: local S (scan order, from zero) and local Z (against it) of one chunk -----------------------------
template <int DK, int DV, typename T> struct StatesSmem {
    static constexpr uint32_t V = 0, O = V + Terms<T>::RAW * C * Pitch<DV>::B, K = O + Terms<T>::RAW * C * Pitch<DV>::B,
                              Q = K + Terms<T>::SC * C * Pitch<DK>::B, SUM = Q + Terms<T>::SC * C * Pitch<DK>::B, BYTES = SUM + 2 * NT * 4;
};

// Whether a chunk's gates stay in the range of the factorised form, as far as my rows show it.  falling: no log-gate is above
// zero, so that the ends bound what lies between.
template <typename T, int RPG> __device__ __forceinline__ bool in_range(const F2 (&G)[RPG], F2 ref, F2 tot, bool falling) {
    const float lim = range_limit<T>();
    const F2 minus = f2_make(-1.f, -1.f), rest = f2_fma(ref, minus, tot);
    bool fine = fabsf(f2_lo(ref)) <= lim && fabsf(f2_hi(ref)) <= lim && fabsf(f2_lo(rest)) <= lim && fabsf(f2_hi(rest)) <= lim;
    if (!falling) {
#pragma unroll
        for (int r = 0; r < RPG; ++r) {
            const F2 y = f2_fma(ref, minus, G[r]);
            fine = fine && fabsf(f2_lo(y)) <= lim && fabsf(f2_hi(y)) <= lim;
        }
    }
    return fine;
}

// States of a chunk outside that range, token by token: half of the threads run S, half its adjoint.  (As 2^(l-G) they are NaN
// after a log-gate of -inf, and lose digits with large gates: the rounding of G grows with it.)  sm: the K and Q tiles.
template <int DK, int DV, typename T> struct ExactStates {
    using L = rec::Lay<DK, DV, NT>;
    static constexpr int SUB = 16, ROW = 3 * DK + DV;                    // tokens staged at a time, floats of a token
    static_assert(L::HALVES == 2 && 2 * SUB * ROW * 4 <= 2 * Terms<T>::SC * C * Pitch<DK>::B, "staged rows fit the scaled tiles");
};
template <int DK, int DV, typename T> __device__ __noinline__ void exact_states(const BwdParams& p, float* sm, int bh, int c, int dir, int n) {
    using E = ExactStates<DK, DV, T>;
    using L = typename E::L;
    const int b = bh / p.H, h = bh % p.H, d0 = L::d0(), j0 = L::j0(), tid = threadIdx.x % L::HT, blocks = (n + E::SUB - 1) / E::SUB;
    const bool adj = L::half() == 1, down = (dir != 0) != adj;           // the adjoint runs against the scan order
    float *sa = sm + L::half() * E::SUB * E::ROW, *sg = sa + E::SUB * DK, *sk = sg + E::SUB * DK, *sv = sk + E::SUB * DK;
    float S[L::JPT][L::DPT], sum = 0.f;
#pragma unroll
    for (int j = 0; j < L::JPT; ++j)
#pragma unroll
        for (int d = 0; d < L::DPT; ++d) S[j][d] = 0.f;
    for (int bb = 0; bb < blocks; ++bb) {
        const int at = (down ? blocks - 1 - bb : bb) * E::SUB, m = min(E::SUB, n - at);
        const int64_t t = (int64_t)c * C + at;
        __syncthreads();
        rec::stage<DK, DV, L::HT, T>(nullptr, sk, sv, sg, sa, nullptr, 0, 0.f, adj ? head_ptr<T>(p.q, p.sq, b, h, t) : head_ptr<T>(p.k, p.sk, b, h, t), adj ? p.sq[2] : p.sk[2],
                                     adj ? p.c : 1.f, adj ? head_ptr<T>(p.dout, p.sdo, b, h, t) : head_ptr<T>(p.v, p.sv, b, h, t), adj ? p.sdo[2] : p.sv[2],
                                     dir ? head_ptr<T>(p.gb, p.sgb, b, h, t) : head_ptr<T>(p.gf, p.sgf, b, h, t), dir ? p.sgb[2] : p.sgf[2], m, p.gate_norm, p.clamp_min, tid);
        __syncthreads();
        if (tid < DK) for (int i = 0; i < m; ++i) sum += sg[i * DK + tid];
        if (adj) rec::each(m, down, [&](int i) { rec::update_adjoint(S, sa + i * DK + d0, sk + i * DK + d0, sv + i * DV + j0); });
        else rec::each(m, down, [&](int i) { rec::update(S, sa + i * DK + d0, sk + i * DK + d0, sv + i * DV + j0); });
    }
    const size_t slot = ((size_t)bh * p.nchunk + c) * 2 + dir;
    float* out = (adj ? p.ws_Z : p.ws_S) + slot * DK * DV;
#pragma unroll
    for (int j = 0; j < L::JPT; ++j)
#pragma unroll
        for (int d = 0; d < L::DPT; ++d) out[(d0 + d) * DV + j0 + j] = S[j][d];
    if (!adj && tid < DK) p.ws_decay[slot * DK + tid] = sum * tc::LOG2E;
}

// CTAs an SM as the registers of the factored form allow; the exact one, which nobody waits for, has to live with them
template <int DK, int DV, typename T> constexpr int states_min_blocks() {
    return DK * DV == 4096 ? (sizeof(T) == 4 ? 1 : 2) : DK * DV == 2048 ? (sizeof(T) == 4 ? 2 : 3) : DK * DV == 1024 ? (sizeof(T) == 4 ? 3 : 4)
           : std::is_same<T, __nv_bfloat16>::value ? 5 : 4;
}

template <int DK, int DV, typename T>
__global__ void __launch_bounds__(NT, states_min_blocks<DK, DV, T>()) bwd_states_mma_kernel(const __grid_constant__ BwdParams p) {
    using CL = ColLay<DK>;
    using SM = StatesSmem<DK, DV, T>;
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
    const bool one_dir = gridDim.z != 1;
    Raw2<T> x[CL::RPG], q[CL::RPG], k[CL::RPG];
    auto load_gate = [&](int dir) {
        load_rows(x, (dir ? head_ptr<T>(p.gb, p.sgb, b, h, t0) : head_ptr<T>(p.gf, p.sgf, b, h, t0)) + 2 * pr, dir ? p.sgb[2] : p.sgf[2], r0, n);
    };
    const int first = one_dir ? blockIdx.z : p.dir_mask & 1 ? 0 : 1;
    pdl_launch();
    load_gate(first);
    load_rows(k, head_ptr<T>(p.k, p.sk, b, h, t0) + 2 * pr, p.sk[2], r0, n);
    load_rows(q, head_ptr<T>(p.q, p.sq, b, h, t0) + 2 * pr, p.sq[2], r0, n);
    float mark = 0.f;
    load_raw<T, DV, RAW>(smem + SM::V, head_ptr<T>(p.v, p.sv, b, h, t0), p.sv[2], n, mark);
    load_raw<T, DV, RAW>(smem + SM::O, head_ptr<T>(p.dout, p.sdo, b, h, t0), p.sdo[2], n, mark);
    zero_rows(k, r0, n); zero_rows(q, r0, n);
    F2 seen = f2_make(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < CL::RPG; ++r) { see(seen, k[r].f2()); see(seen, q[r].f2()); }
    bool finite = clean(seen);
    const int last = one_dir ? first : p.dir_mask & 2 ? 1 : 0;
    int exact = 0;                                                       // directions left to the exact form, after the loop: nothing of it lives across the call
    for (int dir = first; dir <= last; ++dir) {
        const size_t slot = ((size_t)bh * p.nchunk + c) * 2 + dir;
        F2 G[CL::RPG], ref, tot;
        cum_gates<DK, T>(G, ref, tot, gsum, x, n, dir, p.gate_norm, p.clamp_min);
        if (dir < last) load_gate(dir + 1);
        if (r0 == 0) *reinterpret_cast<F2*>(p.ws_decay + slot * DK + 2 * pr) = tot;
        const F2 minus = f2_make(-1.f, -1.f), cc = f2_make(p.c, p.c);
#pragma unroll
        for (int r = 0; r < CL::RPG; ++r) {
            const F2 y = f2_fma(G[r], minus, tot);
            uint32_t t[SC];
            const F2 ks = f2_mul(k[r].f2(), f2_make(ex2_t<T>(f2_lo(y)), ex2_t<T>(f2_hi(y))));
            split2<SC>(f2_lo(ks), f2_hi(ks), t);
#pragma unroll
            for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(smem + SM::K + i * C * Pitch<DK>::B + (r0 + r) * Pitch<DK>::B + pr * 4) = t[i];
            const F2 qs = f2_mul(f2_mul(q[r].f2(), cc), f2_make(ex2_t<T>(f2_lo(G[r])), ex2_t<T>(f2_hi(G[r]))));
            split2<SC>(f2_lo(qs), f2_hi(qs), t);
#pragma unroll
            for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(smem + SM::Q + i * C * Pitch<DK>::B + (r0 + r) * Pitch<DK>::B + pr * 4) = t[i];
        }
        wait_raw();
        if (dir == first) finite = finite && raw_clean<T, DV, RAW>(smem + SM::V, mark) && raw_clean<T, DV, RAW>(smem + SM::O, mark);
        if (__syncthreads_or(!finite || !in_range<T>(G, ref, tot, sizeof(T) == 2 && p.gate_norm > 0.f))) {
            exact |= 1 << dir;
            continue;
        }
        const int which = warp >> 2, mt = (warp & 3) % MT, wn = (warp & 3) / MT;          // warps 0 - 3: S, 4 - 7: Z
        float acc[NTL][4];
#pragma unroll
        for (int i = 0; i < NTL; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
        state_mma<DK, DV, SC, RAW, NTL>(acc, sb + (which ? SM::Q : SM::K) + mt * 32, sb + (which ? SM::O : SM::V) + wn * NC * 2, lane);
        float* out = (which ? p.ws_Z : p.ws_S) + slot * DK * DV + (mt * 16 + (lane >> 2)) * DV + wn * NC + 2 * (lane & 3);
#pragma unroll
        for (int i = 0; i < NTL; ++i) {
            *reinterpret_cast<float2*>(out + i * 8) = make_float2(acc[i][0], acc[i][1]);
            *reinterpret_cast<float2*>(out + 8 * DV + i * 8) = make_float2(acc[i][2], acc[i][3]);
        }
        __syncthreads();
    }
    if (exact) {
#pragma unroll 1
        for (int dir = first; dir <= last; ++dir)
            if (exact >> dir & 1) exact_states<DK, DV, T>(p, reinterpret_cast<float*>(smem + SM::K), bh, c, dir, n);
    }
}

// ---- scan over chunks: local states -> entering states, in place.  S in scan order, Z against it. ---------------------
__global__ void __launch_bounds__(256, 2) bwd_scan_kernel(const __grid_constant__ BwdParams p) {
    pdl_launch();
    pdl_wait();
    const int per = p.dk * p.dv / 4;
    const int64_t it = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int e = (int)(it % per);
    int64_t r = it / per;
    const int which = (int)(r & 1); r >>= 1;
    const int ndir = p.dir_mask == 3 ? 2 : 1;
    const int dir = p.dir_mask == 3 ? (int)(r % 2) : p.dir_mask - 1;
    const int64_t bh = r / ndir;
    if (bh >= (int64_t)p.B * p.H) return;
    const bool descending = (dir != 0) != (which != 0);
    float gsum = 0.f;
    scan_states(reinterpret_cast<float4*>(which ? p.ws_Z : p.ws_S), p.ws_decay, per, e, p.dk, e * 4 / p.dv, p.nchunk, make_float4(0.f, 0.f, 0.f, 0.f), gsum,
                [&](int cc) { return ((size_t)bh * p.nchunk + (descending ? p.nchunk - 1 - cc : cc)) * 2 + dir; }, [](float g) { return exp2f(g); });
}

// the same on a workspace that is not aligned to 16 bytes (vig_bigla_bwd takes any): value by value
__global__ void __launch_bounds__(256) bwd_scan_unaligned_kernel(const __grid_constant__ BwdParams p) {
    pdl_launch();
    pdl_wait();
    const int per = p.dk * p.dv, ndir = p.dir_mask == 3 ? 2 : 1;
    const int64_t it = (int64_t)blockIdx.x * 256 + threadIdx.x, r = it / per;
    const int e = (int)(it % per), which = (int)(r & 1), dir = p.dir_mask == 3 ? (int)(r / 2 % 2) : p.dir_mask - 1;
    const int64_t bh = r / 2 / ndir;
    if (bh >= (int64_t)p.B * p.H) return;
    const bool descending = (dir != 0) != (which != 0);
    float S = 0.f;
    for (int cc = 0; cc < p.nchunk; ++cc) {
        const size_t slot = ((size_t)bh * p.nchunk + (descending ? p.nchunk - 1 - cc : cc)) * 2 + dir;
        float* at = (which ? p.ws_Z : p.ws_S) + slot * per + e;
        const float u = __ldcg(at);
        __stcg(at, S);
        S = fmaf(S, exp2f(__ldcg(p.ws_decay + slot * p.dk + e / p.dv)), u);
    }
}

// ---- chunk gradients -----------------------------------------------------------------------------------------------
template <int DK, int DV, typename T> struct GradSmem {
    static constexpr uint32_t EP = DK + 8, VP = DV + 8;                // row pitches of the fp32 tiles (floats)
    static constexpr uint32_t TQ = Terms<T>::SC * C * Pitch<DK>::B, TS = Terms<T>::SC * DK * Pitch<DV>::B, TD = C * VP * 4;
    static constexpr uint32_t V = 0, O = V + Terms<T>::RAW * C * Pitch<DV>::B, K = O + Terms<T>::RAW * C * Pitch<DV>::B,
                              Q = K + TQ, S = Q + TQ, Z = S + TS, X = S + (2 * TS > TD ? 2 * TS : TD), SUM = X + C * DK * 4, CARRY = SUM + NT * 8,
                              SCL = CARRY + DK * 4, BAR = SCL + 2 * DK * 4, BYTES = BAR + 16,
                              SENT = C * DK * 4 + C / 2 * DV * 4;       // what arrives from the other direction: dq or dk, half of dv's rows
    static_assert(C * EP * 4 <= TQ && TD <= K - V && C / 2 * DV * 4 <= TQ, "the fp32 tiles reuse the operand tiles");
};

// The barrier orders no data here (what it protects has been read before; what is sent carries its own count): an arrival
// that releases waits for every access of the warp, 2500 cycles each time.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// 16 bytes into the other CTA's shared memory; its barrier counts them
__device__ __forceinline__ void send(uint32_t at, float a, float b, float c, float d, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(at), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}

// The contributions of the first m chunks, from the sequence's start or (down) from its end, into the state behind them: what bwd_scan_kernel
// leaves in the chunk that follows, the same operations in the same order.
template <int DK, int DV> __device__ __forceinline__ void sum_states(float4 (&S)[StateLay<DK, DV>::KN], const BwdParams& p, const float* U, int bh, int dir, int down, int m) {
    using ST = StateLay<DK, DV>;
#pragma unroll
    for (float4& s : S) s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int g = 0; g < m; ++g) {
        const size_t slot = ((size_t)bh * p.nchunk + (down ? p.nchunk - 1 - g : g)) * 2 + dir;
        float4 u[ST::KN];
        float a[ST::KN];
        fetch_state<DK, DV>(u, U + slot * DK * DV);
#pragma unroll
        for (int k = 0; k < ST::KN; ++k) a[k] = __ldcg(p.ws_decay + slot * DK + (threadIdx.x + k * NT) / ST::TPR);
#pragma unroll
        for (int k = 0; k < ST::KN; ++k) {
            const float e = exp2f(a[k]);
            S[k].x = fmaf(S[k].x, e, u[k].x); S[k].y = fmaf(S[k].y, e, u[k].y); S[k].z = fmaf(S[k].z, e, u[k].z); S[k].w = fmaf(S[k].w, e, u[k].w);
        }
    }
}

// CTAs an SM as shared memory has room for, where that leaves the registers that the products need (bf16 at 32 / 64: three are
// 2 % faster than two, at 80 registers instead of 128)
template <int DK, int DV, typename T> constexpr int grads_min_blocks() {
    return sizeof(T) == 4 ? 1 : DK == 64 ? 2 : DK * DV == 2048 ? (std::is_same<T, __half>::value ? 2 : 3) : DK == 32 ? 3 : 4;
}

// A CTA forms one chunk's gradients of one direction; with both, the two CTAs of a cluster add them up through each other's
// shared memory, one finishing dq, the other dk, each half of the rows of dv.  Both directions in turn in one CTA keep dq, dk
// and dv of the first, 64 of 128 registers at 64 / 64, alive through the products of the second: the spills were as long as the
// second reading of v and dO is now, and left no registers to ask for the states ahead of a barrier or to keep q, k and the gates
// (backward of 8 x 6 x 4096, bf16: 513 -> 488 us; 128 x 6 x 196: 531 -> 499; 128 x 3 x 196, 32 / 64, where nothing spilled, 148 -> 150).
// Bound, 64 / 64 in 16 bits: latency at 16 warps an SM and shared memory's rate (59 % of it; ldmatrix two thirds of that); the tensor pipe is 27 % busy.
// Smaller heads have 24 or 32 warps an SM (grads_min_blocks), fp32 has 8.
// Eight warps: warps 0 - 3 form dQ and dV inside the chunk, warps 4 - 7 dK and the state's part of dV, 16 rows each: 160 - 288
// products a warp and direction; dV on the other side makes it 136 - 352.  What follows the products -- the factors 2^(G-r), e
// and its sums -- is done by channel pairs, in which q, k and the gates are read coalesced.
// SUM: the contributions are summed here (a form of its own: the other one is 1.5 % slower with this code among its instructions)
template <int DK, int DV, typename T, bool SUM>
__global__ void __launch_bounds__(NT, grads_min_blocks<DK, DV, T>()) bwd_grads_mma_kernel(const __grid_constant__ BwdParams p) {
    using CL = ColLay<DK>;
    using SM = GradSmem<DK, DV, T>;
    using ST = StateLay<DK, DV>;
    constexpr int RAW = Terms<T>::RAW, SC = Terms<T>::SC, RPG = CL::RPG;
    constexpr uint32_t PK = Pitch<DK>::B, PV = Pitch<DV>::B;
    constexpr uint32_t TK = C * PK, TV = C * PV, TS = DK * PV;          // bytes from one term's tile to the next
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t sb = tc::smem_u32(smem);
    F2* X = reinterpret_cast<F2*>(smem + SM::X);                        // [RPG][NT]: 2^(G-r) of each thread's rows, private; then what the other direction sends
    float* gsum = reinterpret_cast<float*>(smem + SM::SUM);
    float* carry = reinterpret_cast<float*>(smem + SM::CARRY);
    float* scl = reinterpret_cast<float*>(smem + SM::SCL);              // [0]: 2^r, [1]: 2^(l-r)
    float* EQ = reinterpret_cast<float*>(smem + SM::Q);                 // dQ, dK once the products are done
    float* EK = reinterpret_cast<float*>(smem + SM::K);
    const int lane = threadIdx.x & 31, role = threadIdx.x >> 7, w = (threadIdx.x >> 5) & 3;
    const bool both = p.dir_mask == 3;
    const int dir = both ? blockIdx.x & 1 : p.dir_mask - 1;
    const int c = both ? blockIdx.x >> 1 : blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H;
    const int64_t t0 = (int64_t)c * C;
    const int n = min(C, p.L - (int)t0);
    const int pr = threadIdx.x % CL::PAIRS, gr = threadIdx.x / CL::PAIRS, r0 = gr * RPG;
    const int fr = 16 * w + (lane >> 2), fc = 2 * (lane & 3);           // my fragment rows fr, fr + 8; columns 8 nt + fc, + 1
    const T* qp = head_ptr<T>(p.q, p.sq, b, h, t0) + 2 * pr;
    const T* kp = head_ptr<T>(p.k, p.sk, b, h, t0) + 2 * pr;
    const T* gp = (dir ? head_ptr<T>(p.gb, p.sgb, b, h, t0) : head_ptr<T>(p.gf, p.sgf, b, h, t0)) + 2 * pr;
    const int64_t sgl = dir ? p.sgb[2] : p.sgf[2];
    const size_t slot = ((size_t)bh * p.nchunk + c) * 2 + dir;
    const F2 cc = f2_make(p.c, p.c), minus = f2_make(-1.f, -1.f), zero = f2_make(0.f, 0.f);
    const bool have_states = p.nchunk > 1;
    bool bad;
    pdl_launch();
    if (both && threadIdx.x == 0) {
        tc::mbar_init(sb + SM::BAR, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc::mbar_expect_tx(sb + SM::BAR, SM::SENT);
    }
    Raw2<T> x[RPG], q[RPG], k[RPG];
    {   // ---- gates, scaled operand tiles
        load_rows(x, gp, sgl, r0, n);
        load_rows(q, qp, p.sq[2], r0, n);
        load_rows(k, kp, p.sk[2], r0, n);
        float mark = 0.f;
        load_raw<T, DV, RAW>(smem + SM::V, head_ptr<T>(p.v, p.sv, b, h, t0), p.sv[2], n, mark);
        load_raw<T, DV, RAW>(smem + SM::O, head_ptr<T>(p.dout, p.sdo, b, h, t0), p.sdo[2], n, mark);
        F2 G[RPG], ref, tot;
        cum_gates<DK, T>(G, ref, tot, gsum, x, n, dir, p.gate_norm, p.clamp_min);
        zero_rows(q, r0, n); zero_rows(k, r0, n);
        F2 seen = zero;
        const float lim = range_limit<T>();
        const F2 rest = f2_fma(ref, minus, tot);
        bool fine = fabsf(f2_lo(ref)) <= lim && fabsf(f2_hi(ref)) <= lim && fabsf(f2_lo(rest)) <= lim && fabsf(f2_hi(rest)) <= lim;
        if (gr == 0) {
            *reinterpret_cast<float2*>(scl + 2 * pr) = make_float2(ex2_t<T>(f2_lo(ref)), ex2_t<T>(f2_hi(ref)));
            *reinterpret_cast<float2*>(scl + DK + 2 * pr) = make_float2(ex2_t<T>(f2_lo(rest)), ex2_t<T>(f2_hi(rest)));
        }
#pragma unroll
        for (int r = 0; r < RPG; ++r) {
            const F2 y = f2_fma(ref, minus, G[r]);
            fine = fine && fabsf(f2_lo(y)) <= lim && fabsf(f2_hi(y)) <= lim;
            const F2 ex = f2_make(ex2_t<T>(f2_lo(y)), ex2_t<T>(f2_hi(y)));
            X[r * NT + threadIdx.x] = ex;
            see(seen, q[r].f2()); see(seen, k[r].f2());
            uint32_t t[SC];
            const F2 qs = f2_mul(f2_mul(q[r].f2(), cc), ex), ks = f2_mul(k[r].f2(), f2_make(ex2_t<T>(-f2_lo(y)), ex2_t<T>(-f2_hi(y))));
            split2<SC>(f2_lo(qs), f2_hi(qs), t);
#pragma unroll
            for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(smem + SM::Q + i * TK + (r0 + r) * PK + pr * 4) = t[i];
            split2<SC>(f2_lo(ks), f2_hi(ks), t);
#pragma unroll
            for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(smem + SM::K + i * TK + (r0 + r) * PK + pr * 4) = t[i];
        }
        pdl_wait();                                                      // all of the above read the call's inputs only
        const int next = dir ? c - 1 : c + 1;                           // the chunk scanned after this one
        float4 st[ST::KN], adj[ST::KN], ahead[ST::KN];
        if (SUM && ST::mine()) {
            sum_states<DK, DV>(st, p, p.ws_S, bh, dir, dir, dir ? p.nchunk - 1 - c : c);
            sum_states<DK, DV>(adj, p, p.ws_Z, bh, dir, dir ^ 1, dir ? c : p.nchunk - 1 - c);
            fetch_state<DK, DV>(ahead, p.ws_S + slot * DK * DV);
#pragma unroll
            for (int k = 0; k < ST::KN; ++k) {
                const float a = exp2f(__ldcg(p.ws_decay + slot * DK + (threadIdx.x + k * NT) / ST::TPR));
                ahead[k].x = fmaf(st[k].x, a, ahead[k].x); ahead[k].y = fmaf(st[k].y, a, ahead[k].y);
                ahead[k].z = fmaf(st[k].z, a, ahead[k].z); ahead[k].w = fmaf(st[k].w, a, ahead[k].w);
            }
            if (next < 0 || next >= p.nchunk) {
#pragma unroll
                for (float4& v : ahead) v = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        } else if (!SUM && have_states && ST::mine()) {                  // asked for ahead of the barrier that the tiles need
            fetch_state<DK, DV>(st, p.ws_S + slot * DK * DV);
            fetch_state<DK, DV>(adj, p.ws_Z + slot * DK * DV);
            if (next >= 0 && next < p.nchunk) {
                fetch_state<DK, DV>(ahead, p.ws_S + (((size_t)bh * p.nchunk + next) * 2 + dir) * DK * DV);
            } else {
#pragma unroll
                for (float4& v : ahead) v = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        wait_raw();
        const bool finite = raw_clean<T, DV, RAW>(smem + SM::V, mark) && raw_clean<T, DV, RAW>(smem + SM::O, mark) && clean(seen);
        bad = __syncthreads_or(!fine || !finite);
        if (!bad && have_states) {
            if (ST::mine()) {
                put_state<DK, DV, SC>(smem + SM::S, st, scl);
                put_state<DK, DV, SC>(smem + SM::Z, adj, scl + DK);
                state_dots<DK, DV>(carry, adj, ahead);
            }
            __syncthreads();
        }
    }
    F2 dq[RPG], dk[RPG], e[RPG];
    if (!bad) {
        float acc[DK / 8][4], dv[DV / 8][4];
#pragma unroll
        for (int i = 0; i < DK / 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll
        for (int i = 0; i < DV / 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dv[i][j] = 0.f;
        const uint32_t aV = sb + SM::V + 16 * w * PV + frag_rows<PV>(lane), aO = sb + SM::O + 16 * w * PV + frag_rows<PV>(lane);
        const uint32_t aK = sb + SM::K + 16 * w * PK + frag_rows<PK>(lane);
        const uint32_t bV = sb + SM::V + frag_cols<PV>(lane), bO = sb + SM::O + frag_cols<PV>(lane), bQ = sb + SM::Q + frag_cols<PK>(lane);
        const uint32_t tK = sb + SM::K + frag_rows<PK>(lane), tQ = sb + SM::Q + frag_rows<PK>(lane), tO = sb + SM::O + frag_rows<PV>(lane);
        uint32_t mine[DV / 16][RAW][4];                                  // my rows of dO (of V): operand of every block and of the state's product
        load_a<DV, RAW>(mine, role ? aV : aO, TV);
        if (role == 0) {                                                 // ---- dQ and dV inside the chunk
#pragma unroll 1
            for (int jb = dir ? w : 0; jb < (dir ? C / 16 : w + 1); ++jb) {   // 16-token blocks scanned at or before my rows
                float pb[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                uint32_t ap[SC][4];
                block_nt<DV, RAW, RAW>(pb, mine, bV + jb * 16 * PV, TV);
                mask_split<SC>(pb, jb == w, lane, [&](int r, int j) { return dir ? j >= r : j <= r; }, ap);
                block_nn<DK, SC, SC>(acc, ap, tK + jb * 16 * PK, TK);
            }
            if (have_states) rows_nt<DK, DV, PV, RAW, SC>(acc, mine, sb + SM::S + frag_cols<PV>(lane), TS);
#pragma unroll 1
            for (int ib = dir ? 0 : w; ib < (dir ? w + 1 : C / 16); ++ib) {   // blocks scanned at or after them
                float pb[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                uint32_t ap[SC][4];
                block_nt<DK, SC, SC>(pb, aK, TK, bQ + ib * 16 * PK, TK);
                mask_split<SC>(pb, ib == w, lane, [&](int j, int i) { return dir ? i <= j : i >= j; }, ap);
                block_nn<DV, SC, RAW>(dv, ap, tO + ib * 16 * PV, TV);
            }
        } else {                                                         // ---- dK, and the state's part of dV
#pragma unroll 1
            for (int ib = dir ? 0 : w; ib < (dir ? w + 1 : C / 16); ++ib) {
                float pb[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                uint32_t ap[SC][4];
                block_nt<DV, RAW, RAW>(pb, mine, bO + ib * 16 * PV, TV);
                mask_split<SC>(pb, ib == w, lane, [&](int j, int i) { return dir ? i <= j : i >= j; }, ap);
                block_nn<DK, SC, SC>(acc, ap, tQ + ib * 16 * PK, TK);
            }
            if (have_states) {
                rows_nt<DK, DV, PV, RAW, SC>(acc, mine, sb + SM::Z + frag_cols<PV>(lane), TS);
                const uint32_t tZ = sb + SM::Z + frag_rows<PV>(lane);
#pragma unroll
                for (int ks = 0; ks < DK / 16; ++ks) {
                    uint32_t fa[SC][4];
#pragma unroll
                    for (int t = 0; t < SC; ++t) ldsm4(aK + t * TK + ks * 32, fa[t]);
                    block_nn<DV, SC, SC>(dv, fa, tZ + ks * 16 * PV, TS);
                }
            }
        }
        __syncthreads();                                                 // the operand tiles are read
        {
            float* E = (role ? EK : EQ) + fr * SM::EP + fc;
            float* D = reinterpret_cast<float*>(smem + (role ? SM::S : SM::V)) + fr * SM::VP + fc;
#pragma unroll
            for (int i = 0; i < DK / 8; ++i) {
                *reinterpret_cast<float2*>(E + 8 * i) = make_float2(acc[i][0], acc[i][1]);
                *reinterpret_cast<float2*>(E + 8 * SM::EP + 8 * i) = make_float2(acc[i][2], acc[i][3]);
            }
#pragma unroll
            for (int i = 0; i < DV / 8; ++i) {
                *reinterpret_cast<float2*>(D + 8 * i) = make_float2(dv[i][0], dv[i][1]);
                *reinterpret_cast<float2*>(D + 8 * SM::VP + 8 * i) = make_float2(dv[i][2], dv[i][3]);
            }
        }
        __syncthreads();
        // ---- by channel pairs: dq, dk, e, and the gate gradient = sum of e over the tokens scanned at or after t plus the value just past the chunk
        F2 sum = zero;
#pragma unroll
        for (int r = 0; r < RPG; ++r) {
            const F2 ex = X[r * NT + threadIdx.x];
            dq[r] = f2_mul(f2_mul(*reinterpret_cast<const F2*>(EQ + (r0 + r) * SM::EP + 2 * pr), ex), cc);
            dk[r] = f2_mul(*reinterpret_cast<const F2*>(EK + (r0 + r) * SM::EP + 2 * pr), f2_make(tc::rcp(f2_lo(ex)), tc::rcp(f2_hi(ex))));
            e[r] = f2_fma(f2_mul(dk[r], minus), k[r].f2(), f2_mul(dq[r], q[r].f2()));
            sum = f2_add(sum, e[r]);
        }
        *reinterpret_cast<F2*>(gsum + gr * DK + 2 * pr) = sum;
        __syncthreads();
        if (both) cluster_arrive();                                      // my X and K tiles may be written by the other direction
        F2 run = have_states ? *reinterpret_cast<const F2*>(carry + 2 * pr) : zero;
#pragma unroll
        for (int o = 0; o < CL::GROUPS; ++o)
            if (dir ? o < gr : o > gr) run = f2_add(run, *reinterpret_cast<const F2*>(gsum + o * DK + 2 * pr));
        // static register indices for both orders: the backward direction sums upwards, the forward one downwards
        if (dir) {
#pragma unroll
            for (int r = 0; r < RPG; ++r) e[r] = run = f2_add(run, e[r]);
        } else {
#pragma unroll
            for (int r = RPG - 1; r >= 0; --r) e[r] = run = f2_add(run, e[r]);
        }
        rows_through_gate(e, x, p.gate_norm, p.clamp_min);
    } else {                                                             // the other direction waits for its share all the same
#pragma unroll
        for (int r = 0; r < RPG; ++r) dq[r] = dk[r] = zero;
        if (both) cluster_arrive();
    }
    // ---- the other direction's share: rank 0 (forward) finishes dq and rows 0 - 31 of dv, rank 1 dk and rows 32 - 63
    constexpr int VPT = C / 2 * DV / NT, VTR = DV / VPT;                 // columns of dv a thread sends or finishes, threads of a row
    const int vr = threadIdx.x / VTR, vc = threadIdx.x % VTR * VPT;
    const float* D0 = reinterpret_cast<const float*>(smem + SM::V);
    const float* D1 = reinterpret_cast<const float*>(smem + SM::S);
    if (both) {
        cluster_wait();
        const uint32_t peer = tc::map_rank(sb, dir ^ 1), bar = peer + SM::BAR;
#pragma unroll
        for (int r = 0; r < RPG; r += 2) {
            const F2 u = dir ? dq[r] : dk[r], v = dir ? dq[r + 1] : dk[r + 1];
            send(peer + SM::X + (r / 2 * NT + threadIdx.x) * 16, f2_lo(u), f2_hi(u), f2_lo(v), f2_hi(v), bar);
        }
        const int row = vr + (dir ? 0 : C / 2);
#pragma unroll
        for (int i = 0; i < VPT; i += 4) {
            const float4 a = *reinterpret_cast<const float4*>(D0 + row * SM::VP + vc + i), z = *reinterpret_cast<const float4*>(D1 + row * SM::VP + vc + i);
            send(peer + SM::K + (vr * DV + vc + i) * 4, a.x + z.x, a.y + z.y, a.z + z.z, a.w + z.w, bar);
        }
        cluster_arrive();                                                // my share is on its way
    }
    if (!bad) {
        T* out = reinterpret_cast<T*>(dir ? p.dgb : p.dgf) + ((int64_t)bh * p.L + t0 + r0) * DK + 2 * pr;
#pragma unroll
        for (int r = 0; r < RPG; ++r)
            if (r0 + r < n) store2<T>(out + r * DK, f2_lo(e[r]), f2_hi(e[r]));
    }
    if (both) {
        // No way out ahead of the other direction's sends, which write into this CTA's shared memory.  What is left to wait for are stores under way:
        // should they take a second, the chunk is left to the exact form like one out of range.
        cluster_wait();
        int tries = 0;
        while (!tc::mbar_try_wait_parked(sb + SM::BAR, 0, 2000u) && tries < 1 << 19) ++tries;
        bad = __syncthreads_or(bad || tries >= 1 << 19);
    }
    // a half of the flag for each direction: a chunk that either leaves is left whole, outputs included
    if (threadIdx.x == 0) {
        int32_t* flag = p.flags + (size_t)bh * p.nchunk + c;
        if (both) reinterpret_cast<int16_t*>(flag)[dir] = bad;
        else *flag = bad;
    }
    if (bad) return;
    const int64_t base = ((int64_t)bh * p.L + t0 + r0) * DK + 2 * pr;
#pragma unroll
    for (int r = 0; r < RPG; ++r) {
        if (r0 + r < n) {
            if (both) {
                const F2 v = f2_add(dir ? dk[r] : dq[r], X[(r / 2 * NT + threadIdx.x) * 2 + (r & 1)]);
                store2<T>(reinterpret_cast<T*>(dir ? p.out_dk : p.out_dq) + base + r * DK, f2_lo(v), f2_hi(v));
            } else {
                store2<T>(reinterpret_cast<T*>(p.out_dq) + base + r * DK, f2_lo(dq[r]), f2_hi(dq[r]));
                store2<T>(reinterpret_cast<T*>(p.out_dk) + base + r * DK, f2_lo(dk[r]), f2_hi(dk[r]));
            }
        }
    }
    const float* sent = reinterpret_cast<const float*>(smem + SM::K) + vr * DV + vc;
    for (int row = vr + (both && dir ? C / 2 : 0); row < (both && !dir ? C / 2 : C); row += C / 2) {
        if (row >= n) break;
        T* out = reinterpret_cast<T*>(p.out_dv) + ((int64_t)bh * p.L + t0 + row) * DV + vc;
#pragma unroll
        for (int i = 0; i < VPT; i += 4) {
            float4 a = *reinterpret_cast<const float4*>(D0 + row * SM::VP + vc + i);
            const float4 z = *reinterpret_cast<const float4*>(D1 + row * SM::VP + vc + i);
            a.x += z.x; a.y += z.y; a.z += z.z; a.w += z.w;
            if (both) { const float4 s = *reinterpret_cast<const float4*>(sent + i); a.x += s.x; a.y += s.y; a.z += s.z; a.w += s.w; }
            store2<T>(out + i, a.x, a.y); store2<T>(out + i + 2, a.z, a.w);
        }
    }
}

template <int DK, int DV, typename T>
int launch_typed(const BwdParams& p, cudaStream_t stream) {
    const int BH = p.B * p.H;
    constexpr uint32_t smA = StatesSmem<DK, DV, T>::BYTES, smC = GradSmem<DK, DV, T>::BYTES;
    auto kA = bwd_states_mma_kernel<DK, DV, T>;
    auto kC = p.nchunk > 1 && !p.scanned ? bwd_grads_mma_kernel<DK, DV, T, true> : bwd_grads_mma_kernel<DK, DV, T, false>;
    cudaError_t e;
    if (p.nchunk > 1) {                                                  // one chunk: both entering states are zero
        if ((e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kA), (int)smA)) != cudaSuccess) return (int)e;
        // few chunks: one CTA per direction, so that more of the GPU works; many: one CTA reads v and d_out once for both
        const int gz = p.dir_mask == 3 && (int64_t)p.nchunk * BH < device_sms() * 4 ? 2 : 1;
        kA<<<dim3(p.nchunk, BH, gz), NT, smA, stream>>>(p);
        if (p.scanned) if (int s = bigla_bwd_scan_launch(p, stream)) return s;
    }
    if ((e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kC), (int)smC)) != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((p.dir_mask == 3 ? 2 : 1) * p.nchunk, BH); cfg.blockDim = dim3(NT); cfg.dynamicSmemBytes = smC; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (p.nchunk > 1) { attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[na++].val.programmaticStreamSerializationAllowed = 1; }
    if (p.dir_mask == 3) { attr[na].id = cudaLaunchAttributeClusterDimension; attr[na].val.clusterDim.x = 2; attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1; ++na; }
    cfg.attrs = attr; cfg.numAttrs = na;
    e = cudaLaunchKernelEx(&cfg, kC, p);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

template <typename T>
int launch_dims(const BwdParams& p, cudaStream_t stream) {
#define VIG_CASE(DKV, DVV) if (p.dk == DKV && p.dv == DVV) return launch_typed<DKV, DVV, T>(p, stream);
    VIG_CASE(16, 32) VIG_CASE(32, 32) VIG_CASE(32, 64) VIG_CASE(64, 64)
#undef VIG_CASE
    return VIG_ERR_SHAPE;
}

}  // namespace

int bigla_bwd_scan_launch(const BwdParams& p, cudaStream_t stream) {
    if (reinterpret_cast<uintptr_t>(p.ws_S) & 15) {
        const int64_t threads = (int64_t)p.B * p.H * (p.dir_mask == 3 ? 2 : 1) * 2 * (p.dk * p.dv);
        return (int)launch_next(bwd_scan_unaligned_kernel, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, stream, p);
    }
    const int64_t threads = (int64_t)p.B * p.H * (p.dir_mask == 3 ? 2 : 1) * 2 * (p.dk * p.dv / 4);
    return (int)launch_next(bwd_scan_kernel, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, stream, p);
}

// Rows are read as 16-byte vectors (16-bit v, d_out) or as pairs of values: base pointers on 16 bytes, strides that are
// multiples of 16 bytes.  Everything else, and heads whose tiles exceed the registers of one warp row (dv = 128), takes
// the token-by-token form.  grid.y holds B*H, hence its limit.
bool bigla_bwd_mma_supported(const BwdParams& p) {
    if (!((p.dk == 16 && p.dv == 32) || (p.dk == 32 && p.dv == 32) || (p.dk == 32 && p.dv == 64) || (p.dk == 64 && p.dv == 64))) return false;
    if ((int64_t)p.B * p.H > 65535) return false;
    const int unit = p.dtype == VIG_DTYPE_F32 ? 4 : 8;
    auto ok = [&](const void* base, const int64_t* s) {
        return !base || (!(reinterpret_cast<uintptr_t>(base) & 15) && s[0] % unit == 0 && s[1] % unit == 0 && s[2] % unit == 0);
    };
    return ok(p.q, p.sq) && ok(p.k, p.sk) && ok(p.v, p.sv) && ok(p.dout, p.sdo) && ok(p.gf, p.sgf) && ok(p.gb, p.sgb);
}

int bigla_bwd_mma_launch(const BwdParams& p, cudaStream_t stream) {
    switch (p.dtype) {
        case VIG_DTYPE_F32: return launch_dims<float>(p, stream);
        case VIG_DTYPE_BF16: return launch_dims<__nv_bfloat16>(p, stream);
        case VIG_DTYPE_F16: return launch_dims<__half>(p, stream);
    }
    return VIG_ERR_DTYPE;
}

}  // namespace vig
