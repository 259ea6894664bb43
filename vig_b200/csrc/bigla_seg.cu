// Bi-directional gated linear attention, segments of up to 32, 64 or 128 tokens on mma.sync tensor cores, both directions of a
// segment in one sweep: the forward of short and medium sequences, of head sizes the tcgen05 kernels do not take (dv = 32),
// and of fp32 calls.
//
// Inside a segment the two directions are one product.  With G the cumulative log-gate of a direction in its scan order, r
// its value near the segment's middle, Q = q 2^(G-r), K = k 2^(r-G):
//     P_ij = Qf_i Kf_j (j < i),  Qb_i Kb_j (j > i),  both for j = i           o_i = c (P_i V + Qf_i (2^rf Sf) + Qb_i (2^rb Sb))
// so a 16 x 16 block off the diagonal is computed once, with the tiles of the direction that owns it, and P V once for both.
// Sf, Sb are the states entering the segment from its two sides.  A segment's own contribution, U = 2^(l-r) K^T V (l = total),
// goes to the workspace; the segments of a sequence form one thread-block cluster, meet at its barrier after their products
// (which need no state) and each sums the contributions that reach it: one launch, every input read once, for sequences of up
// to 16 segments.  Longer ones run as states, scan over segments (bigla_simt_state_scan), outputs.
//
// Against the two-CTAs-per-SM tcgen05 form, which walks 128-token chunks one after the other in each direction with a tensor
// memory round trip for the scores: P stays in registers, a segment's rows spread over all warps at once.  One segment takes
// about 22 k cycles alone in fp32 (loads and gates 5, tiles 3, contribution 5, products 5, states 4; 10 k in bf16): a call of few
// segments is that latency, one of many is bound by instruction issue at 16 warps an SM.
// Operands are split into bf16 terms (mma_common.cuh): one term for bf16 with dv = 64 (as in the two-CTAs-per-SM tcgen05 form), two for
// fp16 and for dv = 32, three for fp32.  A segment whose |G - r| leaves the factorisation's range, contribution included,
// is evaluated token by token (bigla_exact.cuh).
#include <atomic>
#include "bigla_exact.cuh"

namespace vig {
namespace {

using namespace mm;

constexpr int SEG_NO_CLUSTER = -1001;                    // the device cannot place a cluster of this size: three launches instead
enum { SEG_ONE = 0, SEG_STATES = 1, SEG_OUT = 2 };       // one launch (cluster = sequence) / contributions only / outputs from entering states

template <int DK, int DV, typename T> struct SegTerms {
    static constexpr int RAW = Terms<T>::RAW, SC = (sizeof(T) == 2 && RAW == 1 && DV == 64) ? 1 : Terms<T>::SC;
};

// Warps that share 16 rows (CW below), each with its part of the value columns (the scores are formed by each of them): two for fp32, whose
// three-term tiles leave room for one or two 64-token segments an SM (2x3x196 64/64: 28.4 -> 19.5 us; 16x6x1000 64/64: 520 ->
// 320), and for 16-bit segments of 64 tokens and dv = 64 while each has an SM of its own (1x3x196 32/64, bf16: 10.3 -> 8.8 us one call behind
// another); twice as many for segments of 32 tokens.  Where two or more 16-bit segments share an SM, its issue slots go to the scores formed twice: one
// warp (seg_launch_tok has the figures).
template <int DV, typename T, int TOK> constexpr int seg_warps() {
    return (sizeof(T) == 4 ? 2 : TOK == 32 || (TOK == 64 && DV == 64) ? 2 : 1) * (sizeof(T) == 4 && TOK == 32 ? 2 : 1);
}

template <int DK, int DV, typename T, int TOK, int CW> struct SegSmem {
    using TT = SegTerms<DK, DV, T>;
    static constexpr uint32_t QT = TT::SC * (TOK * Pitch<DK>::B > DK * Pitch<DV>::B ? TOK * Pitch<DK>::B : DK * Pitch<DV>::B);   // one direction's Q or K terms, or its entering state
    static constexpr uint32_t V = 0, K = TT::RAW * TOK * Pitch<DV>::B, Q = K + 2 * QT, SUM = Q + 2 * QT,
                              SCL = SUM + 2 * (TOK / 16) * CW * DK * 4,      // per direction and warp: summed log-gates of the warp's rows
                              BYTES = SCL + 4 * DK * 4;                 // [dir][0: 2^r, 1: 2^(l-r)]
};

// x * e of a raw pair and a pair of fp32 factors, in SC bf16 terms: the product in fp32, then rounded
template <typename T, int SC> __device__ __forceinline__ void scaled(const Raw2<T>& x, float ex, float ey, uint32_t* t) {
    const F2 v = f2_mul(x.f2(), f2_make(ex, ey));
    split2<SC>(f2_lo(v), f2_hi(v), t);
}

template <typename T, int COLS, int TERMS, int TOK, int NTH> __device__ __forceinline__ void seg_load_v(uint8_t* dst, const T* src, int64_t stride_l, int n, float& mark) {
    constexpr uint32_t P = Pitch<COLS>::B;
    if constexpr (TERMS == 1) {
        constexpr int VPR = COLS / 8;
#pragma unroll
        for (int i0 = 0; i0 < TOK * VPR; i0 += NTH) {
            const int i = i0 + threadIdx.x, r = i / VPR, v = i % VPR;
            const uint32_t d = tc::smem_u32(dst + r * P + v * 16);
            const T* s = src + (r < n ? r : 0) * stride_l + v * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(s), "r"(r < n ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    } else {
        constexpr int PPR = COLS / 4;
#pragma unroll 4
        for (int i0 = 0; i0 < TOK * PPR; i0 += NTH) {
            const int i = i0 + threadIdx.x, r = i / PPR, v = i % PPR;
            float2 a = make_float2(0.f, 0.f), b = a;
            if (r < n) { a = load2_coherent<T>(src + r * stride_l + 4 * v); b = load2_coherent<T>(src + r * stride_l + 4 * v + 2); }
            see(mark, a.x); see(mark, a.y); see(mark, b.x); see(mark, b.y);
            uint32_t ta[TERMS], tb[TERMS];
            split2<TERMS>(a.x, a.y, ta); split2<TERMS>(b.x, b.y, tb);
#pragma unroll
            for (int t = 0; t < TERMS; ++t) *reinterpret_cast<uint2*>(dst + t * TOK * P + r * P + v * 8) = make_uint2(ta[t], tb[t]);
        }
    }
}

// whether the values this thread copied are finite (one-term tiles, after the copies have landed)
template <int COLS, int TOK, int NTH> __device__ __forceinline__ bool seg_v_clean(const uint8_t* tile) {
    uint32_t bad = 0;
#pragma unroll
    for (int i0 = 0; i0 < TOK * (COLS / 8); i0 += NTH) {
        const int i = i0 + threadIdx.x;
        bad |= bf16_unclean(*reinterpret_cast<const uint4*>(tile + i / (COLS / 8) * Pitch<COLS>::B + i % (COLS / 8) * 16));
    }
    return bad == 0;
}

struct SegParams {
    BiglaParams p;
    int nseg, seglen;            // segments per sequence, tokens per segment (a multiple of 16; the last one may be shorter)
    int need_states;             // contributions are wanted (more than one segment, or final states)
    int finals;                  // final states or summed log-gates are wanted
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// State entering segment c from the side a direction comes from, four values starting at e4 (SEG_ONE: summed here from the
// segments' contributions; SEG_OUT: what the scan left in the segment's slot).
template <int DK, int DV, int MODE> __device__ __forceinline__ float4 entering(const SegParams& s, int bh, int c, int dir, int e4) {
    const BiglaParams& p = s.p;
    const float4* U = reinterpret_cast<const float4*>(p.ws_state);
    constexpr int per = DK * DV / 4;
    if (MODE == SEG_OUT) return __ldcg(U + (((size_t)bh * s.nseg + c) * 2 + dir) * per + e4);
    const float* init = dir ? p.init_b : p.init_f;
    float4 S = init ? __ldcg(reinterpret_cast<const float4*>(init) + (size_t)bh * per + e4) : make_float4(0.f, 0.f, 0.f, 0.f);
    const int d = e4 * 4 / DV, m = dir ? s.nseg - 1 - c : c;
#pragma unroll 4
    for (int i = 0; i < m; ++i) {
        const size_t slot = ((size_t)bh * s.nseg + (dir ? s.nseg - 1 - i : i)) * 2 + dir;
        const float4 u = __ldcg(U + slot * per + e4);
        const float a = __expf(__ldcg(p.ws_decay + slot * DK + d));
        S.x = fmaf(S.x, a, u.x); S.y = fmaf(S.y, a, u.y); S.z = fmaf(S.z, a, u.z); S.w = fmaf(S.w, a, u.w);
    }
    return S;
}

// A segment whose gates leave the factorisation's range, or are growing ones, token by token: what it contributes, and its
// outputs.  Every thread works on it: at 96 sequences of 1000 tokens, fp32 64 / 64, all segments out of range, 14.6 ms with DV
// threads to a segment, 0.83 with all (1.19 in the gate-independent form of bigla_simt.cu).  The segment's tiles give up their shared memory.
template <int DK, int DV, typename T, int TOK, int CW> struct SegExact {
    using SM = SegSmem<DK, DV, T, TOK, CW>;
    using L = rec::Lay<DK, DV, 2 * TOK * CW>;
    static constexpr uint32_t ROW = 3 * DK + DV;                         // floats staged for a token
    static constexpr uint32_t bytes(int sub) { return (L::HALVES * sub * ROW + TOK * DV) * 4; }
    static constexpr int SUB = bytes(32) <= SM::SUM ? 32 : bytes(16) <= SM::SUM ? 16 : 8;      // tokens staged at a time
    static_assert(bytes(SUB) <= SM::SUM && SUB % rec::GROUP == 0, "the exact form works in the tiles");
    // Tokens in an even number of blocks: with both directions under way at once, each block is visited by one, then, steps
    // and barriers later, by the other.
    static __device__ int blocks(int n) { return 2 * ((n + 2 * SUB - 1) / (2 * SUB)); }
};

template <int DK, int DV, typename T, int TOK, int CW> __device__ __noinline__ void exact_contribution(const SegParams& s, float* sm, int bh, int c, int n) {
    using E = SegExact<DK, DV, T, TOK, CW>;
    using L = typename E::L;
    const BiglaParams& p = s.p;
    const int b = bh / p.H, h = bh % p.H, d0 = L::d0(), j0 = L::j0(), tid = threadIdx.x % L::HT;
    const int blocks = E::blocks(n), size = (n + blocks - 1) / blocks;
    float *sa = sm + L::half() * E::SUB * E::ROW, *sg = sa + E::SUB * DK, *sk = sg + E::SUB * DK, *sv = sk + E::SUB * DK;
    for (int pass = 0; pass < 2 / L::HALVES; ++pass) {
        const int dir = L::HALVES == 2 ? L::half() : pass;
        const bool on = p.dir_mask & (1 << dir);
        float S[L::JPT][L::DPT], sum = 0.f;
#pragma unroll
        for (int j = 0; j < L::JPT; ++j)
#pragma unroll
            for (int d = 0; d < L::DPT; ++d) S[j][d] = 0.f;
        for (int bb = 0; bb < blocks; ++bb) {
            const int at = (dir ? blocks - 1 - bb : bb) * size, m = on ? max(0, min(size, n - at)) : 0;
            const int64_t t = (int64_t)c * s.seglen + at;
            __syncthreads();
            if (m > 0)
                rec::stage<DK, DV, L::HT, T>(nullptr, sk, sv, sg, sa, nullptr, 0, 0.f, head_ptr<T>(p.k, p.sk, b, h, t), p.sk[2], 1.f, head_ptr<T>(p.v, p.sv, b, h, t), p.sv[2],
                                             dir ? head_ptr<T>(p.gb, p.sgb, b, h, t) : head_ptr<T>(p.gf, p.sgf, b, h, t), dir ? p.sgb[2] : p.sgf[2], m, p.gate_norm, p.clamp_min, tid);
            __syncthreads();
            if (tid < DK) for (int i = 0; i < m; ++i) sum += sg[i * DK + tid];
            rec::each(m, dir, [&](int i) { rec::update(S, sa + i * DK + d0, sk + i * DK + d0, sv + i * DV + j0); });
        }
        if (!on) continue;
        const size_t slot = ((size_t)bh * s.nseg + c) * 2 + dir;
#pragma unroll
        for (int j = 0; j < L::JPT; ++j)
#pragma unroll
            for (int d = 0; d < L::DPT; ++d) p.ws_state[slot * DK * DV + (d0 + d) * DV + j0 + j] = S[j][d];
        if (tid < DK) p.ws_decay[slot * DK + tid] = sum;
    }
}

// N neighbouring values of a state, read as one vector
template <int N> __device__ __forceinline__ void load_state_row(float (&x)[N], const float* p) {
    if constexpr (N == 4) { const float4 v = __ldcg(reinterpret_cast<const float4*>(p)); x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w; }
    else if constexpr (N == 2) { const float2 v = __ldcg(reinterpret_cast<const float2*>(p)); x[0] = v.x; x[1] = v.y; }
    else x[0] = __ldcg(p);
}

// The state entering segment c, my channels and columns of it (as ``entering``, all of a contribution's values in flight together)
template <int DK, int DV, int MODE, typename L> __device__ __forceinline__ void entering_rows(float (&S)[L::JPT][L::DPT], const SegParams& s, int bh, int c, int dir) {
    const BiglaParams& p = s.p;
    const int at = L::d0() * DV + L::j0(), m = MODE == SEG_OUT ? 0 : dir ? s.nseg - 1 - c : c;
    const float* first = MODE == SEG_OUT ? p.ws_state + (((size_t)bh * s.nseg + c) * 2 + dir) * DK * DV : dir ? p.init_b : p.init_f;
    if (MODE != SEG_OUT && first) first += (size_t)bh * DK * DV;
    float u[L::DPT][L::JPT];
#pragma unroll
    for (int d = 0; d < L::DPT; ++d) {
        if (first) load_state_row(u[d], first + at + d * DV);
#pragma unroll
        for (int j = 0; j < L::JPT; ++j) S[j][d] = first ? u[d][j] : 0.f;
    }
#pragma unroll 2
    for (int g = 0; g < m; ++g) {
        const size_t slot = ((size_t)bh * s.nseg + (dir ? s.nseg - 1 - g : g)) * 2 + dir;
        float a[L::DPT];
#pragma unroll
        for (int d = 0; d < L::DPT; ++d) { load_state_row(u[d], p.ws_state + slot * DK * DV + at + d * DV); a[d] = __ldcg(p.ws_decay + slot * DK + L::d0() + d); }
#pragma unroll
        for (int d = 0; d < L::DPT; ++d) {
            const float e = __expf(a[d]);
#pragma unroll
            for (int j = 0; j < L::JPT; ++j) S[j][d] = fmaf(S[j][d], e, u[d][j]);
        }
    }
}

template <int DK, int DV, typename T, int TOK, int CW, int MODE> __device__ __noinline__ void exact_outputs(const SegParams& s, float* sm, int bh, int c, int n) {
    using E = SegExact<DK, DV, T, TOK, CW>;
    using L = typename E::L;
    constexpr int NTH = L::HT * L::HALVES, NV = rec::GROUP * L::JPT;
    const BiglaParams& p = s.p;
    const int b = bh / p.H, h = bh % p.H, d0 = L::d0(), j0 = L::j0(), tid = threadIdx.x % L::HT;
    const int blocks = E::blocks(n), size = (n + blocks - 1) / blocks;
    float *so = sm, *sa = so + TOK * DV + L::half() * E::SUB * E::ROW, *sq = sa + E::SUB * DK, *sk = sq + E::SUB * DK, *sv = sk + E::SUB * DK;
    for (int pass = 0; pass < 2 / L::HALVES; ++pass) {
        const int dir = L::HALVES == 2 ? L::half() : pass;
        const bool on = p.dir_mask & (1 << dir), both = p.dir_mask == 3;
        float S[L::JPT][L::DPT];
        if (on) entering_rows<DK, DV, MODE, L>(S, s, bh, c, dir);
        for (int bb = 0; bb < blocks; ++bb) {
            const int at = (dir ? blocks - 1 - bb : bb) * size, m = on ? max(0, min(size, n - at)) : 0;
            const int64_t t = (int64_t)c * s.seglen + at;
            const bool add = both && (L::HALVES == 2 ? bb >= blocks / 2 : dir == 1);       // the block's second visit
            __syncthreads();
            if (m > 0)
                rec::stage<DK, DV, L::HT, T>(sq, sk, sv, nullptr, sa, head_ptr<T>(p.q, p.sq, b, h, t), p.sq[2], p.qscale, head_ptr<T>(p.k, p.sk, b, h, t), p.sk[2], 1.f,
                                             head_ptr<T>(p.v, p.sv, b, h, t), p.sv[2], dir ? head_ptr<T>(p.gb, p.sgb, b, h, t) : head_ptr<T>(p.gf, p.sgf, b, h, t), dir ? p.sgb[2] : p.sgf[2], m, p.gate_norm, p.clamp_min, tid);
            __syncthreads();
            const int np = rec::padded(m);
#pragma unroll 1
            for (int i0 = 0; i0 < np; i0 += rec::GROUP) {
                float o[NV];
#pragma unroll
                for (int u = 0; u < rec::GROUP; ++u) {
                    const int i = dir ? np - 1 - i0 - u : i0 + u;
                    rec::update(S, sa + i * DK + d0, sk + i * DK + d0, sv + i * DV + j0);
                    rec::read_out(o + u * L::JPT, S, sq + i * DK + d0);
                }
                const int first = rec::reduce_scatter<L::DG>(o);
#pragma unroll
                for (int e = 0; e < rec::Share<L::DG, NV>::V; ++e) {
                    const int u = (first + e) / L::JPT, i = dir ? np - 1 - i0 - u : i0 + u;
                    float* out = so + (at + i) * DV + j0 + (first + e) % L::JPT;
                    if (first >= 0 && i < m) *out = add ? *out + o[e] : o[e];
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * (DV / 2); i += NTH) {
        const int r = i / (DV / 2), v = i % (DV / 2) * 2;
        store2<T>(reinterpret_cast<T*>(p.o) + b * p.so[0] + h * p.so[1] + ((int64_t)c * s.seglen + r) * p.so[2] + v, so[r * DV + v], so[r * DV + v + 1]);
    }
}

template <int DK, int DV, typename T, int TOK, int CW> constexpr int seg_min_blocks() {
    constexpr int fit = 225 * 1024 / (int)(SegSmem<DK, DV, T, TOK, CW>::BYTES + 1024), regs = (DK == 16 ? 640 : 512) / (2 * TOK * CW);   // 128 registers a thread, 96 at DK = 16
    return fit < 1 ? 1 : fit < regs ? fit : regs;
}

template <int DK, int DV, typename T, int TOK, int CW, int MODE>
__global__ void __launch_bounds__(2 * TOK * CW, seg_min_blocks<DK, DV, T, TOK, CW>()) bigla_seg_kernel(const __grid_constant__ SegParams s) {
    using SM = SegSmem<DK, DV, T, TOK, CW>;
    constexpr int RAW = SM::TT::RAW, SC = SM::TT::SC, NTH = 2 * TOK * CW, W = NTH / 32, DC = DV / CW;   // DC: a warp's value columns
    constexpr int PAIRS = DK / 2, SUB = 32 / PAIRS, RPG = 16 / CW / SUB, MT = DK / 16;   // a warp's gates: 16 / CW rows, SUB groups of RPG
    constexpr uint32_t PK = Pitch<DK>::B, PV = Pitch<DV>::B, TK = TOK * PK, TV = TOK * PV, TS = DK * PV;   // TK, TV, TS: from term to term
    const BiglaParams& p = s.p;
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t sb = tc::smem_u32(smem);
    float* gsum = reinterpret_cast<float*>(smem + SM::SUM);              // [dir][warp][DK]
    float* scl = reinterpret_cast<float*>(smem + SM::SCL);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rb = w / CW, cb = w % CW;     // my block of 16 rows and part of the value columns in the products
    const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H;
    const int64_t t0 = (int64_t)c * s.seglen;
    const int n = min(s.seglen, p.L - (int)t0), nb = (n + 15) / 16;
    const int pr = threadIdx.x % PAIRS, gr = threadIdx.x / PAIRS, r0 = gr * RPG;   // my channel pair, my rows
    pdl_launch();                                                        // a chained successor may fetch its weights meanwhile
    if (MODE == SEG_ONE) pdl_wait();                                     // chained itself: the launch before it may have written the inputs
    const bool want_out = MODE != SEG_STATES && p.o;
    const bool fwd = p.dir_mask & 1, bwd = p.dir_mask & 2;
    F2 G[2][RPG], ref[2];
    Raw2<T> kr[RPG];
    bool fine = true, bad;
    {   // ---- every input of the segment requested at once, gates cumulated, operand tiles written
        // fp32 calls and heads of dv = 32 keep infinities and NaN to the tokens that see them, as the recurrences do; the other
        // 16-bit heads share a tcgen05 form in which they reach a chunk
        constexpr bool CHECK = sizeof(T) == 4 || DV == 32;
        float mark = 0.f;
        F2 seen = f2_make(0.f, 0.f);
        seg_load_v<T, DV, RAW, TOK, NTH>(smem + SM::V, head_ptr<T>(p.v, p.sv, b, h, t0), p.sv[2], n, mark);
        const bool logits = p.gate_norm > 0.f, clamp = p.clamp_min == p.clamp_min;
        Raw2<T> qr[RPG];
        {
            Raw2<T> xr[2][RPG];
            // rows past the end read the last row (no branch between the loads) and are neutralised afterwards; an absent
            // tensor reads k in its place
            const T* kp = head_ptr<T>(p.k, p.sk, b, h, t0) + 2 * pr;
            const T* qp = want_out ? head_ptr<T>(p.q, p.sq, b, h, t0) + 2 * pr : kp;
            const T* fp = fwd ? head_ptr<T>(p.gf, p.sgf, b, h, t0) + 2 * pr : kp;
            const T* bp = bwd ? head_ptr<T>(p.gb, p.sgb, b, h, t0) + 2 * pr : kp;
            const int64_t lk = p.sk[2], lq = want_out ? p.sq[2] : lk, lf = fwd ? p.sgf[2] : lk, lb = bwd ? p.sgb[2] : lk;
#pragma unroll
            for (int r = 0; r < RPG; ++r) {
                const int64_t row = min(r0 + r, n - 1);
                xr[0][r].load_coherent(fp + row * lf);
                xr[1][r].load_coherent(bp + row * lb);
                kr[r].load_coherent(kp + row * lk);
                if (MODE != SEG_STATES) qr[r].load_coherent(qp + row * lq); else qr[r].zero();
            }
            if (r0 + RPG > n) {
#pragma unroll
                for (int r = 0; r < RPG; ++r)
                    if (r0 + r >= n) { kr[r].zero(); qr[r].zero(); xr[0][r].open_gate(logits); xr[1][r].open_gate(logits); }
            }
            if (CHECK) {
#pragma unroll
                for (int r = 0; r < RPG; ++r) { see(seen, kr[r].f2()); see(seen, qr[r].f2()); }
            }
            const F2 zero = f2_make(0.f, 0.f);
            const F2 nlog2e = f2_make(-tc::LOG2E, -tc::LOG2E);
#pragma unroll
            for (int dir = 0; dir < 2; ++dir) {
                F2 run = zero;
                if (sizeof(T) == 2 && logits && !clamp) {                // the models' form: -log2(1 + 2^(-x log2 e)) / norm
                    const float ni = -1.f / p.gate_norm;
                    const F2 ninv = f2_make(ni, ni);
#pragma unroll
                    for (int rr = 0; rr < RPG; ++rr) {
                        const int r = dir ? RPG - 1 - rr : rr;
                        run = f2_fma(softplus2(f2_mul(xr[dir][r].f2(), nlog2e)), ninv, run);
                        G[dir][r] = run;
                    }
                } else {
                    row_gates(G[dir], xr[dir], p.gate_norm, p.clamp_min);
                    float top = 0.f;
#pragma unroll
                    for (int rr = 0; rr < RPG; ++rr) {
                        const int r = dir ? RPG - 1 - rr : rr;
                        if (r0 + r < n && (dir ? bwd : fwd)) { top = fmaxf(top, fmaxf(f2_lo(G[dir][r]), f2_hi(G[dir][r]))); run = f2_add(run, G[dir][r]); }
                        G[dir][r] = run;
                    }
                    fine = fine && top <= 0.f;                            // growing gates: G is not monotone, its ends do not bound it
                }
                // across the warp's groups: what those scanned before mine contribute, and the warp's sum
                const F2 mine = run;
                F2 ahead = zero;
#pragma unroll
                for (int k = 1; k < SUB; ++k) {
                    const int from = dir ? lane + k * PAIRS : lane - k * PAIRS;
                    const F2 x = __shfl_sync(0xffffffffu, mine, from & 31);
                    if (dir ? from < 32 : from >= 0) ahead = f2_add(ahead, x);
                }
                if constexpr (SUB > 1) {
#pragma unroll
                    for (int r = 0; r < RPG; ++r) G[dir][r] = f2_add(G[dir][r], ahead);
                }
                if (lane / PAIRS == (dir ? 0 : SUB - 1)) *reinterpret_cast<F2*>(gsum + (dir * W + w) * DK + 2 * pr) = f2_add(ahead, mine);
            }
        }
        __syncthreads();
        const int wm = nb / 2 * CW;                                           // the reference lies between the rows of warps wm - 1 and wm
        const float lim = range_limit<T>();
        F2 shift[2];
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            F2 run = f2_make(0.f, 0.f), before = run, lo = run, mine = run;
#pragma unroll
            for (int o = 0; o < W; ++o) {
                const F2 x = *reinterpret_cast<const F2*>(gsum + (dir * W + o) * DK + 2 * pr);
                if (o == w) { before = run; mine = x; }
                if (o == wm) lo = run;
                run = f2_add(run, x);
            }
            const F2 minus = f2_make(-1.f, -1.f);
            const F2 off = dir ? f2_fma(f2_add(before, mine), minus, run) : before;        // what the warps scanned earlier contribute
            ref[dir] = dir ? f2_fma(lo, minus, run) : lo;
            const F2 rest = f2_fma(ref[dir], minus, run);
            // gates are <= 0, so |G - ref| is largest at the segment's two ends
            if (dir ? bwd : fwd) fine = fine && fabsf(f2_lo(ref[dir])) <= lim && fabsf(f2_hi(ref[dir])) <= lim && fabsf(f2_lo(rest)) <= lim && fabsf(f2_hi(rest)) <= lim;
            if (gr == 0) {
                float* sc = scl + dir * 2 * DK + 2 * pr;
                *reinterpret_cast<float2*>(sc) = make_float2(ex2_t<T>(f2_lo(ref[dir])), ex2_t<T>(f2_hi(ref[dir])));
                *reinterpret_cast<float2*>(sc + DK) = MODE == SEG_STATES ? make_float2(1.f, 1.f) : make_float2(ex2_t<T>(f2_lo(rest)), ex2_t<T>(f2_hi(rest)));
                if (MODE != SEG_OUT && s.need_states && (dir ? bwd : fwd))
                    *reinterpret_cast<float2*>(p.ws_decay + (((size_t)bh * s.nseg + c) * 2 + dir) * DK + 2 * pr) = make_float2(f2_lo(run) * tc::LN2, f2_hi(run) * tc::LN2);
            }
            shift[dir] = MODE == SEG_STATES ? f2_fma(run, minus, off) : f2_fma(ref[dir], minus, off);        // G - (total or reference)
        }
        if (CHECK) {
            if (RAW == 1) asm volatile("cp.async.wait_all;" ::: "memory");
            fine = fine && clean(seen) && (RAW == 1 ? seg_v_clean<DV, TOK, NTH>(smem + SM::V) : clean(mark));
        }
        bad = __syncthreads_or(!fine);
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            if (bad || !(dir ? bwd : fwd) || rb >= nb) continue;
            uint8_t* kt = smem + SM::K + dir * SM::QT + r0 * PK + pr * 4;
            uint8_t* qt = smem + SM::Q + dir * SM::QT + r0 * PK + pr * 4;
#pragma unroll
            for (int r = 0; r < RPG; ++r) {
                const F2 x = f2_add(G[dir][r], shift[dir]);
                uint32_t t[SC];
                if (MODE != SEG_STATES) {
                    scaled<T, SC>(qr[r], ex2_t<T>(f2_lo(x)), ex2_t<T>(f2_hi(x)), t);
#pragma unroll
                    for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(qt + i * TK + r * PK) = t[i];
                }
                scaled<T, SC>(kr[r], ex2_t<T>(-f2_lo(x)), ex2_t<T>(-f2_hi(x)), t);
#pragma unroll
                for (int i = 0; i < SC; ++i) *reinterpret_cast<uint32_t*>(kt + i * TK + r * PK) = t[i];
            }
        }
    }
    if (RAW == 1) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (MODE != SEG_OUT && s.need_states && bad) {
        exact_contribution<DK, DV, T, TOK, CW>(s, reinterpret_cast<float*>(smem), bh, c, n);
    } else if (MODE != SEG_OUT && s.need_states) {                       // ---- contributions: units of 16 key channels x NC value columns of one direction
        constexpr int UNITS = 2 * MT, NSPLIT = W <= UNITS ? 1 : W / UNITS < DV / 8 ? W / UNITS : DV / 8, NC = DV / NSPLIT, NTL = NC / 8;
        for (int u = w; u < UNITS * NSPLIT; u += W) {
            const int dir = u / (MT * NSPLIT), mt = (u / NSPLIT) % MT, ns = u % NSPLIT;
            if (!(dir ? bwd : fwd)) continue;
            float acc[NTL][4];
#pragma unroll
            for (int i = 0; i < NTL; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
            const uint32_t x = sb + SM::K + dir * SM::QT + mt * 32 + frag_cols<PK>(lane), y = sb + SM::V + ns * NC * 2 + frag_rows<PV>(lane);
#pragma unroll 2
            for (int ks = 0; ks < nb; ++ks) {
                uint32_t a[SC][4];
#pragma unroll
                for (int t = 0; t < SC; ++t) ldsm4t(x + t * TK + ks * 16 * PK, a[t]);
                block_nn<NC, SC, RAW>(acc, a, y + ks * 16 * PV, TV);
            }
            const float* sc = scl + dir * 2 * DK + DK + mt * 16 + (lane >> 2);
            const float s0 = sc[0], s1 = sc[8];
            float* out = p.ws_state + (((size_t)bh * s.nseg + c) * 2 + dir) * DK * DV + (mt * 16 + (lane >> 2)) * DV + ns * NC + 2 * (lane & 3);
#pragma unroll
            for (int i = 0; i < NTL; ++i) {
                *reinterpret_cast<float2*>(out + i * 8) = make_float2(acc[i][0] * s0, acc[i][1] * s0);
                *reinterpret_cast<float2*>(out + 8 * DV + i * 8) = make_float2(acc[i][2] * s1, acc[i][3] * s1);
            }
        }
    }
    if (MODE == SEG_STATES) return;
    if (MODE == SEG_ONE && s.nseg > 1) cluster_arrive();
    float o[DC / 8][4];
#pragma unroll
    for (int i = 0; i < DC / 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] = 0.f;
    const uint32_t aQ = sb + SM::Q + 16 * rb * PK + frag_rows<PK>(lane);
    if (want_out && !bad && rb < nb) {                                    // ---- products inside the segment, my 16 rows
        const uint32_t bK = sb + SM::K + frag_cols<PK>(lane), tV = sb + SM::V + cb * DC * 2 + frag_rows<PV>(lane);
        uint32_t ap[SC][4];
#pragma unroll 1
        for (int dir = 0; dir < 2; ++dir) {                              // off-diagonal blocks: before mine with the forward tiles, after it with the backward ones
            if (!(dir ? bwd : fwd)) continue;
            const uint32_t q = aQ + dir * SM::QT, k = bK + dir * SM::QT;
            uint32_t fq[DK / 16][SC][4];
#pragma unroll
            for (int ks = 0; ks < DK / 16; ++ks)
#pragma unroll
                for (int t = 0; t < SC; ++t) ldsm4(q + t * TK + ks * 32, fq[ks][t]);
            const int j1 = dir ? nb : rb;
#pragma unroll 1
            for (int jb = dir ? rb + 1 : 0; jb < j1; jb += 2) {           // two blocks at a time: four independent chains of products
                const bool two = jb + 1 < j1;
                float pb[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) pb[i][j] = 0.f;
#pragma unroll
                for (int ks = 0; ks < DK / 16; ++ks) {
                    uint32_t bf[4][SC][2];
                    if (two) {
                        load_b_nt<SC, 4, PK>(bf, k + jb * 16 * PK + ks * 32, TK);
                        mma_group<SC, SC, 4>(pb, fq[ks], bf);
                    } else {
                        load_b_nt<SC, 2, PK>(bf, k + jb * 16 * PK + ks * 32, TK);
                        mma_group<SC, SC, 2>(pb, fq[ks], bf);
                    }
                }
                mask_split<SC>(pb, false, lane, [](int, int) { return true; }, ap);
                block_nn<DC, SC, RAW>(o, ap, tV + jb * 16 * PV, TV);
                if (two) {
                    mask_split<SC>(pb + 2, false, lane, [](int, int) { return true; }, ap);
                    block_nn<DC, SC, RAW>(o, ap, tV + (jb + 1) * 16 * PV, TV);
                }
            }
        }
        float pd[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {                              // the diagonal block: both directions' halves, a token sees itself in each
            if (!(dir ? bwd : fwd)) continue;
            float pb[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            block_nt<DK, SC, SC>(pb, aQ + dir * SM::QT, TK, bK + dir * SM::QT + rb * 16 * PK, TK);
            const int r = lane >> 2, q = 2 * (lane & 3);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int row = r + 8 * (j >> 1), col = nt * 8 + q + (j & 1);
                    if (dir ? col >= row : col <= row) pd[nt][j] += pb[nt][j];
                }
        }
        mask_split<SC>(pd, false, lane, [](int, int) { return true; }, ap);
        block_nn<DC, SC, RAW>(o, ap, tV + rb * 16 * PV, TV);
    }
    const bool has_init = MODE == SEG_ONE && (p.init_f || p.init_b);
    if (MODE == SEG_ONE && s.nseg > 1) cluster_wait();                   // the other segments' contributions have landed
    else {
        if (MODE == SEG_OUT) pdl_wait();                                 // all before this overlaps the scan over segments
        __syncthreads();
    }
    if (MODE == SEG_ONE && s.finals) {
#pragma unroll 1
        for (int dir = 0; dir < 2; ++dir) {                              // final states, summed log-gates: by the segment scanned last
            float* fin = dir ? p.final_b : p.final_f;
            float* ld = dir ? p.logdecay_b : p.logdecay_f;
            if (!(dir ? bwd : fwd) || (!fin && !ld) || c != (dir ? 0 : s.nseg - 1)) continue;
            const size_t slot = ((size_t)bh * s.nseg + c) * 2 + dir;
            for (int i = threadIdx.x; i < DK * DV / 4; i += NTH) {
                const int d = i * 4 / DV;
                if (fin) {
                    float4 S = entering<DK, DV, MODE>(s, bh, c, dir, i);
                    const float4 u = __ldcg(reinterpret_cast<const float4*>(p.ws_state) + slot * (DK * DV / 4) + i);
                    const float a = __expf(__ldcg(p.ws_decay + slot * DK + d));
                    S.x = fmaf(S.x, a, u.x); S.y = fmaf(S.y, a, u.y); S.z = fmaf(S.z, a, u.z); S.w = fmaf(S.w, a, u.w);
                    reinterpret_cast<float4*>(fin)[(size_t)bh * (DK * DV / 4) + i] = S;
                }
                if (ld && i * 4 % DV == 0) {
                    float g = 0.f;
                    for (int k = 0; k < s.nseg; ++k) g += __ldcg(p.ws_decay + (((size_t)bh * s.nseg + k) * 2 + dir) * DK + d);
                    ld[(size_t)bh * DK + d] = g;
                }
            }
        }
    }
    if (!want_out) return;
    if (bad) {
        exact_outputs<DK, DV, T, TOK, CW, MODE>(s, reinterpret_cast<float*>(smem), bh, c, n);
        return;
    }
    if (MODE == SEG_OUT || s.nseg > 1 || has_init) {                     // ---- entering states, scaled, over the K tiles
        if (MODE == SEG_ONE && s.nseg > 1) __syncthreads();              // all warps are past their products (they arrived at the cluster barrier before them)
#pragma unroll 1
        for (int dir = 0; dir < 2; ++dir) {
            if (!(dir ? bwd : fwd)) continue;
            // KB states of four values per thread and pass, the contributions of two segments in flight for all of them: a
            // chain of dependent loads per state took as long as everything else in the kernel
            constexpr int KN = (DK * DV / 4 + NTH - 1) / NTH, KB = KN < 4 ? KN : 4;
            const int m = MODE == SEG_OUT ? 0 : dir ? s.nseg - 1 - c : c;
            const float* init = dir ? p.init_b : p.init_f;
#pragma unroll 1
            for (int k0 = 0; k0 < KN; k0 += KB) {
                float4 S[KB];
                const int i0 = threadIdx.x + k0 * NTH;
                if (DK * DV / 4 < NTH && i0 >= DK * DV / 4) break;
#pragma unroll
                for (int k = 0; k < KB; ++k) {
                    const int i = i0 + k * NTH;
                    S[k] = MODE == SEG_OUT ? __ldcg(reinterpret_cast<const float4*>(p.ws_state) + (((size_t)bh * s.nseg + c) * 2 + dir) * (DK * DV / 4) + i)
                           : init ? __ldcg(reinterpret_cast<const float4*>(init) + (size_t)bh * (DK * DV / 4) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll 2
                for (int g = 0; g < m; ++g) {
                    const size_t from = ((size_t)bh * s.nseg + (dir ? s.nseg - 1 - g : g)) * 2 + dir;
                    float4 u[KB];
                    float a[KB];
#pragma unroll
                    for (int k = 0; k < KB; ++k) {
                        u[k] = __ldcg(reinterpret_cast<const float4*>(p.ws_state) + from * (DK * DV / 4) + i0 + k * NTH);
                        a[k] = __ldcg(p.ws_decay + from * DK + (i0 + k * NTH) * 4 / DV);
                    }
#pragma unroll
                    for (int k = 0; k < KB; ++k) {
                        const float e = __expf(a[k]);
                        S[k].x = fmaf(S[k].x, e, u[k].x); S[k].y = fmaf(S[k].y, e, u[k].y); S[k].z = fmaf(S[k].z, e, u[k].z); S[k].w = fmaf(S[k].w, e, u[k].w);
                    }
                }
#pragma unroll
                for (int k = 0; k < KB; ++k) {
                    const int i = i0 + k * NTH, d = i * 4 / DV, v = i % (DV / 4);
                    const float a = scl[dir * 2 * DK + d];
                    uint32_t ta[SC], tb[SC];
                    split2<SC>(S[k].x * a, S[k].y * a, ta); split2<SC>(S[k].z * a, S[k].w * a, tb);
#pragma unroll
                    for (int t = 0; t < SC; ++t) *reinterpret_cast<uint2*>(smem + SM::K + dir * SM::QT + t * TS + d * PV + v * 8) = make_uint2(ta[t], tb[t]);
                }
            }
        }
        __syncthreads();
        if (rb < nb) {
#pragma unroll 1
            for (int dir = 0; dir < 2; ++dir) {
                if (!(dir ? bwd : fwd)) continue;
                const uint32_t tS = sb + SM::K + dir * SM::QT + cb * DC * 2 + frag_rows<PV>(lane);
#pragma unroll
                for (int ks = 0; ks < DK / 16; ++ks) {
                    uint32_t fa[SC][4];
#pragma unroll
                    for (int t = 0; t < SC; ++t) ldsm4(aQ + dir * SM::QT + t * TK + ks * 32, fa[t]);
                    block_nn<DC, SC, SC>(o, fa, tS + ks * 16 * PV, TS);
                }
            }
        }
    }
    if (rb >= nb) return;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
        const int row = 16 * rb + (lane >> 2) + 8 * hf;
        if (row >= n) continue;
        T* out = reinterpret_cast<T*>(p.o) + b * p.so[0] + h * p.so[1] + (t0 + row) * p.so[2] + cb * DC + 2 * (lane & 3);
#pragma unroll
        for (int i = 0; i < DC / 8; ++i) store2<T>(out + 8 * i, p.qscale * o[i][2 * hf], p.qscale * o[i][2 * hf + 1]);
    }
}

template <int DK, int DV, typename T, int TOK, int CW, int MODE>
int seg_launch_mode(const SegParams& s, cudaStream_t stream) {
    auto kern = bigla_seg_kernel<DK, DV, T, TOK, CW, MODE>;
    constexpr uint32_t smem = SegSmem<DK, DV, T, TOK, CW>::BYTES;
    cudaError_t e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kern), (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(s.nseg, s.p.B * s.p.H);
    cfg.blockDim = dim3(2 * TOK * CW);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    if (MODE == SEG_OUT) return (int)launch_next(kern, cfg.gridDim, cfg.blockDim, smem, stream, s);
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (MODE == SEG_ONE && s.nseg > 1) {
        cudaLaunchAttribute& c = attr[cfg.numAttrs++];
        c.id = cudaLaunchAttributeClusterDimension;
        c.val.clusterDim.x = s.nseg; c.val.clusterDim.y = 1; c.val.clusterDim.z = 1;
    }
    if (MODE == SEG_ONE && s.nseg > 8) {                 // more than the portable cluster size: the device is asked once whether it can place it
        static std::atomic<uint32_t> answers[64];        // two bits a size: asked, yes
        int dev = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return (int)e;
        const uint32_t asked = 1u << (2 * (s.nseg - 9)), yes = 2u << (2 * (s.nseg - 9));
        uint32_t have = answers[dev & 63].load();
        if (!(have & asked)) {
            int n = 0;
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) n = 0;
            cudaGetLastError();                          // a refusal is an answer
            have = asked | (n > 0 ? yes : 0u);
            answers[dev & 63].fetch_or(have);
        }
        if (!(have & yes)) return SEG_NO_CLUSTER;
    }
    // Begins before the launch ahead of it ends, and reads its inputs coherently for that reason (ViG-T of one 224 x 224 image 253 -> 248 us a forward).  Not
    // the first of three launches: the later ones read the inputs before they wait, for launches of this call only.  Nor with more segments than SMs: they
    // crowd on the SMs that the projection ahead leaves idle, and the block tail behind finds its SMs late (ViG-T bf16, 128 x 128 x 128: 626 - 637 us
    // chained, in 9 of 9 processes; 598 - 603 in 11 of 17 otherwise, 619 - 634 in the others; 32 of 224 x 224: 651 - 660 in 4 of 4, 635 - 638 in 8 of 12).
    if (MODE == SEG_ONE && chain_launches && (int64_t)s.nseg * s.p.B * s.p.H <= device_sms()) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    e = cudaLaunchKernelEx(&cfg, kern, s);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

template <int DK, int DV, typename T, int TOK, int CW = seg_warps<DV, T, TOK>()>
int seg_launch(SegParams& s, cudaStream_t stream) {
    constexpr int CLUSTER = 16;                          // largest cluster of the architecture (1x3x2048 dk = 32: 12 us in one launch, 16 in three)
    BiglaParams& p = s.p;
    s.nseg = (p.L + TOK - 1) / TOK;
    s.seglen = ((p.L + s.nseg - 1) / s.nseg + 15) / 16 * 16;   // even segments: no nearly empty last one
    s.nseg = (p.L + s.seglen - 1) / s.seglen;
    s.need_states = s.nseg > 1 || s.finals;
    p.nchunk = s.nseg;
    p.ws_decay = p.ws_state ? p.ws_state + (size_t)p.B * p.H * s.nseg * 2 * DK * DV : nullptr;
    if constexpr (CW < seg_warps<DV, T, TOK>()) {        // sequences of one segment
        return seg_launch_mode<DK, DV, T, TOK, CW, SEG_ONE>(s, stream);
    } else {
        if (s.nseg <= CLUSTER) {
            const int r = seg_launch_mode<DK, DV, T, TOK, CW, SEG_ONE>(s, stream);
            if (r != SEG_NO_CLUSTER) return r;
        }
        if (int e = seg_launch_mode<DK, DV, T, TOK, CW, SEG_STATES>(s, stream)) return e;
        if (int e = bigla_scan_launch(p, stream)) return e;
        return p.o ? seg_launch_mode<DK, DV, T, TOK, CW, SEG_OUT>(s, stream) : 0;
    }
}

// 16-bit calls of dv = 64 have 64-token segments on a shared SM only where a sequence is one of them (bigla_seg_launch).  us with one warp / two to 16
// rows at sequences x tokens: bf16 32/64 147 x 64 5.1 / 5.1, 198 x 64 5.9 / 6.4, 768 x 49 12.0 / 15.7, 1596 x 64 20.0 / 28.9; 64/64 147 x 64 6.8 / 6.6, 198 x 64 8.4 / 8.8, 399 x 64
// 10.5 / 12.9; fp16 32/64 147 x 64 6.7 / 6.3, 198 x 49 7.7 / 8.3.
template <int DK, int DV, typename T>
int seg_launch_tok(SegParams& s, int tok, cudaStream_t stream) {
    if constexpr (SegTerms<DK, DV, T>::SC > 1) if (tok == 32) return seg_launch<DK, DV, T, 32>(s, stream);
    if constexpr (sizeof(T) == 4 || DV == 32) {
        return seg_launch<DK, DV, T, 64>(s, stream);
    } else {
        if (s.p.L <= 64 && (int64_t)s.p.B * s.p.H > device_sms()) return seg_launch<DK, DV, T, 64, 1>(s, stream);
        return tok == 64 ? seg_launch<DK, DV, T, 64>(s, stream) : seg_launch<DK, DV, T, 128>(s, stream);
    }
}

template <typename T>
int seg_launch_dims(SegParams& s, int tok, cudaStream_t stream) {
#define VIG_CASE(DKV, DVV) if (s.p.dk == DKV && s.p.dv == DVV) return seg_launch_tok<DKV, DVV, T>(s, tok, stream);
    VIG_CASE(16, 32) VIG_CASE(32, 32) VIG_CASE(32, 64) VIG_CASE(64, 64)
#undef VIG_CASE
    return VIG_ERR_SHAPE;
}

}  // namespace

// Rows are read as pairs of values and (16-bit v) 16-byte vectors: base pointers on 16 bytes, strides multiples of 16 bytes.
// grid.y holds B*H, hence its limit.  Everything else stays with the other forms.
bool bigla_seg_supported(const BiglaParams& p) {
    if (!((p.dk == 16 && p.dv == 32) || (p.dk == 32 && p.dv == 32) || (p.dk == 32 && p.dv == 64) || (p.dk == 64 && p.dv == 64))) return false;
    if ((int64_t)p.B * p.H > 65535) return false;
    const int unit = p.dtype == VIG_DTYPE_F32 ? 4 : 8;
    auto ok = [&](const void* base, const int64_t* s) {
        return !base || (!(reinterpret_cast<uintptr_t>(base) & 15) && s[0] % unit == 0 && s[1] % unit == 0 && s[2] % unit == 0);
    };
    auto ok16 = [](const void* x) { return !(reinterpret_cast<uintptr_t>(x) & 15); };
    return ok(p.q, p.sq) && ok(p.k, p.sk) && ok(p.v, p.sv) && ok(p.gf, p.sgf) && ok(p.gb, p.sgb) && ok(p.o, p.so) && ok16(p.init_f) && ok16(p.init_b) &&
           ok16(p.final_f) && ok16(p.final_b);
}

// Against the tcgen05 forms (16-bit, dv = 64), by the number of 128-token segments in the call; microseconds here / the
// better of theirs at B x H x L:
//   bf16 dk = 64: 1x3x196 11 / 16, 5x6x450 14 / 22, 8x3x1024 21 / 35, 8x3x4096 85 / 79, 128x6x196 90 / 76
//   bf16 dk = 32: 1x3x196 8 / 16, 8x3x1024 15 / 31, 6x12x999 39 / 45, 128x6x196 64 / 68, 32x3x3136 150 / 125, 1x3x16384 49 / 54
//   fp16 (two operand terms): dk = 32 3x3x836 15 / 30, dk = 64 4x12x1000 80 / 41
// Small calls are bound by the latency of one segment, where this form is two to three times shorter; large ones by
// instruction issue, where the persistent forms overlap their phases better.
bool bigla_seg_preferred(const BiglaParams& p) {
    if (p.dtype == VIG_DTYPE_F32 || p.dv != 64) return true;
    const int64_t segs = (int64_t)p.B * p.H * ((p.L + 127) / 128);
    if (p.dtype == VIG_DTYPE_F16) return segs <= (p.dk == 32 ? 200 : 120);
    return segs <= (p.dk == 32 ? (p.L <= 256 ? 1600 : p.L <= 1024 ? 600 : 400) : p.L <= 1024 ? 400 : 200);
}

// Segments of 32 tokens: calls of few segments, whose operands have two or three terms (bigla_seg_launch says why).
static bool seg_fine(int dtype, int dv, int L) { return !(dtype == VIG_DTYPE_BF16 && dv == 64) && L > 64 && L <= (dtype == VIG_DTYPE_F16 && dv == 64 ? 256 : 512); }
static size_t seg_fine_bytes(int64_t BH, int L, int dk, int dv) { return (size_t)BH * ((L + 31) / 32) * 2 * ((size_t)dk * dv + dk) * sizeof(float); }

size_t bigla_seg_workspace(int B, int H, int L, int dk, int dv, int dtype) {
    const int64_t BH = (int64_t)B * H;
    return seg_fine(dtype, dv, L) && BH * ((L + 31) / 32) <= 256 ? seg_fine_bytes(BH, L, dk, dv) : 0;   // asked without a device: a bound for all
}

int bigla_seg_launch(const BiglaParams& p, size_t ws_bytes, cudaStream_t stream) {
    SegParams s{};
    s.p = p;
    s.finals = p.final_f || p.final_b || p.logdecay_f || p.logdecay_b;
    // 64-token segments where more SMs can share the work of few sequences (1x3x196 dk = 64: 11 us against 13) and for dv = 32,
    // whose segments are too little work for eight warps (64x12x196 dk = 16: 46 us against 56; 64x6x784 91 / 114, 64x3x3136 154 / 215; dk = 32 161 / 155);
    // otherwise 128, half as many states.  Clusters of more than eight want room around them: fp16 32/64 1x3x836 12.6 / 16.7, bf16 1x3x1024
    // 10.6 / 12.5, 64/64 1x6x784 14.5 / 16.5, but 1x12x784 (156 segments) 18.7 / 16.6 and 3x3x836 (126) no difference.
    // 32 tokens where operands have two or three terms and all segments find an SM of their own, clusters placed whole (us of a launch at 32 / 64
    // tokens): fp32 2x3x196 64/64 14.4 / 19.9, 4x3x256 32/64 11.9 / 13.2, 2x3x512 16/32 9.3 / 10.2; fp16 1x3x196 32/64 9.0 / 10.4, but 3x3x480 (135
    // segments) 12.4 / 11.5, 1x3x512 11.3 / 11.3, 64/64 1x6x196 13.1 / 13.7, 1x3x400 15.9 / 14.2; bf16 32/32 2x12x128 7.8 / 9.0; fp16 16/32 1x24x49 6.5 / 5.9, 1x24x98 6.8 / 7.4.
    // One-term operands gain nothing: bf16 1x3x196 32/64 8.4 / 8.5,
    // 1x12x196 64/64 11.9 / 11.1.
    // Final states are summed over all segments by the one scanned last, so there calls take fewer.  One direction with states at both ends, 32 / 64 tokens: fp16 64/64
    // 3x100 15.8 / 11.1, 3x196 18.4 / 12.6, 32/64 3x196 11.0 / 8.4; fp32 64/64 3x100 11.4 / 12.1, 6x300 13.7 / 13.3, 6x512 18.9 / 18.3, 16/32 6x512 8.8 / 8.1; 64 / 128
    // tokens: bf16 64/64 3x700 15.5 / 13.8, 6x1000 18.4 / 16.9, 32/64 6x700 10.5 / 9.3; fp16 64/64 6x700 17.1 / 15.8, 32/64 6x850 11.7 / 12.3.
    const int64_t BH = (int64_t)p.B * p.H;
    const bool fine = seg_fine(p.dtype, p.dv, p.L) && !(s.finals && (p.L > 256 || (p.dtype == VIG_DTYPE_F16 && p.dv == 64)));
    const int tok = fine && 3 * BH * ((p.L + 31) / 32) <= 2 * device_sms() && ws_bytes >= seg_fine_bytes(BH, p.L, p.dk, p.dv) ? 32
                    : p.dtype == VIG_DTYPE_F32 || p.dv == 32 || p.L <= 64 || (p.L <= (s.finals ? 512 : 1024) && 3 * BH * ((p.L + 63) / 64) <= (p.L <= 512 ? 3 : 2) * device_sms()) ? 64 : 128;
    switch (p.dtype) {
        case VIG_DTYPE_F32: return seg_launch_dims<float>(s, tok, stream);
        case VIG_DTYPE_BF16: return seg_launch_dims<__nv_bfloat16>(s, tok, stream);
        case VIG_DTYPE_F16: return seg_launch_dims<__half>(s, tok, stream);
    }
    return VIG_ERR_DTYPE;
}

}  // namespace vig
