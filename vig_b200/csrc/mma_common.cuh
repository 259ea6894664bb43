// Register-level tensor-core building blocks (mma.sync m16n8k16, ldmatrix) for the chunked bi-GLA kernels whose operands
// change with every chunk and head size: the backward pass and the forward at full precision.
//
// Precision: an operand that is not exactly a bf16 number is carried as a sum of bf16 terms, x = t0 + t1 (+ t2) with
// t_i = bf16(x - t_0 - .. - t_{i-1}): two terms hold 16 mantissa bits, three hold fp32's 24.  A product of two such
// operands is the sum of the term products of order < max(terms); accumulation is fp32 in the tensor core.  So bf16 inputs
// enter with one (exact) term, fp16 inputs with two (exact), fp32 inputs with three, and every scaled or intermediate
// operand with two (16-bit callers: 2^-17 relative, far below the rounding of the results) or three (fp32 callers).
#pragma once
#include "tc_common.cuh"

namespace vig {
namespace mm {

using tc::F2; using tc::f2_make; using tc::f2_lo; using tc::f2_hi; using tc::f2_add; using tc::f2_mul; using tc::f2_fma;

constexpr int C = 64;                  // tokens per chunk
constexpr int NT = 256;                // threads per CTA: two warps per 16 rows

template <typename T> struct Terms;    // RAW: terms of an input value, SC: terms of a scaled / intermediate value
template <> struct Terms<__nv_bfloat16> { static constexpr int RAW = 1, SC = 2; };
template <> struct Terms<__half> { static constexpr int RAW = 2, SC = 2; };
template <> struct Terms<float> { static constexpr int RAW = 3, SC = 3; };

// pitch of a bf16 tile row in bytes: 16 bytes of padding make the 8 rows of an ldmatrix hit 8 different 16-byte bank groups
template <int COLS> struct Pitch { static constexpr uint32_t B = COLS * 2 + 16; };

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm2(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void ldsm2t(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, const uint32_t* b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// the same on operands of the type itself
template <typename T> __device__ __forceinline__ void mma_t(float* c, const uint32_t* a, const uint32_t* b);
template <> __device__ __forceinline__ void mma_t<__nv_bfloat16>(float* c, const uint32_t* a, const uint32_t* b) { mma16816(c, a, b); }
template <> __device__ __forceinline__ void mma_t<__half>(float* c, const uint32_t* a, const uint32_t* b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Infinities and NaN among inputs.  In a masked product they would reach the tokens that the mask keeps from them (0 times inf),
// and of an infinity's second term only NaN is left; the recurrences have neither.  ``mark`` becomes NaN once it has seen one;
// packed bf16 pairs are asked by their exponent bits.
__device__ __forceinline__ void see(float& mark, float x) { mark = fmaf(x, 0.f, mark); }
__device__ __forceinline__ void see(F2& mark, F2 x) { mark = f2_fma(x, f2_make(0.f, 0.f), mark); }
__device__ __forceinline__ bool clean(float mark) { return mark == 0.f; }
__device__ __forceinline__ bool clean(F2 mark) { return f2_lo(mark) == 0.f && f2_hi(mark) == 0.f; }
__device__ __forceinline__ uint32_t bf16_unclean(uint4 v) {
    auto bits = [](uint32_t w) { return (w & 0x7F807F80u) + 0x00800080u; };
    return (bits(v.x) | bits(v.y) | bits(v.z) | bits(v.w)) & 0x80008000u;
}

// Lane's address offset inside a tile for the four 8x8 matrices of an ldmatrix.x4 (PITCH in bytes):
//   frag_rows: matrices (rows 0-7, cols 0-7), (rows 8-15, cols 0-7), (rows 0-7, cols 8-15), (rows 8-15, cols 8-15)
//              A operand of a [m][k] tile; with .trans the B operand pair (n tiles 0, 1) of a [k][n] tile
//   frag_cols: matrices (0-7, 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15)
//              B operand pair of an [n][k] tile; with .trans the A operand of a [k][m] tile
template <uint32_t PITCH> __device__ __forceinline__ uint32_t frag_rows(int lane) { return (lane & 15) * PITCH + (lane >> 4) * 16; }
template <uint32_t PITCH> __device__ __forceinline__ uint32_t frag_cols(int lane) { return ((lane & 7) + (lane >> 4) * 8) * PITCH + ((lane >> 3) & 1) * 16; }

// two fp32 values -> NTERM packed bf16 pairs
template <int NTERM> __device__ __forceinline__ void split2(float a, float b, uint32_t* t) {
#pragma unroll
    for (int i = 0; i < NTERM; ++i) {
        t[i] = tc::Pack2<__nv_bfloat16>::pack(a, b);
        if (i + 1 < NTERM) {
            const float2 f = tc::Pack2<__nv_bfloat16>::unpack(t[i]);
            a -= f.x; b -= f.y;
        }
    }
}

// c[g] += a b[g] over one k step for G accumulators, all term pairs of order < max(NA, NB); a[term][4], b[g][term][2].  The
// accumulators alternate, so that a chain of dependent products never waits for its own latency.
// An addition inside the tensor core loses more than a rounding to nearest, and always to the same side: with every product added
// there, fp32 calls at 64 / 64 came out 1.7e-6 from fp64, gradients 1.2e-6.  So with three terms a k step starts from zero, small
// terms first, and joins the accumulator in an ordinary addition: 1.7e-7 both, for 5 - 7 % of the time (16 x 3 x 4096: 499 ->
// 537 us, with gradients 1522 -> 1621); token by token in fp32 it is 2.9e-7.
template <int NA, int NB, int G> __device__ __forceinline__ void mma_group(float (*c)[4], const uint32_t (*a)[4], const uint32_t (*b)[NB][2]) {
    constexpr int ORD = NA > NB ? NA : NB;
    float fresh[G][4];
    float (*d)[4] = ORD == 3 ? fresh : c;
    if constexpr (ORD == 3) {
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int j = 0; j < 4; ++j) fresh[g][j] = 0.f;
    }
#pragma unroll
    for (int o = ORD - 1; o >= 0; --o)               // small terms first
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int j = o - i;
            if (j >= 0 && j < NB) {
#pragma unroll
                for (int g = 0; g < G; ++g) mma16816(d[g], a[i], b[g][j]);
            }
        }
    if constexpr (ORD == 3) {
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int j = 0; j < 4; ++j) c[g][j] += fresh[g][j];
    }
}

template <typename T> __device__ __forceinline__ float2 load2(const T* p);
template <> __device__ __forceinline__ float2 load2<float>(const float* p) { return __ldg(reinterpret_cast<const float2*>(p)); }
template <> __device__ __forceinline__ float2 load2<__nv_bfloat16>(const __nv_bfloat16* p) { return tc::Pack2<__nv_bfloat16>::unpack(__ldg(reinterpret_cast<const uint32_t*>(p))); }
template <> __device__ __forceinline__ float2 load2<__half>(const __half* p) { return tc::Pack2<__half>::unpack(__ldg(reinterpret_cast<const uint32_t*>(p))); }
// the same for kernels that may have begun before the launch that writes what they read
__device__ __forceinline__ uint32_t ld_coherent32(const void* p) { uint32_t v; asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p)); return v; }
template <typename T> __device__ __forceinline__ float2 load2_coherent(const T* p) { return tc::Pack2<T>::unpack(ld_coherent32(p)); }
template <> __device__ __forceinline__ float2 load2_coherent<float>(const float* p) { const uint2 v = ld_coherent(p); return make_float2(__uint_as_float(v.x), __uint_as_float(v.y)); }
template <typename T> __device__ __forceinline__ void store2(T* p, float a, float b);
template <> __device__ __forceinline__ void store2<float>(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
template <> __device__ __forceinline__ void store2<__nv_bfloat16>(__nv_bfloat16* p, float a, float b) { *reinterpret_cast<uint32_t*>(p) = tc::Pack2<__nv_bfloat16>::pack(a, b); }
template <> __device__ __forceinline__ void store2<__half>(__half* p, float a, float b) { *reinterpret_cast<uint32_t*>(p) = tc::Pack2<__half>::pack(a, b); }

// log-gate in log2 units: the short hardware form for 16-bit callers, the exact form for fp32
template <typename T> __device__ __forceinline__ float gate_log2(float x, float gate_norm, float inv_norm, float clamp_min) {
    float g;
    if (sizeof(T) == 4) g = (gate_norm > 0.f ? log_sigmoid(x) / gate_norm : x) * tc::LOG2E;
    else g = tc::fast_gate2(x, gate_norm > 0.f, inv_norm);
    return clamp_min == clamp_min ? fmaxf(g, clamp_min * tc::LOG2E) : g;
}

// log2(1 + 2^y) of a pair, the models' gate form.  The power overflows from y = 128 on; long before that the result is y itself.
__device__ __forceinline__ F2 softplus2(F2 y) {
    const float a = f2_lo(y), b = f2_hi(y);
    const F2 z = f2_add(f2_make(tc::ex2(a), tc::ex2(b)), f2_make(1.f, 1.f));
    return f2_make(a > 100.f ? a : tc::lg2(f2_lo(z)), b > 100.f ? b : tc::lg2(f2_hi(z)));
}

// derivative of the gate transform: d loss / d (gate input x) from d loss / d (log-gate)
__device__ __forceinline__ float through_gate(float dg, float x, float gate_norm, float clamp_min) {
    if (clamp_min == clamp_min) {                                       // the gradient passes where the unclamped gate is at or above the bound
        const float g = gate_norm > 0.f ? log_sigmoid(x) / gate_norm : x;
        if (!(g >= clamp_min)) return 0.f;
    }
    return gate_norm > 0.f ? dg * __fdividef(1.f, 1.f + __expf(x)) / gate_norm : dg;
}

// 2^x: the hardware form for 16-bit callers, the 2-ulp one for fp32
template <typename T> __device__ __forceinline__ float ex2_t(float x) { return sizeof(T) == 4 ? exp2f(x) : tc::ex2(x); }

// [C x COLS] rows of a strided tensor -> TERMS bf16 tiles (rows past n are zero); tile t at dst + t * C * pitch.  One term is
// copied asynchronously: wait_raw() before the barrier that publishes the tiles.
template <typename T, int COLS, int TERMS> __device__ __forceinline__ void load_raw(uint8_t* dst, const T* src, int64_t stride_l, int n, float& mark) {
    constexpr uint32_t P = Pitch<COLS>::B;
    if constexpr (sizeof(T) == 2 && TERMS == 1) {
        constexpr int VPR = COLS / 8;                                  // 16-byte vectors per row
#pragma unroll
        for (int i0 = 0; i0 < C * VPR; i0 += NT) {
            const int i = i0 + threadIdx.x, r = i / VPR, v = i % VPR;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst + r * P + v * 16)), "l"(src + (r < n ? r : 0) * stride_l + v * 8),
                         "r"(r < n ? 16 : 0) : "memory");
        }
    } else {
        constexpr int PPR = COLS / 4;                                  // groups of four values per row
#pragma unroll 4
        for (int i0 = 0; i0 < C * PPR; i0 += NT) {
            const int i = i0 + threadIdx.x, r = i / PPR, v = i % PPR;
            float2 a = make_float2(0.f, 0.f), b = a;
            if (r < n) { a = load2<T>(src + r * stride_l + 4 * v); b = load2<T>(src + r * stride_l + 4 * v + 2); }
            see(mark, a.x); see(mark, a.y); see(mark, b.x); see(mark, b.y);
            uint32_t ta[TERMS], tb[TERMS];
            split2<TERMS>(a.x, a.y, ta); split2<TERMS>(b.x, b.y, tb);
#pragma unroll
            for (int t = 0; t < TERMS; ++t) *reinterpret_cast<uint2*>(dst + t * C * P + r * P + v * 8) = make_uint2(ta[t], tb[t]);
        }
    }
}

// whether the values this thread loaded are finite (after wait_raw(); one-term tiles are looked at where they lie)
template <typename T, int COLS, int TERMS> __device__ __forceinline__ bool raw_clean(const uint8_t* tile, float mark) {
    if constexpr (sizeof(T) == 2 && TERMS == 1) {
        uint32_t bad = 0;
#pragma unroll
        for (int i0 = 0; i0 < C * (COLS / 8); i0 += NT) {
            const int i = i0 + threadIdx.x;
            bad |= bf16_unclean(*reinterpret_cast<const uint4*>(tile + i / (COLS / 8) * Pitch<COLS>::B + i % (COLS / 8) * 16));
        }
        return bad == 0;
    } else return clean(mark);
}

// Thread layout of the per-channel passes over a chunk: thread = (pair of channels, group of RPG consecutive tokens).
template <int DK> struct ColLay {
    static constexpr int PAIRS = DK / 2, GROUPS = NT / PAIRS, RPG = C / GROUPS;
    static_assert(PAIRS <= NT && RPG >= 1, "head size");
};

__device__ __forceinline__ void wait_raw() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Two neighbouring values as they lie in memory.  ``open_gate``: a pair that stands for log-gate 0 (rows past the end) --
// the logit +inf, or the log-gate 0 itself.
template <typename T> struct Raw2 {
    uint32_t w;
    __device__ __forceinline__ void load(const T* p) { w = __ldg(reinterpret_cast<const uint32_t*>(p)); }
    __device__ __forceinline__ void load_coherent(const T* p) { w = ld_coherent32(p); }
    __device__ __forceinline__ void zero() { w = 0u; }
    __device__ __forceinline__ void open_gate(bool logits) { w = logits ? (std::is_same<T, __half>::value ? 0x7C007C00u : 0x7F807F80u) : 0u; }
    __device__ __forceinline__ F2 f2() const {
        if constexpr (std::is_same<T, __half>::value) { const float2 f = tc::Pack2<__half>::unpack(w); return f2_make(f.x, f.y); }
        else return f2_make(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
    }
};
template <> struct Raw2<float> {
    float2 w;
    __device__ __forceinline__ void load(const float* p) { w = __ldg(reinterpret_cast<const float2*>(p)); }
    __device__ __forceinline__ void load_coherent(const float* p) { w = load2_coherent<float>(p); }
    __device__ __forceinline__ void zero() { w = make_float2(0.f, 0.f); }
    __device__ __forceinline__ void open_gate(bool logits) { w.x = w.y = logits ? INFINITY : 0.f; }
    __device__ __forceinline__ F2 f2() const { return f2_make(w.x, w.y); }
};
// The RPG rows of a thread's channel pair, from row r0 of the chunk; rows past the end read the last row (no branch between
// the loads) and are neutralised afterwards.
template <int RPG, typename T> __device__ __forceinline__ void load_rows(Raw2<T> (&x)[RPG], const T* p, int64_t stride_l, int r0, int n) {
    if (r0 + RPG <= n) {                                                 // one addition a row: with a product for each, addresses were a tenth of the instructions
        p += r0 * stride_l;
#pragma unroll
        for (int r = 0; r < RPG; ++r, p += stride_l) x[r].load(p);
    } else {
#pragma unroll
        for (int r = 0; r < RPG; ++r) x[r].load(p + min(r0 + r, n - 1) * stride_l);
    }
}
template <int RPG, typename T> __device__ __forceinline__ void zero_rows(Raw2<T> (&x)[RPG], int r0, int n) {
    if (r0 + RPG > n) {
#pragma unroll
        for (int r = 0; r < RPG; ++r) if (r0 + r >= n) x[r].zero();
    }
}

// Log-gates in log2 units of a thread's rows.  One branch for all rows: with the form chosen row by row the instructions of the
// other forms (log1p, divisions) lie between those of the rows, and fetching around them takes longer than the rows: the loop
// over a chunk's gate gradients took 7800 cycles, 1400 now (backward of 8 x 6 x 4096, 64 / 64, bf16: 609 -> 559 us).
template <int RPG, typename T> __device__ __forceinline__ void row_gates(F2 (&g)[RPG], const Raw2<T> (&x)[RPG], float gate_norm, float clamp_min) {
    const bool logits = gate_norm > 0.f, clamp = clamp_min == clamp_min;
    if (!logits) {
        const F2 log2e = f2_make(tc::LOG2E, tc::LOG2E);
        const float lowest = clamp_min * tc::LOG2E;
#pragma unroll
        for (int r = 0; r < RPG; ++r) {
            g[r] = f2_mul(x[r].f2(), log2e);
            if (clamp) g[r] = f2_make(fmaxf(f2_lo(g[r]), lowest), fmaxf(f2_hi(g[r]), lowest));
        }
    } else if (sizeof(T) == 2 && !clamp) {                               // the models' form: -log2(1 + 2^(-x log2 e)) / norm
        const float ni = -1.f / gate_norm;
        const F2 nlog2e = f2_make(-tc::LOG2E, -tc::LOG2E), ninv = f2_make(ni, ni);
#pragma unroll
        for (int r = 0; r < RPG; ++r) g[r] = f2_mul(softplus2(f2_mul(x[r].f2(), nlog2e)), ninv);
    } else {
        const float inv = 1.f / gate_norm;
#pragma unroll
        for (int r = 0; r < RPG; ++r) {
            const F2 v = x[r].f2();
            g[r] = f2_make(gate_log2<T>(f2_lo(v), gate_norm, inv, clamp_min), gate_log2<T>(f2_hi(v), gate_norm, inv, clamp_min));
        }
    }
}

// Gradients of log-gates -> of the gates' inputs, for a thread's rows; one branch for all of them, as above.
template <int RPG, typename T> __device__ __forceinline__ void rows_through_gate(F2 (&dg)[RPG], const Raw2<T> (&x)[RPG], float gate_norm, float clamp_min) {
    const bool logits = gate_norm > 0.f, clamp = clamp_min == clamp_min;
    if (sizeof(T) == 2 && logits && !clamp) {                            // times 1 / (1 + e^x) / norm
        const float inv = 1.f / gate_norm;
        const F2 log2e = f2_make(tc::LOG2E, tc::LOG2E), norm = f2_make(inv, inv), one = f2_make(1.f, 1.f);
#pragma unroll
        for (int r = 0; r < RPG; ++r) {
            const F2 y = f2_mul(x[r].f2(), log2e), z = f2_add(f2_make(tc::ex2(f2_lo(y)), tc::ex2(f2_hi(y))), one);
            dg[r] = f2_mul(f2_mul(dg[r], norm), f2_make(tc::rcp(f2_lo(z)), tc::rcp(f2_hi(z))));
        }
    } else if (logits || clamp) {
#pragma unroll
        for (int r = 0; r < RPG; ++r) {
            const F2 v = x[r].f2();
            dg[r] = f2_make(through_gate(f2_lo(dg[r]), f2_lo(v), gate_norm, clamp_min), through_gate(f2_hi(dg[r]), f2_hi(v), gate_norm, clamp_min));
        }
    }
}

// Inclusive cumulative log-gates of the chunk in scan order (log2 units): G[r] of my rows; also the sum at the chunk's
// middle (reference of the factorisation) and the total.  gsum: GROUPS x DK floats of shared memory, written again only behind the caller's next barrier; contains one.
template <int DK, typename T> __device__ __forceinline__ void cum_gates(F2 (&G)[ColLay<DK>::RPG], F2& ref, F2& tot, float* gsum, const Raw2<T> (&x)[ColLay<DK>::RPG],
                                                                        int n, int dir, float gate_norm, float clamp_min) {
    using CL = ColLay<DK>;
    const int pr = threadIdx.x % CL::PAIRS, gr = threadIdx.x / CL::PAIRS, r0 = gr * CL::RPG;
    const F2 zero = f2_make(0.f, 0.f), minus = f2_make(-1.f, -1.f);
    row_gates(G, x, gate_norm, clamp_min);
    if (r0 + CL::RPG > n) {
#pragma unroll
        for (int r = 0; r < CL::RPG; ++r) if (r0 + r >= n) G[r] = zero;
    }
#pragma unroll
    for (int r = 1; r < CL::RPG; ++r) G[r] = f2_add(G[r - 1], G[r]);
    *reinterpret_cast<F2*>(gsum + gr * DK + 2 * pr) = G[CL::RPG - 1];
    __syncthreads();
    F2 sum = zero, before = zero, lo = zero;
#pragma unroll
    for (int o = 0; o < CL::GROUPS; ++o) {
        if (o == gr) before = sum;
        if (o == CL::GROUPS / 2) lo = sum;
        sum = f2_add(sum, *reinterpret_cast<const F2*>(gsum + o * DK + 2 * pr));
    }
    tot = sum;
    if (dir) {                                                           // total minus everything before the row
        ref = f2_fma(lo, minus, sum);
        const F2 rest = f2_fma(before, minus, sum);
#pragma unroll
        for (int r = CL::RPG - 1; r > 0; --r) G[r] = f2_fma(G[r - 1], minus, rest);
        G[0] = rest;
    } else {                                                             // what the groups before mine add
        ref = lo;
#pragma unroll
        for (int r = 0; r < CL::RPG; ++r) G[r] = f2_add(G[r], before);
    }
}

// Largest |G - r| (log2 units) of the factorised form.  The exponent's own rounding grows with it (2^-24 |G|): 24 keeps it
// below 2e-6 for fp32 callers, 96 below 1e-5 for 16-bit ones and every scaled operand inside bf16's exponent range.
template <typename T> __device__ __forceinline__ float range_limit() { return sizeof(T) == 4 ? 24.f : 96.f; }

template <typename T> __device__ __forceinline__ const T* head_ptr(const void* base, const int64_t* s, int b, int h, int64_t t0) {
    return reinterpret_cast<const T*>(base) + b * s[0] + h * s[1] + t0 * s[2];
}

// B operands of G neighbouring n tiles (8 columns each) of one k step: [k][n] tile (trans) or [n][k] tile of pitch PB
template <int NB, int G> __device__ __forceinline__ void load_b_nn(uint32_t (*b)[NB][2], uint32_t at, uint32_t b_term) {
    if constexpr (G == 1) {
#pragma unroll
        for (int t = 0; t < NB; ++t) ldsm2t(at + t * b_term, b[0][t]);
    } else {
#pragma unroll
        for (int n = 0; n < G; n += 2)
#pragma unroll
            for (int t = 0; t < NB; ++t) {
                uint32_t r[4];
                ldsm4t(at + t * b_term + n * 16, r);
                b[n][t][0] = r[0]; b[n][t][1] = r[1]; b[n + 1][t][0] = r[2]; b[n + 1][t][1] = r[3];
            }
    }
}
template <int NB, int G, uint32_t PB> __device__ __forceinline__ void load_b_nt(uint32_t (*b)[NB][2], uint32_t at, uint32_t b_term) {
#pragma unroll
    for (int n = 0; n < G; n += 2)
#pragma unroll
        for (int t = 0; t < NB; ++t) {
            uint32_t r[4];
            ldsm4(at + t * b_term + n * 8 * PB, r);
            b[n][t][0] = r[0]; b[n][t][1] = r[1]; b[n + 1][t][0] = r[2]; b[n + 1][t][1] = r[3];
        }
}
// n tiles handled together: four, where there are four
template <int TILES> struct Group { static constexpr int G = TILES < 4 ? TILES : 4; static_assert(TILES % G == 0, "tiles"); };

// acc[NTILES][4] += X^T Y: X [C tokens][DK] scaled tiles (my 16 rows of X^T at column byte offset), Y [C][DV] raw tiles
template <int DK, int DV, int NA, int NB, int NTILES> __device__ __forceinline__ void state_mma(float (*acc)[4], uint32_t x, uint32_t y, int lane) {
    constexpr uint32_t PX = Pitch<DK>::B, PY = Pitch<DV>::B;
    constexpr int G = Group<NTILES>::G;
    x += frag_cols<PX>(lane);
    y += frag_rows<PY>(lane);
#pragma unroll
    for (int ks = 0; ks < C / 16; ++ks) {
        uint32_t a[NA][4];
#pragma unroll
        for (int t = 0; t < NA; ++t) ldsm4t(x + t * C * PX + ks * 16 * PX, a[t]);
#pragma unroll
        for (int n = 0; n < NTILES; n += G) {
            uint32_t b[G][NB][2];
            load_b_nn<NB, G>(b, y + ks * 16 * PY + n * 16, C * PY);
            mma_group<NA, NB, G>(acc + n, a, b);
        }
    }
}

// fp32 states [DK][DV] times a per-row scale -> bf16 terms.  A thread's loads are issued together, ahead of the shared-memory
// writes, which no load passes: one by one each waited for L2 (6600 -> 3300 cycles a chunk and direction; 559 -> 518 us).
template <int DK, int DV> struct StateLay {
    static constexpr int TPR = DV / 4, KN = (DK * TPR + NT - 1) / NT;    // threads of a row (8 .. 16), vectors of a thread
    __device__ static bool mine() { return DK * TPR >= NT || (int)threadIdx.x < DK * TPR; }   // whole warps
};
template <int DK, int DV> __device__ __forceinline__ void fetch_state(float4 (&x)[StateLay<DK, DV>::KN], const float* st) {
    using L = StateLay<DK, DV>;
#pragma unroll
    for (int k = 0; k < L::KN; ++k) x[k] = __ldcg(reinterpret_cast<const float4*>(st) + threadIdx.x + k * NT);
}
template <int DK, int DV, int SC> __device__ __forceinline__ void put_state(uint8_t* dst, const float4 (&x)[StateLay<DK, DV>::KN], const float* scale) {
    using L = StateLay<DK, DV>;
    constexpr uint32_t P = Pitch<DV>::B;
#pragma unroll
    for (int k = 0; k < L::KN; ++k) {
        const int i = threadIdx.x + k * NT, d = i / L::TPR, v = i % L::TPR;
        const float s = scale[d];
        uint32_t ta[SC], tb[SC];
        split2<SC>(x[k].x * s, x[k].y * s, ta); split2<SC>(x[k].z * s, x[k].w * s, tb);
#pragma unroll
        for (int t = 0; t < SC; ++t) *reinterpret_cast<uint2*>(dst + t * DK * P + d * P + v * 8) = make_uint2(ta[t], tb[t]);
    }
}
// carry[d] = <x[d], y[d]>
template <int DK, int DV> __device__ __forceinline__ void state_dots(float* carry, const float4 (&x)[StateLay<DK, DV>::KN], const float4 (&y)[StateLay<DK, DV>::KN]) {
    using L = StateLay<DK, DV>;
#pragma unroll
    for (int k = 0; k < L::KN; ++k) {
        const int i = threadIdx.x + k * NT;
        float a = x[k].x * y[k].x + x[k].y * y[k].y + x[k].z * y[k].z + x[k].w * y[k].w;
#pragma unroll
        for (int m = 1; m < L::TPR; m <<= 1) a += __shfl_xor_sync(0xffffffffu, a, m);
        if (i % L::TPR == 0) carry[i / L::TPR] = a;
    }
}

// acc[2][4] += A_rows B_rows^T over KD: A fragments of my 16 rows (tile a, [row][k]), 16 B rows (tile b, [n][k], pitch PB)
template <int KD, int NA, int NB> __device__ __forceinline__ void block_nt(float (*acc)[4], uint32_t a, uint32_t a_term, uint32_t b, uint32_t b_term) {
#pragma unroll
    for (int ks = 0; ks < KD / 16; ++ks) {
        uint32_t fa[NA][4], fb[2][NB][2];
#pragma unroll
        for (int t = 0; t < NA; ++t) ldsm4(a + t * a_term + ks * 32, fa[t]);
        load_b_nt<NB, 2, 0>(fb, b + ks * 32, b_term);
        mma_group<NA, NB, 2>(acc, fa, fb);
    }
}

// A operand of my 16 rows, all k steps
template <int KD, int NA> __device__ __forceinline__ void load_a(uint32_t (*fa)[NA][4], uint32_t a, uint32_t a_term) {
#pragma unroll
    for (int ks = 0; ks < KD / 16; ++ks)
#pragma unroll
        for (int t = 0; t < NA; ++t) ldsm4(a + t * a_term + ks * 32, fa[ks][t]);
}
// as block_nt with the A operand at hand
template <int KD, int NA, int NB> __device__ __forceinline__ void block_nt(float (*acc)[4], const uint32_t (*fa)[NA][4], uint32_t b, uint32_t b_term) {
#pragma unroll
    for (int ks = 0; ks < KD / 16; ++ks) {
        uint32_t fb[2][NB][2];
        load_b_nt<NB, 2, 0>(fb, b + ks * 32, b_term);
        mma_group<NA, NB, 2>(acc, fa[ks], fb);
    }
}

// zero the entries of a diagonal 16 x 16 block that ``keep(row, col)`` rejects, then split it into an A operand
template <int SC, typename F> __device__ __forceinline__ void mask_split(float (*p)[4], bool diag, int lane, F keep, uint32_t (*out)[4]) {
    if (diag) {
        const int r = lane >> 2, q = 2 * (lane & 3);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j) if (!keep(r + 8 * (j >> 1), nt * 8 + q + (j & 1))) p[nt][j] = 0.f;
    }
    uint32_t t[SC];
    split2<SC>(p[0][0], p[0][1], t);
#pragma unroll
    for (int i = 0; i < SC; ++i) out[i][0] = t[i];
    split2<SC>(p[0][2], p[0][3], t);
#pragma unroll
    for (int i = 0; i < SC; ++i) out[i][1] = t[i];
    split2<SC>(p[1][0], p[1][1], t);
#pragma unroll
    for (int i = 0; i < SC; ++i) out[i][2] = t[i];
    split2<SC>(p[1][2], p[1][3], t);
#pragma unroll
    for (int i = 0; i < SC; ++i) out[i][3] = t[i];
}

// acc[ND/8][4] += A (16 x 16, registers) B: B rows of one k step in a [k][n] tile
template <int ND, int NA, int NB> __device__ __forceinline__ void block_nn(float (*acc)[4], const uint32_t (*a)[4], uint32_t b, uint32_t b_term) {
    constexpr int G = Group<ND / 8>::G;
#pragma unroll
    for (int n = 0; n < ND / 8; n += G) {
        uint32_t fb[G][NB][2];
        load_b_nn<NB, G>(fb, b + n * 16, b_term);
        mma_group<NA, NB, G>(acc + n, a, fb);
    }
}

// acc[ND/8][4] += A B^T over KD: A = my 16 rows, all k steps, B an [n][k] tile of ND rows with pitch PB
template <int ND, int KD, uint32_t PB, int NA, int NB> __device__ __forceinline__ void rows_nt(float (*acc)[4], const uint32_t (*fa)[NA][4], uint32_t b, uint32_t b_term) {
    constexpr int G = Group<ND / 8>::G;
#pragma unroll
    for (int ks = 0; ks < KD / 16; ++ks)
#pragma unroll
        for (int n = 0; n < ND / 8; n += G) {
            uint32_t fb[G][NB][2];
            load_b_nt<NB, G, PB>(fb, b + n * 8 * PB + ks * 32, b_term);
            mma_group<NA, NB, G>(acc + n, fa[ks], fb);
        }
}

}  // namespace mm
}  // namespace vig
