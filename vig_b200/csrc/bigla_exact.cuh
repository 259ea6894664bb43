// Token-by-token recurrences with a [DK][DV] state in the registers of a group of threads: what the tensor-core forms fall back
// to for a segment or chunk whose gates they cannot factor.  Any gates, log-gates of -inf and growing ones included; fp32 sums.
//
// Bound by instruction issue and the chain from token to token.  A thread holds DPT key channels x JPT value columns, so that a
// token costs it a few 16-byte loads of shared memory for 4 to 32 state values; the DG threads that share value columns are
// neighbouring lanes, and the parts of q S of four tokens meet in one reduce-scatter over them.
#pragma once
#include "mma_common.cuh"

namespace vig {
namespace rec {

constexpr int GROUP = 4;                                                 // tokens handled together; staged rows are padded to a multiple

// NTH threads; with HALVES = 2 each half of them runs a recurrence of its own (the two directions, or S and its adjoint), where
// that leaves a thread no more than 32 state values: twice the arithmetic for each load and half the steps
template <int DK, int DV, int NTH> struct Lay {
    static constexpr int HALVES = DK * DV * 2 / NTH <= 32 ? 2 : 1, HT = NTH / HALVES;
    static constexpr int PER = DK * DV / HT, DPT = PER >= 32 ? 8 : PER >= 8 ? 4 : 2, JPT = PER / DPT, DG = DK / DPT;
    static_assert(DPT * JPT * HT == DK * DV && DG >= 2 && DG <= 16 && (JPT == 1 || JPT == 2 || JPT == 4) && HT % 32 == 0, "state layout");
    __device__ static int half() { return (int)threadIdx.x / HT; }
    __device__ static int d0() { return (int)threadIdx.x % DG * DPT; }   // my key channels and value columns
    __device__ static int j0() { return (int)threadIdx.x % HT / DG * JPT; }
};

template <int N> __device__ __forceinline__ void take(float (&x)[N], const float* p) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4) { const float4 v = *reinterpret_cast<const float4*>(p + i); x[i] = v.x; x[i + 1] = v.y; x[i + 2] = v.z; x[i + 3] = v.w; }
    } else if constexpr (N == 2) { const float2 v = *reinterpret_cast<const float2*>(p); x[0] = v.x; x[1] = v.y; }
    else { x[0] = p[0]; }
}

__device__ __forceinline__ int padded(int n) { return (n + GROUP - 1) / GROUP * GROUP; }

// Rows of a block of n tokens -> fp32 rows of shared memory, all four tensors' loads in flight together; q, k and v times their
// factors, gates as log-gates (lg, may be null) and decay factors a.  Padding rows: q = k = v = 0, gate 0, decay 1.  q may be
// null.  tid: of HT threads.
template <int DK, int DV, int HT, typename T>
__device__ __forceinline__ void stage(float* sq, float* sk, float* sv, float* lg, float* a, const T* q, int64_t lq, float qmul, const T* k, int64_t lk, float kmul, const T* v,
                                      int64_t lv, const T* g, int64_t lgs, int n, float gate_norm, float clamp_min, int tid) {
    constexpr int VP = DV / DK;                                          // pairs of v for each pair of k
#pragma unroll 4
    for (int i = tid; i < padded(n) * (DK / 2); i += HT) {
        const int r = i / (DK / 2), c = i % (DK / 2) * 2;
        float2 xq = make_float2(0.f, 0.f), xk = xq, xg = xq, xv[VP];
#pragma unroll
        for (int e = 0; e < VP; ++e) xv[e] = xq;
        if (r < n) {
            xk = mm::load2_coherent<T>(k + r * lk + c);
            if (q) xq = mm::load2_coherent<T>(q + r * lq + c);
            xg = mm::load2_coherent<T>(g + r * lgs + c);
#pragma unroll
            for (int e = 0; e < VP; ++e) xv[e] = mm::load2_coherent<T>(v + r * lv + c * VP + 2 * e);
            xg = make_float2(gate_transform(xg.x, gate_norm, clamp_min), gate_transform(xg.y, gate_norm, clamp_min));
        }
        *reinterpret_cast<float2*>(sk + r * DK + c) = make_float2(xk.x * kmul, xk.y * kmul);
        if (q) *reinterpret_cast<float2*>(sq + r * DK + c) = make_float2(xq.x * qmul, xq.y * qmul);
        if (lg) *reinterpret_cast<float2*>(lg + r * DK + c) = xg;
        *reinterpret_cast<float2*>(a + r * DK + c) = make_float2(__expf(xg.x), __expf(xg.y));
#pragma unroll
        for (int e = 0; e < VP; ++e) *reinterpret_cast<float2*>(sv + r * DV + c * VP + 2 * e) = xv[e];
    }
}

// S = diag(a) S + k^T v (rows already offset to my channels and columns)
template <int DPT, int JPT> __device__ __forceinline__ void update(float (&S)[JPT][DPT], const float* a, const float* k, const float* v) {
    float av[DPT], kv[DPT], vv[JPT];
    take(av, a); take(kv, k); take(vv, v);
#pragma unroll
    for (int j = 0; j < JPT; ++j)
#pragma unroll
        for (int d = 0; d < DPT; ++d) S[j][d] = fmaf(S[j][d], av[d], kv[d] * vv[j]);
}
// the adjoint's step: Z = diag(a) (Z + k^T v)
template <int DPT, int JPT> __device__ __forceinline__ void update_adjoint(float (&S)[JPT][DPT], const float* a, const float* k, const float* v) {
    float av[DPT], kv[DPT], vv[JPT];
    take(av, a); take(kv, k); take(vv, v);
#pragma unroll
    for (int j = 0; j < JPT; ++j)
#pragma unroll
        for (int d = 0; d < DPT; ++d) S[j][d] = fmaf(kv[d], vv[j], S[j][d]) * av[d];
}
// my channels' part of my columns of q S
template <int DPT, int JPT> __device__ __forceinline__ void read_out(float* o, const float (&S)[JPT][DPT], const float* q) {
    float qv[DPT];
    take(qv, q);
#pragma unroll
    for (int j = 0; j < JPT; ++j) {
        o[j] = 0.f;
#pragma unroll
        for (int d = 0; d < DPT; ++d) o[j] = fmaf(qv[d], S[j][d], o[j]);
    }
}
// Sums of N values over DG neighbouring lanes; each lane is left with its share: returns the index of its first value, or -1
// where another lane has the same one.
template <int DG, int N> __device__ __forceinline__ int reduce_scatter(float (&v)[N]) {
    int at = 0, n = N;
    bool mine = true;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int m = DG / 2; m >= 1; m >>= 1) {
        const bool hi = lane & m;
        if (n > 1) {
            n /= 2;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                if (i < n) {
                    const float send = hi ? v[i] : v[i + n], keep = hi ? v[i + n] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                }
            }
            if (hi) at += n;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
            mine = mine && !hi;
        }
    }
    return mine ? at : -1;
}
template <int DG, int N> struct Share { static constexpr int V = N > DG ? N / DG : 1; };

// Tokens of a block in scan order, GROUP at a time: f(i) for each
template <typename F> __device__ __forceinline__ void each(int m, bool down, F f) {
    const int np = padded(m);
#pragma unroll 1
    for (int i0 = 0; i0 < np; i0 += GROUP)
#pragma unroll
        for (int u = 0; u < GROUP; ++u) f(down ? np - 1 - i0 - u : i0 + u);
}

}  // namespace rec
}  // namespace vig
