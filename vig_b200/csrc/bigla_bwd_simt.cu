// Backward of the bi-directional gated linear attention (gradients of q, k, v and of both log-gate tensors),
// SIMT fp32.  Replaces, for the merged operator, what the reference's training path does with
// FusedChunkGLAFunction.backward (flash-linear-attention/fla/ops/gla/chunk_fuse.py:413-518): a sweep that
// rebuilds the scan state for dq, a reverse sweep for dk / dv, and the gate gradient as a cumulative sum of
// dq*q - dk*k (chunk_fuse.py:506-516).
//
// For one scan direction, in scan order (a_t = exp(g_t), c = scale * out_scale):
//     S_t  = diag(a_t) S_{t-1} + k_t^T v_t                      o_t = c q_t S_t
//     dq_t = c S_t do_t
//     D_t  = c q_t^T do_t + Z_{t+1},  Z_t = diag(a_t) D_t        (reverse scan order)
//     dk_t = D_t v_t,  dv_t = k_t D_t
//     e_t  = dq_t * q_t - dk_t * k_t ;  dg_t = sum of e over the tokens scanned at or after t
// The kernels are chunk-parallel like the forward SIMT path: local S and Z per 64-token chunk, a scan over
// chunks in each direction, then one CTA per chunk that replays both recurrences from its entering states.
// Exact for any gates.  It is the whole backward where the tensor-core form (bigla_bwd_mma.cu) does not take the call, the
// per-chunk fallback of that form, and it writes either e per direction or the finished gate gradients.
#include <atomic>
#include <cmath>
#include "bigla_bwd.cuh"
#include "mma_common.cuh"

namespace vig {
namespace {

constexpr int CH = BWD_CHUNK;
constexpr int NT = 256;

template <typename T>
__device__ __forceinline__ const T* rowp(const void* base, const int64_t* s, int b, int h, int l) {
    return reinterpret_cast<const T*>(base) + b * s[0] + h * s[1] + (int64_t)l * s[2];
}

template <int D, typename T>
__device__ __forceinline__ void load_tile(float* dst, const void* x, const int64_t* sx, int b, int h, int t0, int n) {
    for (int idx = threadIdx.x; idx < CH * D; idx += NT) {
        const int i = idx / D, d = idx % D;
        dst[idx] = i < n ? DType<T>::to_f(rowp<T>(x, sx, b, h, t0 + i)[d]) : 0.f;
    }
}

// gates of the chunk (raw logits transformed) -> per-channel sum in log2 units to `sum_out` (may be null) -> decay factors
// exp(g) in place
template <int DK, typename T>
__device__ __forceinline__ void load_gates_exp(float* g, const BwdParams& p, int dir, int b, int h, int t0, int n, float* sum_out) {
    load_tile<DK, T>(g, dir ? p.gb : p.gf, dir ? p.sgb : p.sgf, b, h, t0, n);           // rows past the end: log-gate 0, decay 1
    if (p.gate_norm > 0.f || p.clamp_min == p.clamp_min)
        for (int idx = threadIdx.x; idx < n * DK; idx += NT) g[idx] = gate_transform(g[idx], p.gate_norm, p.clamp_min);
    __syncthreads();
    if (threadIdx.x < DK && sum_out) {
        float s = 0.f;
        for (int i = 0; i < CH; ++i) s += g[i * DK + threadIdx.x];
        sum_out[threadIdx.x] = s * tc::LOG2E;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < CH * DK; idx += NT) g[idx] = __expf(g[idx]);
    __syncthreads();
}

// Layout A: thread = (value column j, slice s of DK/TPC key channels).  Layout B: thread = (key channel d,
// slice s of DV/TPB value columns).  A reduces over key channels inside TPC neighbouring lanes, B over value
// columns inside TPB neighbouring lanes.
template <int DK, int DV> struct LayA { static constexpr int TPC = NT / DV, DPT = DK / TPC; };
template <int DK, int DV> struct LayB { static constexpr int TPB = NT / DK, JPT = DV / TPB; };

// ---- phase A: local S (scan order, from zero) and local Z (reverse scan order, from zero) per chunk ------------
template <int DK, int DV, typename T>
__global__ void __launch_bounds__(NT) bwd_chunk_states(BwdParams p) {
    using A = LayA<DK, DV>;
    extern __shared__ float smem[];
    float* sq = smem;
    float* sk = sq + CH * DK;
    float* sg = sk + CH * DK;
    float* sv = sg + CH * DK;
    float* sdo = sv + CH * DV;
    const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H;
    const int t0 = c * CH, n = min(CH, p.L - t0);
    const int j = threadIdx.x / A::TPC, s = threadIdx.x % A::TPC;
    load_tile<DK, T>(sq, p.q, p.sq, b, h, t0, n);
    load_tile<DK, T>(sk, p.k, p.sk, b, h, t0, n);
    load_tile<DV, T>(sv, p.v, p.sv, b, h, t0, n);
    load_tile<DV, T>(sdo, p.dout, p.sdo, b, h, t0, n);
    for (int dir = 0; dir < 2; ++dir) {
        if (!(p.dir_mask & (1 << dir))) continue;
        const size_t slot = ((size_t)bh * p.nchunk + c) * 2 + dir;
        __syncthreads();
        load_gates_exp<DK, T>(sg, p, dir, b, h, t0, n, p.ws_decay + slot * DK);
        float st[A::DPT];
#pragma unroll
        for (int dd = 0; dd < A::DPT; ++dd) st[dd] = 0.f;
        for (int ii = 0; ii < n; ++ii) {                              // S: scan order
            const int i = dir ? n - 1 - ii : ii;
            const float vj = sv[i * DV + j];
#pragma unroll
            for (int dd = 0; dd < A::DPT; ++dd) {
                const int d = s * A::DPT + dd;
                st[dd] = fmaf(st[dd], sg[i * DK + d], sk[i * DK + d] * vj);
            }
        }
#pragma unroll
        for (int dd = 0; dd < A::DPT; ++dd) p.ws_S[slot * DK * DV + (s * A::DPT + dd) * DV + j] = st[dd];
#pragma unroll
        for (int dd = 0; dd < A::DPT; ++dd) st[dd] = 0.f;
        for (int ii = n - 1; ii >= 0; --ii) {                         // Z: reverse scan order, add then decay
            const int i = dir ? n - 1 - ii : ii;
            const float dj = p.c * sdo[i * DV + j];
#pragma unroll
            for (int dd = 0; dd < A::DPT; ++dd) {
                const int d = s * A::DPT + dd;
                st[dd] = (st[dd] + sq[i * DK + d] * dj) * sg[i * DK + d];
            }
        }
#pragma unroll
        for (int dd = 0; dd < A::DPT; ++dd) p.ws_Z[slot * DK * DV + (s * A::DPT + dd) * DV + j] = st[dd];
    }
}

// N values of a row from x; vec: on 16 bytes, as folded contributions are (vig_bigla_bwd_full)
template <int N> __device__ __forceinline__ void load_row(float (&y)[N], const float* x, bool vec) {
    if (N % 4 == 0 && vec) {
#pragma unroll
        for (int i = 0; i < N; i += 4) { const float4 t = *reinterpret_cast<const float4*>(x + i); y[i] = t.x; y[i + 1] = t.y; y[i + 2] = t.z; y[i + 3] = t.w; }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) y[i] = x[i];
    }
}

// Values d * dv + e0 .. e0 + N - 1 of the state and of the adjoint state entering chunk c, and <state leaving the chunk, adjoint state entering from there>
// over these.  Where no launch has summed the contributions (p.scanned = 0) they are summed here, a thread's values of both states at a time: one by one
// each waited for the one before.  Training steps of bf16 64x3x384, 64/64, with the forward gates of every chunk out of range: 2180 us (one by one
// 3980, a launch that sums them 2184), of one chunk 461 (725, 531).
template <int N> __device__ __forceinline__ float entering(float (&S)[N], float (&Z)[N], const BwdParams& p, int bh, int c, int dir, int d, int e0) {
    const int per = p.dk * p.dv, at = d * p.dv + e0, next = dir ? c - 1 : c + 1;
    const size_t row = (size_t)bh * p.nchunk;
    const bool goes_on = next >= 0 && next < p.nchunk;
    float leaving[N], past = 0.f;
    if (p.scanned) {
        load_row(S, p.ws_S + ((row + c) * 2 + dir) * per + at, false);
        load_row(Z, p.ws_Z + ((row + c) * 2 + dir) * per + at, false);
        if (goes_on) load_row(leaving, p.ws_S + ((row + next) * 2 + dir) * per + at, false);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) S[i] = Z[i] = 0.f;
        const int before = dir ? p.nchunk - 1 - c : c, behind = p.nchunk - 1 - before;   // chunks scanned ahead of this one, and after it
#pragma unroll 1
        for (int g = 0; g < max(before, behind); ++g) {
            const size_t sa = (row + (dir ? p.nchunk - 1 - g : g)) * 2 + dir, sz = (row + (dir ? g : p.nchunk - 1 - g)) * 2 + dir;
            float x[N], y[N], a = 0.f, z = 0.f;
            if (g < before) { load_row(x, p.ws_S + sa * per + at, true); a = p.ws_decay[sa * p.dk + d]; }
            if (g < behind) { load_row(y, p.ws_Z + sz * per + at, true); z = p.ws_decay[sz * p.dk + d]; }
            a = exp2f(a); z = exp2f(z);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (g < before) S[i] = fmaf(S[i], a, x[i]);
                if (g < behind) Z[i] = fmaf(Z[i], z, y[i]);
            }
        }
        if (goes_on) {
            load_row(leaving, p.ws_S + ((row + c) * 2 + dir) * per + at, true);
            const float a = exp2f(p.ws_decay[((row + c) * 2 + dir) * p.dk + d]);
#pragma unroll
            for (int i = 0; i < N; ++i) leaving[i] = fmaf(S[i], a, leaving[i]);
        }
    }
    if (goes_on) {
#pragma unroll
        for (int i = 0; i < N; ++i) past = fmaf(leaving[i], Z[i], past);
    }
    return past;
}

// ---- phase C: gradients of one chunk -----------------------------------------------------------------------------
template <int DK, int DV, typename T>
__global__ void __launch_bounds__(NT) bwd_chunk_grads(BwdParams p, int flagged_only) {
    using A = LayA<DK, DV>;
    using Bl = LayB<DK, DV>;
    extern __shared__ float smem[];
    float* sq = smem;
    float* sk = sq + CH * DK;
    float* sg = sk + CH * DK;
    float* se = sg + CH * DK;              // dq*q - dk*k of the current direction
    float* sdq = se + CH * DK;
    float* sdk = sdq + CH * DK;
    float* sv = sdk + CH * DK;
    float* sdo = sv + CH * DV;
    float* sdv = sdo + CH * DV;
    __shared__ float carry[DK];            // gradient of the log-gates just past the chunk
    pdl_wait();
    const bool have_states = !flagged_only || p.nchunk > 1;          // the tensor-core form leaves the states of a lone chunk unwritten (zero)
    const int items = p.nchunk * p.B * p.H;
    for (int item = blockIdx.x, look = 0; item < items; item += gridDim.x, ++look) {
    if (flagged_only) {
        // the flags of my next NT items at once: a chain of dependent loads otherwise
        if (look % NT == 0) {
            const int64_t mine = item + (int64_t)threadIdx.x * gridDim.x;
            if (!__syncthreads_or(mine < items && p.flags[mine])) {
                const int64_t next = item + (int64_t)(NT - 1) * gridDim.x;
                if (next >= items) break;
                item = (int)next; look += NT - 1;
                continue;
            }
        }
        if (!p.flags[item]) continue;
    }
    const int c = item % p.nchunk, bh = item / p.nchunk, b = bh / p.H, h = bh % p.H;
    const int t0 = c * CH, n = min(CH, p.L - t0);
    load_tile<DK, T>(sq, p.q, p.sq, b, h, t0, n);
    load_tile<DK, T>(sk, p.k, p.sk, b, h, t0, n);
    load_tile<DV, T>(sv, p.v, p.sv, b, h, t0, n);
    load_tile<DV, T>(sdo, p.dout, p.sdo, b, h, t0, n);
    for (int idx = threadIdx.x; idx < CH * DK; idx += NT) { sdq[idx] = 0.f; sdk[idx] = 0.f; }
    for (int idx = threadIdx.x; idx < CH * DV; idx += NT) sdv[idx] = 0.f;
    for (int dir = 0; dir < 2; ++dir) {
        if (!(p.dir_mask & (1 << dir))) continue;
        const size_t slot = ((size_t)bh * p.nchunk + c) * 2 + dir;
        __syncthreads();
        load_gates_exp<DK, T>(sg, p, dir, b, h, t0, n, nullptr);
        const int d = threadIdx.x / Bl::TPB, s = threadIdx.x % Bl::TPB;
        float st[Bl::JPT], adj[Bl::JPT], past = 0.f;
#pragma unroll
        for (int jj = 0; jj < Bl::JPT; ++jj) st[jj] = adj[jj] = 0.f;
        if (have_states) past = entering(st, adj, p, bh, c, dir, d, s * Bl::JPT);
#pragma unroll
        for (int m = 1; m < Bl::TPB; m <<= 1) past += __shfl_xor_sync(0xffffffffu, past, m);
        if (s == 0) carry[d] = past;
        {   // layout A: dv from Z (reverse scan order)
            const int j = threadIdx.x / A::TPC, s = threadIdx.x % A::TPC;
            float st[A::DPT];
#pragma unroll
            for (int dd = 0; dd < A::DPT; ++dd) st[dd] = have_states && p.scanned ? p.ws_Z[slot * DK * DV + (s * A::DPT + dd) * DV + j] : 0.f;
            if constexpr (DK * DV <= CH * DK) {
                if (have_states && !p.scanned) {                         // summed by the threads of layout B; se is not in use yet
#pragma unroll
                    for (int jj = 0; jj < Bl::JPT; ++jj) se[threadIdx.x * Bl::JPT + jj] = adj[jj];
                    __syncthreads();
#pragma unroll
                    for (int dd = 0; dd < A::DPT; ++dd) st[dd] = se[(s * A::DPT + dd) * DV + j];
                    __syncthreads();
                }
            }
            for (int ii = n - 1; ii >= 0; --ii) {
                const int i = dir ? n - 1 - ii : ii;
                const float dj = p.c * sdo[i * DV + j];
                float acc = 0.f;
#pragma unroll
                for (int dd = 0; dd < A::DPT; ++dd) {
                    const int d = s * A::DPT + dd;
                    const float ds = fmaf(sq[i * DK + d], dj, st[dd]);
                    acc = fmaf(sk[i * DK + d], ds, acc);
                    st[dd] = ds * sg[i * DK + d];
                }
#pragma unroll
                for (int m = 1; m < A::TPC; m <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
                if (s == 0) sdv[i * DV + j] += acc;
            }
        }
        {   // layout B: dq from the rebuilt state (scan order), then dk from Z (reverse scan order)
            for (int ii = 0; ii < n; ++ii) {
                const int i = dir ? n - 1 - ii : ii;
                const float a = sg[i * DK + d], kd = sk[i * DK + d];
                float acc = 0.f;
#pragma unroll
                for (int jj = 0; jj < Bl::JPT; ++jj) {
                    const int j = s * Bl::JPT + jj;
                    st[jj] = fmaf(st[jj], a, kd * sv[i * DV + j]);
                    acc = fmaf(st[jj], sdo[i * DV + j], acc);
                }
#pragma unroll
                for (int m = 1; m < Bl::TPB; m <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
                if (s == 0) {
                    const float dqd = p.c * acc;
                    sdq[i * DK + d] += dqd;
                    se[i * DK + d] = dqd * sq[i * DK + d];
                }
            }
            for (int ii = n - 1; ii >= 0; --ii) {
                const int i = dir ? n - 1 - ii : ii;
                const float a = sg[i * DK + d], cq = p.c * sq[i * DK + d];
                float acc = 0.f;
#pragma unroll
                for (int jj = 0; jj < Bl::JPT; ++jj) {
                    const int j = s * Bl::JPT + jj;
                    const float ds = fmaf(cq, sdo[i * DV + j], adj[jj]);
                    acc = fmaf(ds, sv[i * DV + j], acc);
                    adj[jj] = ds * a;
                }
#pragma unroll
                for (int m = 1; m < Bl::TPB; m <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
                if (s == 0) {
                    sdk[i * DK + d] += acc;
                    se[i * DK + d] -= acc * sk[i * DK + d];
                }
            }
        }
        __syncthreads();
        if (float* e_dir = dir ? p.eb : p.ef) {
            float* e_out = e_dir + ((size_t)bh * p.L + t0) * DK;
            for (int idx = threadIdx.x; idx < n * DK; idx += NT) e_out[idx] = se[idx];
        }
        if (void* dg = dir ? p.dgb : p.dgf) {
            // finished gate gradient: the value just past the chunk plus the sum of e over the tokens scanned at or after t;
            // then the derivative of the gate transform
            if (threadIdx.x < DK) {
                const int d = threadIdx.x;
                float run = carry[d];
                for (int ii = n - 1; ii >= 0; --ii) {
                    const int i = dir ? n - 1 - ii : ii;
                    run += se[i * DK + d];
                    float g = run;
                    if (p.gate_norm > 0.f || p.clamp_min == p.clamp_min) {
                        const float x = DType<T>::to_f(rowp<T>(dir ? p.gb : p.gf, dir ? p.sgb : p.sgf, b, h, t0 + i)[d]);
                        g = mm::through_gate(g, x, p.gate_norm, p.clamp_min);
                    }
                    const size_t at = ((size_t)bh * p.L + t0 + i) * DK + d;
                    if (p.dg_f32) reinterpret_cast<float*>(dg)[at] = g;
                    else reinterpret_cast<T*>(dg)[at] = DType<T>::from_f(g);
                }
            }
        }
    }
    __syncthreads();
    T* dq = reinterpret_cast<T*>(p.out_dq) + ((size_t)bh * p.L + t0) * DK;
    T* dk = reinterpret_cast<T*>(p.out_dk) + ((size_t)bh * p.L + t0) * DK;
    T* dv = reinterpret_cast<T*>(p.out_dv) + ((size_t)bh * p.L + t0) * DV;
    for (int idx = threadIdx.x; idx < n * DK; idx += NT) { dq[idx] = DType<T>::from_f(sdq[idx]); dk[idx] = DType<T>::from_f(sdk[idx]); }
    for (int idx = threadIdx.x; idx < n * DV; idx += NT) dv[idx] = DType<T>::from_f(sdv[idx]);
    __syncthreads();
    }
}

template <int DK, int DV, typename T>
int launch_typed(const BwdParams& p, int flagged_only, cudaStream_t stream) {
    dim3 grid(p.nchunk, p.B * p.H);
    const size_t smA = (size_t)CH * (3 * DK + 2 * DV) * sizeof(float);
    const size_t smC = (size_t)CH * (6 * DK + 3 * DV) * sizeof(float);
    auto kA = bwd_chunk_states<DK, DV, T>;
    auto kC = bwd_chunk_grads<DK, DV, T>;
    cudaError_t e;
    if ((e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kC), (int)smC)) != cudaSuccess) return (int)e;
    if (!flagged_only) {
        if ((e = tc::ensure_smem_attr(reinterpret_cast<const void*>(kA), (int)smA)) != cudaSuccess) return (int)e;
        kA<<<grid, NT, smA, stream>>>(p);
        if (int st = bigla_bwd_scan_launch(p, stream)) return st;
    }
    const int items = p.nchunk * p.B * p.H;
    // flagged chunks are rare: as many CTAs as the GPU holds walk the flags (one an SM at 64 / 64, four at 16 / 32); as one
    // CTA per chunk the launch alone took 15 us for 3072 unflagged chunks
    int ctas = items;
    if (flagged_only) {
        static std::atomic<int> per_sm{0};                               // a property of the kernel, the same on every B200
        int fit = per_sm.load();
        if (!fit) {
            if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kC, NT, smC)) != cudaSuccess) return (int)e;
            per_sm.store(fit = fit < 1 ? 1 : fit);
        }
        ctas = items < fit * device_sms() ? items : fit * device_sms();
    }
    return (int)launch_next(kC, dim3(ctas), dim3(NT), smC, stream, p, flagged_only);
}

template <typename T>
int launch_dims(const BwdParams& p, int flagged_only, cudaStream_t stream) {
#define VIG_CASE(DKV, DVV) if (p.dk == DKV && p.dv == DVV) return launch_typed<DKV, DVV, T>(p, flagged_only, stream);
    VIG_CASE(16, 32) VIG_CASE(32, 32) VIG_CASE(32, 64) VIG_CASE(64, 64) VIG_CASE(64, 128)   // larger heads exceed shared memory
#undef VIG_CASE
    return VIG_ERR_SHAPE;
}

void fill(int64_t* dst, const int64_t* src, int H, int L, int d) {
    if (src) { dst[0] = src[0]; dst[1] = src[1]; dst[2] = src[2]; }
    else { dst[0] = (int64_t)H * L * d; dst[1] = (int64_t)L * d; dst[2] = d; }
}

}  // namespace
}  // namespace vig

using namespace vig;

static size_t bwd_ws_bytes(int B, int H, int L, int dk, int dv) {
    const size_t nchunk = (L + BWD_CHUNK - 1) / BWD_CHUNK;
    return (size_t)B * H * nchunk * 2 * (2 * (size_t)dk * dv + dk) * sizeof(float);
}

static int bwd_fill(BwdParams& p, const void* q, const void* k, const void* v, const void* g_fwd, const void* g_bwd, const void* d_out,
                    void* dq, void* dk_out, void* dv_out, int B, int H, int L, int dk, int dv, int dtype,
                    const int64_t* strides_q, const int64_t* strides_k, const int64_t* strides_v,
                    const int64_t* strides_gf, const int64_t* strides_gb, const int64_t* strides_do,
                    float scale, float out_scale, int dir_mask, void* workspace) {
    if (dtype < 0 || dtype > 2) return VIG_ERR_DTYPE;
    if (B < 0 || H <= 0 || L < 0) return VIG_ERR_SHAPE;
    if (dir_mask < 1 || dir_mask > 3) return VIG_ERR_ARG;
    if (B == 0 || L == 0) return VIG_OK;
    if (!q || !k || !v || !d_out || !dq || !dk_out || !dv_out) return VIG_ERR_NULL;
    if (((dir_mask & 1) && !g_fwd) || ((dir_mask & 2) && !g_bwd)) return VIG_ERR_NULL;
    p.q = q; p.k = k; p.v = v; p.gf = g_fwd; p.gb = g_bwd; p.dout = d_out;
    p.out_dq = dq; p.out_dk = dk_out; p.out_dv = dv_out;
    fill(p.sq, strides_q, H, L, dk); fill(p.sk, strides_k, H, L, dk); fill(p.sv, strides_v, H, L, dv);
    fill(p.sgf, strides_gf, H, L, dk); fill(p.sgb, strides_gb, H, L, dk); fill(p.sdo, strides_do, H, L, dv);
    p.B = B; p.H = H; p.L = L; p.dk = dk; p.dv = dv; p.dtype = dtype;
    if (scale < 0.f) scale = 1.0f / sqrtf((float)dk);
    p.c = scale * out_scale;
    p.gate_norm = 0.f; p.clamp_min = nanf("");
    p.dir_mask = dir_mask;
    p.nchunk = (L + BWD_CHUNK - 1) / BWD_CHUNK;
    p.scanned = 1;
    const size_t states = bwd_state_floats(B, H, p.nchunk, dk, dv);
    p.ws_S = reinterpret_cast<float*>(workspace);
    p.ws_Z = p.ws_S + states;
    p.ws_decay = p.ws_Z + states;
    p.flags = reinterpret_cast<int32_t*>(p.ws_decay + (size_t)B * H * p.nchunk * 2 * dk);   // past vig_bigla_bwd's workspace, which has none
    return VIG_OK;
}

static int bwd_simt(const BwdParams& p, int flagged_only, cudaStream_t stream) {
    switch (p.dtype) {
        case VIG_DTYPE_F32: return launch_dims<float>(p, flagged_only, stream);
        case VIG_DTYPE_BF16: return launch_dims<__nv_bfloat16>(p, flagged_only, stream);
        case VIG_DTYPE_F16: return launch_dims<__half>(p, flagged_only, stream);
    }
    return VIG_ERR_DTYPE;
}

extern "C" size_t vig_bigla_bwd_workspace_bytes(int B, int H, int L, int dk, int dv) {
    if (B <= 0 || H <= 0 || L <= 0 || dk <= 0 || dv <= 0) return 0;
    return bwd_ws_bytes(B, H, L, dk, dv);
}

extern "C" int vig_bigla_bwd(const void* q, const void* k, const void* v, const void* g_fwd, const void* g_bwd, const void* d_out,
                             void* dq, void* dk_out, void* dv_out, float* e_fwd, float* e_bwd,
                             int B, int H, int L, int dk, int dv, int dtype,
                             const int64_t* strides_q, const int64_t* strides_k, const int64_t* strides_v,
                             const int64_t* strides_gf, const int64_t* strides_gb, const int64_t* strides_do,
                             float scale, float out_scale, int dir_mask,
                             void* workspace, size_t workspace_bytes, void* stream) {
    BwdParams p{};
    const int s = bwd_fill(p, q, k, v, g_fwd, g_bwd, d_out, dq, dk_out, dv_out, B, H, L, dk, dv, dtype, strides_q, strides_k, strides_v,
                           strides_gf, strides_gb, strides_do, scale, out_scale, dir_mask, workspace);
    if (s || B == 0 || L == 0) return s;
    if (((dir_mask & 1) && !e_fwd) || ((dir_mask & 2) && !e_bwd)) return VIG_ERR_NULL;
    if (!workspace || workspace_bytes < bwd_ws_bytes(B, H, L, dk, dv)) return VIG_ERR_WORKSPACE;
    if (reinterpret_cast<uintptr_t>(workspace) & 3) return VIG_ERR_ALIGN;
    p.ef = e_fwd; p.eb = e_bwd;
    return bwd_simt(p, 0, (cudaStream_t)stream);
}

extern "C" size_t vig_bigla_bwd_full_workspace_bytes(int B, int H, int L, int dk, int dv) {
    if (B <= 0 || H <= 0 || L <= 0 || dk <= 0 || dv <= 0) return 0;
    const size_t nchunk = (L + BWD_CHUNK - 1) / BWD_CHUNK;
    return bwd_ws_bytes(B, H, L, dk, dv) + (size_t)B * H * nchunk * sizeof(int32_t);
}

extern "C" int vig_bigla_bwd_full(const void* q, const void* k, const void* v, const void* g_fwd, const void* g_bwd, const void* d_out,
                                  void* dq, void* dk_out, void* dv_out, void* dg_fwd, void* dg_bwd, int dg_fp32,
                                  int B, int H, int L, int dk, int dv, int dtype,
                                  const int64_t* strides_q, const int64_t* strides_k, const int64_t* strides_v,
                                  const int64_t* strides_gf, const int64_t* strides_gb, const int64_t* strides_do,
                                  float scale, float out_scale, float gate_logit_normalizer, float clamp_min, int dir_mask,
                                  void* workspace, size_t workspace_bytes, void* stream) {
    BwdParams p{};
    const int s = bwd_fill(p, q, k, v, g_fwd, g_bwd, d_out, dq, dk_out, dv_out, B, H, L, dk, dv, dtype, strides_q, strides_k, strides_v,
                           strides_gf, strides_gb, strides_do, scale, out_scale, dir_mask, workspace);
    if (s || B == 0 || L == 0) return s;
    if (((dir_mask & 1) && !dg_fwd) || ((dir_mask & 2) && !dg_bwd)) return VIG_ERR_NULL;
    if (!(gate_logit_normalizer >= 0.f)) return VIG_ERR_ARG;
    if (!workspace || workspace_bytes < vig_bigla_bwd_full_workspace_bytes(B, H, L, dk, dv)) return VIG_ERR_WORKSPACE;
    if (reinterpret_cast<uintptr_t>(workspace) & 15) return VIG_ERR_ALIGN;
    p.dgf = dg_fwd; p.dgb = dg_bwd; p.dg_f32 = dg_fp32 != 0;
    p.gate_norm = gate_logit_normalizer; p.clamp_min = clamp_min;
    // fp32 gate gradients of 16-bit inputs: token by token, whose sums are fp32 (1e-6 of them; the tensor-core form's operands
    // carry 16 bits there, 1e-5)
    if (!bigla_bwd_mma_supported(p) || (p.dg_f32 && dtype != VIG_DTYPE_F32)) return bwd_simt(p, 0, (cudaStream_t)stream);
    p.scanned = p.nchunk > bwd_fold(dtype);
    const int st = bigla_bwd_mma_launch(p, (cudaStream_t)stream);
    return st ? st : bwd_simt(p, 1, (cudaStream_t)stream);             // the chunks whose gates left the factorisation range
}
