// Parameter block and workspace layout shared by the two forms of the bi-GLA backward (tensor-core and SIMT).
#pragma once
#include "common.cuh"

namespace vig {

struct BwdParams {
    const void *q, *k, *v, *gf, *gb, *dout;
    void *out_dq, *out_dk, *out_dv;  // [B,H,L,d] contiguous, input dtype
    float *ef, *eb;                  // [B,H,L,dk] contiguous fp32: dq*q - dk*k per direction (or NULL)
    void *dgf, *dgb;                 // [B,H,L,dk] contiguous: finished gate gradients, input dtype or fp32 (or NULL)
    int dg_f32;
    int64_t sq[3], sk[3], sv[3], sgf[3], sgb[3], sdo[3];
    int B, H, L, dk, dv, dtype;
    float c;                         // scale * out_scale
    float gate_norm, clamp_min;      // as in the forward: > 0 = raw logits; NaN = no clamp
    int dir_mask;
    float *ws_S, *ws_Z, *ws_decay;   // [BH][nchunk][2][dk*dv] x2, [BH][nchunk][2][dk] (summed log-gates, log2 units)
    int32_t* flags;                  // [BH][nchunk]: not 0 = the chunk's gates left the factorisation range, take the exact form
    int nchunk;
    int scanned;                     // 1: ws_S, ws_Z hold the states entering each chunk; 0: what each chunk contributes, summed by who needs them
};

constexpr int BWD_CHUNK = 64;
// Chunks of a sequence up to which the contributions are summed where they are used instead of by a launch over chunks.  With n chunks that reads
// n - 1 states more a chunk and direction; the launch reads and writes two each.  Forward + backward in us, summed / launched: 2 chunks 128x3x128 32/64
// bf16 92 / 105; 4 chunks 128x3x196 32/64 179 / 189, 128x6x196 64/64 529 / 590, fp32 128x3x196 243 / 243, 2x3x196 84 / 88; 6 chunks 64x3x384 64/64 227 / 236; 8 chunks
// 64x3x512 64/64 304 / 308, 64x6x512 32/64 371 / 374; fp32 64x3x320 (5) 323 / 322, 64x3x512 449 / 444.
inline int bwd_fold(int dtype) { return dtype == VIG_DTYPE_F32 ? 4 : 6; }

inline size_t bwd_state_floats(int B, int H, int nchunk, int dk, int dv) { return (size_t)B * H * nchunk * 2 * dk * dv; }

// tensor-core form: whether it takes this call, and the launch (states, scan, gradients; flagged chunks are left to the caller)
bool bigla_bwd_mma_supported(const BwdParams& p);
int bigla_bwd_mma_launch(const BwdParams& p, cudaStream_t stream);
int bigla_bwd_scan_launch(const BwdParams& p, cudaStream_t stream);

}  // namespace vig
