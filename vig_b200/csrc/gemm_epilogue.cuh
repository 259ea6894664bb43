// What the epilogues of the tcgen05 GEMMs share: SwiGLU of accumulator columns, and a warp's way out through a box of shared memory.
#pragma once
#include "tc_common.cuh"

namespace vig {
namespace tc {

constexpr int OUT_BOX_BYTES = 32 * 32 * 2;     // one epilogue warp's [32 rows x 32 columns] box

// silu(g) * y for 32 features of a row, packed to 16-bit pairs.  The arithmetic runs two-wide (mul / fma .f32x2 on register
// pairs: the epilogue warps are bound by instruction issue); each lane of those is the scalar IEEE operation.
template <typename T>
__device__ __forceinline__ void swiglu_pack(const float* g, const float* y, uint32_t* pk) {
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
        unsigned long long g2, y2, h2, half2, s2, r2;
        asm("mov.b64 %0, {%1, %2};" : "=l"(g2) : "f"(g[e]), "f"(g[e + 1]));
        asm("mov.b64 %0, {%1, %2};" : "=l"(y2) : "f"(y[e]), "f"(y[e + 1]));
        asm("mov.b64 %0, {%1, %1};" : "=l"(half2) : "f"(0.5f));
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(h2) : "l"(g2), "l"(half2));
        float h0, h1, t0, t1;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(h0), "=f"(h1) : "l"(h2));
        asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(h0));
        asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(h1));
        asm("mov.b64 %0, {%1, %2};" : "=l"(s2) : "f"(t0), "f"(t1));
        asm("fma.rn.f32x2 %0, %1, %2, %2;" : "=l"(s2) : "l"(s2), "l"(half2));   // sigmoid = 0.5 tanh(g / 2) + 0.5
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r2) : "l"(g2), "l"(y2));
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r2) : "l"(r2), "l"(s2));
        float r0, r1;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(r0), "=f"(r1) : "l"(r2));
        pk[e / 2] = Pack2<T>::pack(r0, r1);
    }
}

// A warp's [32 rows x 32 columns] piece goes out through its 2 KB box of shared memory as one TMA store.  A row is 64 bytes, its
// 16-byte pieces swizzled (64-byte swizzle) so that eight lanes write all banks; unswizzled they met on a quarter of them, and the
// operands of the MMAs come out of the same shared memory.
__device__ __forceinline__ void send_box(uint8_t* box, const uint32_t* pk, const CUtensorMap* map, int col, int row, bool in_range, int lane) {
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the warp's earlier store has read the box
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; ++j)
        *reinterpret_cast<uint4*>(box + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
        if (in_range) tma_store_2d(map, col, row, smem_u32(box));      // rows past M are clipped by the tensor map
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
}

// [rows, cols] output with leading dimension ld: boxes of 32 rows x 32 columns as send_box writes them
inline bool make_out_map(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int64_t ld, int dtype) {
    MapKey key{};
    key.base = base; key.rank = 2; key.dtype = dtype; key.swizzle = 2;
    key.dims[0] = (uint64_t)cols; key.dims[1] = (uint64_t)rows;
    key.strides[0] = (uint64_t)ld * 2;
    key.box[0] = 32; key.box[1] = 32;
    return encode_cached(m, key);
}

}  // namespace tc
}  // namespace vig
