// Fused epilogue arithmetic of the tensor-core kernels: one thread turns 64
// FP32 accumulators of its output row into 32 packed BF16 pairs,
//   y = relu?(acc * scale + shift),
// with two-wide FMAs (fma.rn.f32x2: each lane rounds exactly as fmaf) and the
// ReLU folded into the BF16 conversion (cvt.rn.relu.bf16x2.f32).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tc {

template <bool RELU>
__device__ __forceinline__ uint32_t cvt_bf16x2(float lo, float hi) {
    uint32_t d;
    if (RELU)
        asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    else
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// v0: columns 0-31, v1: columns 32-63 (tcgen05.ld 32x32b.x32 results); sc/sh:
// the 64 columns' scale and shift, 16-byte aligned (shared memory).
template <bool RELU>
__device__ __forceinline__ void epi_bf16_64(const uint32_t (&v0)[32], const uint32_t (&v1)[32],
                                            const float *__restrict__ sc, const float *__restrict__ sh,
                                            uint32_t (&pk)[32]) {
    const float4 *s4 = reinterpret_cast<const float4 *>(sc);
    const float4 *t4 = reinterpret_cast<const float4 *>(sh);
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const float4 s = s4[q], t = t4[q];
        const int j = 4 * q;
        float2 a = make_float2(__uint_as_float(j < 32 ? v0[j] : v1[j - 32]),
                               __uint_as_float(j < 32 ? v0[j + 1] : v1[j - 31]));
        float2 b = make_float2(__uint_as_float(j < 32 ? v0[j + 2] : v1[j - 30]),
                               __uint_as_float(j < 32 ? v0[j + 3] : v1[j - 29]));
        a = __ffma2_rn(a, make_float2(s.x, s.y), make_float2(t.x, t.y));
        b = __ffma2_rn(b, make_float2(s.z, s.w), make_float2(t.z, t.w));
        pk[2 * q] = cvt_bf16x2<RELU>(a.x, a.y);
        pk[2 * q + 1] = cvt_bf16x2<RELU>(b.x, b.y);
    }
}

// Column sums (SQ: and sums of squares) of z = v * sc + sh (AFFINE; else v) over a warp's 32 rows and 32 columns:
// lane l returns them for columns 2 (l % 16), + 1. The values pass through the warp's 4 KB staging buffer, rows in
// (rows that do not count, `in` false, as zeros), columns out: each lane adds up two columns of the rows of its
// parity l / 16, in two running sums. Exchanged by shuffles the same sums were about a thousand instructions of
// straight-line code per 64 columns and bound by instruction fetches: 56 x 56, 64 -> 256 forward with statistics
// 111 us, 27 this way; 224 x 224 stem forward with statistics 93 us, STEMNOW this way and with eight epilogue warps.
template <bool AFFINE, bool SQ>
__device__ __forceinline__ void staged_col_sums32(uint8_t *stg, const uint32_t (&v)[32], const float *sc, const float *sh,
                                                  bool in, float2 &sum, float2 &sq) {
    const int lane = threadIdx.x & 31, l16 = lane & 15;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        float z[4];
#pragma unroll
        for (int e = 0; e < 4; e++) z[e] = __uint_as_float(v[4 * q + e]);
        if (AFFINE) {
            const float4 a = *reinterpret_cast<const float4 *>(sc + 4 * q);
            const float4 b = *reinterpret_cast<const float4 *>(sh + 4 * q);
            z[0] = fmaf(z[0], a.x, b.x);
            z[1] = fmaf(z[1], a.y, b.y);
            z[2] = fmaf(z[2], a.z, b.z);
            z[3] = fmaf(z[3], a.w, b.w);
        }
        *reinterpret_cast<float4 *>(stg + lane * 128 + ((q ^ (lane & 7)) << 4)) =
            in ? make_float4(z[0], z[1], z[2], z[3]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncwarp();
    float2 s2[2] = {}, q2[2] = {};
#pragma unroll 2
    for (int r = lane >> 4; r < 32; r += 4)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int rr = r + 2 * e;
            const float2 z = *reinterpret_cast<const float2 *>(stg + rr * 128 + (((l16 >> 1) ^ (rr & 7)) << 4) + (l16 & 1) * 8);
            s2[e].x += z.x;
            s2[e].y += z.y;
            if (SQ) q2[e] = __ffma2_rn(z, z, q2[e]);
        }
    sum = make_float2(s2[0].x + s2[1].x, s2[0].y + s2[1].y);
    sum.x += __shfl_xor_sync(0xFFFFFFFFu, sum.x, 16);
    sum.y += __shfl_xor_sync(0xFFFFFFFFu, sum.y, 16);
    if (SQ) {
        sq = make_float2(q2[0].x + q2[1].x, q2[0].y + q2[1].y);
        sq.x += __shfl_xor_sync(0xFFFFFFFFu, sq.x, 16);
        sq.y += __shfl_xor_sync(0xFFFFFFFFu, sq.y, 16);
    }
    __syncwarp();
}

}  // namespace tc
