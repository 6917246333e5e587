// Fused epilogue of the tensor-core kernels, by fragments: a warp reads its 32 accumulator rows 16 x 256 bits at a
// time (tcgen05.ld.16x256b), so that lane l holds columns 8q + 2 (l % 4), + 1 of rows l / 4 + 8k, the words of row
// l / 4 + 8k being v[k / 2][4q + 2 (k % 2)], + 1. Then
//   y = relu?(acc * scale + shift)
// with two-wide FMAs (fma.rn.f32x2: each lane rounds exactly as fmaf) and the ReLU folded into the BF16 conversion.
// What bounds it is the shared-memory pipe: with a row per lane (32x32b) each lane needs the scale and shift of all 64
// columns, 128 wavefronts per warp and 64 columns beside 32 for the staging; here of 16 columns, and column sums take
// 28 exchanges instead of a pass through the staging buffer. Batch 64: 56 x 56, 64 -> 256 1 x 1 forward 28.5 -> 23.8 us
// (19 at the memory's rate), the 224 x 224 stem's forward with statistics 71 -> 57.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tc_ptx.cuh"

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

// 32 rows x 64 columns of FP32 accumulators; ta: the warp's lane quarter and the first column.
__device__ __forceinline__ void frag_load(uint32_t ta, uint32_t (&v)[2][32]) {
    tmem_ld_16x256b_x8(ta, v[0]);
    tmem_ld_16x256b_x8(ta + (16u << 16), v[1]);
    tmem_ld_wait();
}

// v = v * sc + sh (sc, sh: the first column's, 8-byte aligned); without either v + 0, which is the same for 1 and 0.
__device__ __forceinline__ void frag_affine(uint32_t (&v)[2][32], bool affine, const float *__restrict__ sc,
                                            const float *__restrict__ sh) {
    const int fc = 2 * (threadIdx.x & 3);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        float2 s = make_float2(1.0f, 1.0f), t = make_float2(0.0f, 0.0f);
        if (affine) {
            s = *reinterpret_cast<const float2 *>(sc + 8 * q + fc);
            t = *reinterpret_cast<const float2 *>(sh + 8 * q + fc);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t *w = &v[k >> 1][4 * q + 2 * (k & 1)];
            const float2 z = __ffma2_rn(make_float2(__uint_as_float(w[0]), __uint_as_float(w[1])), s, t);
            w[0] = __float_as_uint(z.x);
            w[1] = __float_as_uint(z.y);
        }
    }
}

// Packed BF16 pairs, pk[4q + k]: row l / 4 + 8k, columns 8q + 2 (l % 4), + 1.
template <bool RELU>
__device__ __forceinline__ void frag_pack(const uint32_t (&v)[2][32], uint32_t (&pk)[32]) {
#pragma unroll
    for (int q = 0; q < 8; q++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t *w = &v[k >> 1][4 * q + 2 * (k & 1)];
            pk[4 * q + k] = cvt_bf16x2<RELU>(__uint_as_float(w[0]), __uint_as_float(w[1]));
        }
}
__device__ __forceinline__ void frag_pack(const uint32_t (&v)[2][32], bool relu, uint32_t (&pk)[32]) {
    if (relu) frag_pack<true>(v, pk);
    else frag_pack<false>(v, pk);
}

// This lane's word of packed pair (q, k) in a staging buffer of 32 rows x 128 bytes, 128-byte swizzle.
__device__ __forceinline__ uint8_t *frag_word(uint8_t *stg, int q, int k) {
    const int lane = threadIdx.x & 31, fr = lane >> 2;
    return stg + fr * 128 + k * 1024 + ((q ^ fr) << 4) + (lane & 3) * 4;
}
__device__ __forceinline__ void frag_stage(uint8_t *stg, const uint32_t (&pk)[32]) {
#pragma unroll
    for (int q = 0; q < 8; q++)
#pragma unroll
        for (int k = 0; k < 4; k++) *reinterpret_cast<uint32_t *>(frag_word(stg, q, k)) = pk[4 * q + k];
}

// The rows from `rows` on become zeros.
__device__ __forceinline__ void frag_clear_rows(uint32_t (&v)[2][32], int rows) {
    const int fr = (threadIdx.x & 31) >> 2;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (fr + 8 * k >= rows)
#pragma unroll
            for (int q = 0; q < 8; q++) v[k >> 1][4 * q + 2 * (k & 1)] = v[k >> 1][4 * q + 2 * (k & 1) + 1] = 0u;
}

// One exchange of the column sums: lanes with bit 4N set keep the upper half of s, the others the lower half.
template <int N>
__device__ __forceinline__ void frag_round(float2 (&s)[8]) {
    const bool up = (threadIdx.x & (4 * N)) != 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const float2 keep = up ? s[i + N] : s[i], send = up ? s[i] : s[i + N];
        s[i].x = keep.x + __shfl_xor_sync(0xFFFFFFFFu, send.x, 4 * N);
        s[i].y = keep.y + __shfl_xor_sync(0xFFFFFFFFu, send.y, 4 * N);
    }
}
// Sums (SQ: and sums of squares) of the 64 columns over the 32 rows; lane l gets columns 2l, 2l + 1. Four rows are
// added up by each lane, then eight lanes' sums in three exchanges of halves.
template <bool SQ>
__device__ __forceinline__ void frag_col_sums(const uint32_t (&v)[2][32], float2 &sum, float2 &sq) {
    float2 s[8], p[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        float2 z[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
            z[k] = make_float2(__uint_as_float(v[k >> 1][4 * q + 2 * (k & 1)]), __uint_as_float(v[k >> 1][4 * q + 2 * (k & 1) + 1]));
        s[q] = make_float2((z[0].x + z[1].x) + (z[2].x + z[3].x), (z[0].y + z[1].y) + (z[2].y + z[3].y));
        if (SQ) {
            p[q] = make_float2(z[0].x * z[0].x, z[0].y * z[0].y);
#pragma unroll
            for (int k = 1; k < 4; k++) p[q] = __ffma2_rn(z[k], z[k], p[q]);
        }
    }
    frag_round<4>(s);
    frag_round<2>(s);
    frag_round<1>(s);
    sum = s[0];
    if (SQ) {
        frag_round<4>(p);
        frag_round<2>(p);
        frag_round<1>(p);
        sq = p[0];
    }
}

}  // namespace tc
