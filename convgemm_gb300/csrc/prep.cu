// Preparation kernels of the tensor-core forms: weight packing into the
// K-major operand the tcgen05 kernels load with TMA, the FP64 batch-norm fold,
// activation casts, and the fixed-order reduction of weight-gradient splits.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "cg_common.cuh"
#include "prep.h"
#include "tc_ptx.cuh"

#include <algorithm>

namespace {

using bf16 = __nv_bfloat16;

// Weight element (ci, kx, ky, co) of the reference layouts:
//   NHWC API: [c][kh][kw][kn]  (src/convGemm.c:66, ld = kn)
//   NCHW API: [kn][c][kh][kw]  (src/convGemm.c:117, ld = K)
__device__ __forceinline__ float wref(const float *w, int nchw, int C, int kh, int kw, int kn, int ci, int kx, int ky,
                                      int co) {
    const size_t k = ((size_t) ci * kh + kx) * kw + ky;
    return nchw ? w[(size_t) co * ((size_t) C * kh * kw) + k] : w[k * kn + co];
}

// out[co][k], k = (kx*kw + ky)*Cp + ci, zero for padded ci and k.  One 32x32 tile of
// (ci, co) at one tap per block: reads along co (contiguous in the NHWC-API layout),
// writes along ci (contiguous in the packed row) through shared memory.
__global__ void pack_fwd_tiled_kernel(const float *__restrict__ w, int C, int khw, int kn, int Cp, int Kpad,
                                      bf16 *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    __shared__ float tile[32][33];
    const int tap = blockIdx.z, ci0 = blockIdx.x * 32, co0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int i = ty; i < 32; i += 8) {
        const int ci = ci0 + i, co = co0 + tx;
        tile[i][tx] = (ci < C && co < kn) ? w[((size_t) ci * khw + tap) * kn + co] : 0.0f;
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8) {
        const int co = co0 + j, ci = ci0 + tx;
        if (co < kn && ci < Cp) out[(size_t) co * Kpad + (size_t) tap * Cp + ci] = __float2bfloat16_rn(tile[tx][j]);
    }
}

// zero of the K padding columns [khw*Cp, Kpad) of every row
__global__ void pack_fwd_tail_kernel(int kn, int Kbeg, int Kpad, bf16 *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const int width = Kpad - Kbeg;
    const long long total = (long long) kn * width;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x)
        out[(i / width) * Kpad + Kbeg + i % width] = __float2bfloat16_rn(0.0f);
}

__global__ void pack_fwd_kernel(const float *__restrict__ w, int nchw, int C, int kh, int kw, int kn, int Cp,
                                int Kpad, bf16 *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const long long total = (long long) kn * Kpad;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x) {
        const int co = (int) (i / Kpad), k = (int) (i % Kpad);
        const int tap = k / Cp, ci = k % Cp;
        float v = 0.0f;
        if (tap < kh * kw && ci < C) v = wref(w, nchw, C, kh, kw, kn, ci, tap / kw, tap % kw, co);
        out[i] = __float2bfloat16_rn(v);
    }
}

// Input-gradient operand: out[ci][kbeg_c + t*knp + co] = W(ci, kx_t, ky_t, co) for each class c.
__global__ void pack_dgrad_kernel(const float *__restrict__ w, int nchw, int C, int kh, int kw, int kn, int knp,
                                  const PackDgradInfo info, bf16 *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const long long total = (long long) C * info.Ktot;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x) {
        const int ci = (int) (i / info.Ktot), col = (int) (i % info.Ktot);
        int c = 0;
        while (c + 1 < info.ncls && col >= info.kbeg[c + 1]) c++;
        const int k = col - info.kbeg[c];
        const int t = k / knp, co = k % knp;
        float v = 0.0f;
        if (t < info.ntaps[c] && co < kn) v = wref(w, nchw, C, kh, kw, kn, ci, info.kx[info.tap0[c] + t], info.ky[info.tap0[c] + t], co);
        out[i] = __float2bfloat16_rn(v);
    }
}

// scale = gamma*inv_std, shift = beta + (bias - mean)*scale, in double (the one place
// besides the oracle where FP64 runs on the GPU).
__global__ void fold_kernel(int kn, const float *bias, const float *mean, const float *inv_std, const float *gamma,
                            const float *beta, float *scale, float *shift) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= kn) return;
    double s = 1.0, t = bias ? (double) bias[n] : 0.0;
    if (mean) {
        s = (double) gamma[n] * (double) inv_std[n];
        t = (double) beta[n] + (t - (double) mean[n]) * s;
    }
    scale[n] = (float) s;
    shift[n] = (float) t;
}

// FP32 NHWC or NCHW [B][C][H][W] -> BF16 NHWC [B][H][W][Cp] (padding channels zero).
__global__ void to_bf16_nhwc_kernel(const float *__restrict__ in, int nchw, int B, int C, int H, int W, int Cp,
                                    bf16 *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const long long total = (long long) B * H * W * Cp;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x) {
        const int c = (int) (i % Cp);
        const long long pix = i / Cp;
        float v = 0.0f;
        if (c < C) {
            if (nchw) {
                const long long hw = (long long) H * W;
                const long long b = pix / hw, q = pix % hw;
                v = in[(b * C + c) * hw + q];
            } else {
                v = in[pix * C + c];
            }
        }
        out[i] = __float2bfloat16_rn(v);
    }
}

__device__ __forceinline__ uint32_t bf16x2_of(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint4 bf16x8_of(const float (&v)[8]) {
    return make_uint4(bf16x2_of(v[0], v[1]), bf16x2_of(v[2], v[3]), bf16x2_of(v[4], v[5]), bf16x2_of(v[6], v[7]));
}

// The same cast for 16-byte aligned outputs. All three forms are HBM-bound and store whole
// 16-byte groups of eight channels; the element form above divides per element, reads NCHW planes with
// one value per lane and line, and ran at 1.0 TB/s (64 x 3 x 224 x 224: 87 us) to 1.5 TB/s.
//
// NCHW with c <= 8: a thread reads its pixels from every plane (neighbouring lanes, neighbouring pixels), four
// pixels at a time, an image per blockIdx.y: 64 x 3 x 224 x 224 in 14.9 us (18.7 with one pixel at a time, found by
// 64-bit division; 13.3 at the rate of a copy).
__global__ void __launch_bounds__(256) nchw_few_to_bf16_kernel(const float *__restrict__ in, int C, int HW, uint4 *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const float *src = in + (size_t) blockIdx.y * C * HW;
    uint4 *dst = out + (size_t) blockIdx.y * HW;
    const int p0 = blockIdx.x * 1024 + threadIdx.x;
    float v[4][8];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int c = 0; c < 8; c++)
            v[k][c] = c < C && p0 + 256 * k < HW ? __ldg(src + (size_t) c * HW + p0 + 256 * k) : 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (p0 + 256 * k < HW) dst[p0 + 256 * k] = bf16x8_of(v[k]);
}

// NCHW: 64 channels x 64 pixels per block through shared memory; planes read along the pixels (16-byte
// vectors when HW % 4 == 0 and the input is aligned), pixels written along the channels.
__global__ void __launch_bounds__(256) nchw_tiled_to_bf16_kernel(const float *__restrict__ in, int C, int HW, int Cp, int vec,
                                                                 uint4 *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    __shared__ float t[64][65];
    const int q0 = blockIdx.x * 64, c0 = blockIdx.y * 64, tid = threadIdx.x;
    const float *src = in + (size_t) blockIdx.z * C * HW;
    if (vec) {
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int c = c0 + tid / 16 + 16 * k, q = q0 + 4 * (tid % 16);
            v[k] = c < C && q < HW ? __ldg(reinterpret_cast<const float4 *>(src + (size_t) c * HW + q))
                                   : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float *o = &t[tid / 16 + 16 * k][4 * (tid % 16)];
            o[0] = v[k].x;
            o[1] = v[k].y;
            o[2] = v[k].z;
            o[3] = v[k].w;
        }
    } else {
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int c = c0 + tid / 64 + 4 * k, q = q0 + tid % 64;
            v[k] = c < C && q < HW ? __ldg(src + (size_t) c * HW + q) : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < 16; k++) t[tid / 64 + 4 * k][tid % 64] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int q = tid / 8 + 32 * k, g = tid % 8;   // pixel, group of eight channels
        if (q0 + q >= HW || c0 + 8 * g >= Cp) continue;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = t[8 * g + j][q];
        out[(((size_t) blockIdx.z * HW + q0 + q) * Cp + c0) / 8 + g] = bf16x8_of(v);
    }
}

// NHWC: eight channels of a pixel per thread.
__global__ void __launch_bounds__(256) nhwc_to_bf16_kernel(const float *__restrict__ in, int C, int Cp, long long n8, int vec,
                                                           uint4 *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const int k8 = Cp / 8;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n8; i += gridDim.x * 256LL) {
        float v[8];
        if (vec) {   // C % 8 == 0, 16-byte aligned
            const float4 a = __ldg(reinterpret_cast<const float4 *>(in) + 2 * i), b = __ldg(reinterpret_cast<const float4 *>(in) + 2 * i + 1);
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
            const long long pix = i / k8;
            const int c = (int) (i - pix * k8) * 8;
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = c + j < C ? __ldg(in + pix * C + c + j) : 0.0f;
        }
        out[i] = bf16x8_of(v);
    }
}

// ------------------------------------------------------ FP8 and 3xBF16 forms
constexpr float E4M3_MAX = 448.0f;

__device__ __forceinline__ uint8_t to_e4m3(float v) {
    return (uint8_t) __nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}

// Eight consecutive values from element 8 * i, both input types; 16-byte aligned.
template <bool BF>
__device__ __forceinline__ void load8(const void *in, long long i, float (&v)[8]) {
    if (BF) {
        const uint4 u = __ldg(reinterpret_cast<const uint4 *>(in) + i);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[2 * j] = __uint_as_float(w[j] << 16);
            v[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
        }
    } else {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(in) + 2 * i), b = __ldg(reinterpret_cast<const float4 *>(in) + 2 * i + 1);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    }
}
template <bool BF>
__device__ __forceinline__ float load1(const void *in, long long i) {
    return BF ? __bfloat162float(((const bf16 *) in)[i]) : ((const float *) in)[i];
}

// amax (as the bit pattern of a non-negative float, so atomicMax on unsigned orders it). One atomic
// per block: one per warp, 39k of them on one word, took longer than the reads (25 M values: 28 us).
// n8: groups of eight read as vectors (0 when `in` is not 16-byte aligned).
template <bool BF>
__global__ void __launch_bounds__(256) amax_kernel(const void *__restrict__ in, long long n8, long long n, unsigned *amax_bits) {
    tc::pdl_wait();
    tc::pdl_trigger();
    __shared__ float red[8];
    const long long step = gridDim.x * 256LL, i0 = blockIdx.x * 256LL + threadIdx.x;
    float m = 0.0f;
    long long i = i0;
    for (; i + 3 * step < n8; i += 4 * step) {
        float v[4][8];
#pragma unroll
        for (int k = 0; k < 4; k++) load8<BF>(in, i + k * step, v[k]);
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int j = 0; j < 8; j++) m = fmaxf(m, fabsf(v[k][j]));
    }
    for (; i < n8; i += step) {
        float v[8];
        load8<BF>(in, i, v);
#pragma unroll
        for (int j = 0; j < 8; j++) m = fmaxf(m, fabsf(v[j]));
    }
    for (long long k = 8 * n8 + i0; k < n; k += step) m = fmaxf(m, fabsf(load1<BF>(in, k)));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 1; k < 8; k++) m = fmaxf(m, red[k]);
        atomicMax(amax_bits, __float_as_uint(m));
    }
}

// per-tensor scale = amax / 448 (1 for an all-zero tensor); x_q = e4m3(x / scale). Eight values per
// thread and 8-byte stores where input (16) and output (8) are aligned (n8 as above). HBM-bound: four loads in
// flight per thread and one wave of four blocks per SM, 12.8 M values in 5.7 us (8.5 with one load and four waves;
// 38 MB at the rate of a copy: 5.7).
template <bool BF>
__global__ void __launch_bounds__(256) quant_e4m3_kernel(const void *__restrict__ in, long long n8, long long n,
                                                         const unsigned *amax_bits, uint8_t *__restrict__ out, float *scale_out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const float amax = __uint_as_float(*amax_bits);
    const float sc = amax > 0.0f ? amax / E4M3_MAX : 1.0f;
    const float inv = 1.0f / sc;
    const long long step = gridDim.x * 256LL, i0 = blockIdx.x * 256LL + threadIdx.x;
    if (i0 == 0) *scale_out = sc;
    for (long long i = i0; i < n8; i += 4 * step) {   // four loads in flight
        float v[4][8];
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (i + k * step < n8) load8<BF>(in, i + k * step, v[k]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i + k * step >= n8) break;
            uint32_t q[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                q[j] = __nv_cvt_float2_to_fp8x2(make_float2(v[k][2 * j] * inv, v[k][2 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
            reinterpret_cast<uint2 *>(out)[i + k * step] = make_uint2(q[0] | q[1] << 16, q[2] | q[3] << 16);
        }
    }
    for (long long i = 8 * n8 + i0; i < n; i += step) out[i] = to_e4m3(load1<BF>(in, i) * inv);
}

// per-output-channel weight scale (NHWC-API weights [K][kn]: threads along co, loop over K)
__global__ void wscale_kernel(const float *__restrict__ w, int nchw, int K, int kn, float *wscale) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const int co = blockIdx.x * blockDim.x + threadIdx.x;
    if (co >= kn) return;
    float m = 0.0f;
    for (int k = 0; k < K; k++) m = fmaxf(m, fabsf(nchw ? w[(size_t) co * K + k] : w[(size_t) k * kn + co]));
    wscale[co] = m > 0.0f ? m / E4M3_MAX : 1.0f;
}

// E4M3 operand [co][tap*Cp + ci] = w / wscale[co]
__global__ void pack_fp8_kernel(const float *__restrict__ w, int nchw, int C, int kh, int kw, int kn, int Cp, int Kpad,
                                const float *__restrict__ wscale, uint8_t *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const long long total = (long long) kn * Kpad;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x) {
        const int co = (int) (i / Kpad), k = (int) (i % Kpad);
        const int tap = k / Cp, ci = k % Cp;
        float v = 0.0f;
        if (tap < kh * kw && ci < C) v = wref(w, nchw, C, kh, kw, kn, ci, tap / kw, tap % kw, co) / wscale[co];
        out[i] = to_e4m3(v);
    }
}

// scale' = scale * wscale * xscale (the two quantisation scales folded into the epilogue)
__global__ void fp8_scales_kernel(int kn, const float *scale, const float *shift, const float *wscale,
                                  const float *xscale, float *out_scale, float *out_shift) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= kn) return;
    out_scale[n] = (scale ? scale[n] : 1.0f) * wscale[n] * xscale[0];
    out_shift[n] = shift ? shift[n] : 0.0f;
}

// x = hi + lo with hi = bf16(x), lo = bf16(x - hi); n8: groups of eight as 16-byte vectors (0 when a
// tensor is not 16-byte aligned).
__global__ void __launch_bounds__(256) split_kernel(const float *__restrict__ in, long long n8, long long n, bf16 *__restrict__ hi,
                                                    bf16 *__restrict__ lo) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const long long step = gridDim.x * 256LL, i0 = blockIdx.x * 256LL + threadIdx.x;
    for (long long i = i0; i < n8; i += step) {
        float v[8], r[8];
        load8<false>(in, i, v);
#pragma unroll
        for (int j = 0; j < 8; j++) r[j] = v[j] - __bfloat162float(__float2bfloat16_rn(v[j]));
        reinterpret_cast<uint4 *>(hi)[i] = bf16x8_of(v);
        reinterpret_cast<uint4 *>(lo)[i] = bf16x8_of(r);
    }
    for (long long i = 8 * n8 + i0; i < n; i += step) {
        const float v = in[i];
        const bf16 h = __float2bfloat16_rn(v);
        hi[i] = h;
        lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
    }
}

__global__ void pack_split_kernel(const float *__restrict__ w, int nchw, int C, int kh, int kw, int kn, int Cp, int Kpad,
                                  bf16 *__restrict__ hi, bf16 *__restrict__ lo) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const long long total = (long long) kn * Kpad;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x) {
        const int co = (int) (i / Kpad), k = (int) (i % Kpad);
        const int tap = k / Cp, ci = k % Cp;
        float v = 0.0f;
        if (tap < kh * kw && ci < C) v = wref(w, nchw, C, kh, kw, kn, ci, tap / kw, tap % kw, co);
        const bf16 h = __float2bfloat16_rn(v);
        hi[i] = h;
        lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
    }
}

// n values by 256 threads, B loads in flight per thread.
template <int B, class T, class Load, class Store>
__device__ __forceinline__ void batched(int n, Load load, Store store) {
    for (int i0 = threadIdx.x; i0 < n; i0 += 256 * B) {
        T v[B];
#pragma unroll
        for (int j = 0; j < B; j++)
            if (i0 + 256 * j < n) v[j] = load(i0 + 256 * j);
#pragma unroll
        for (int j = 0; j < B; j++)
            if (i0 + 256 * j < n) store(i0 + 256 * j, v[j]);
    }
}

// Grouped preparation: every block finds its job by binary search over the jobs'
// first blocks and runs that job's body for its block (256 threads).
// What bounds it is the chain of latencies within a block, and how many blocks share an SM: the jobs' first blocks (b0,
// njobs ints) are staged in shared memory, so the search costs one global round trip, then the job itself (read field by
// field from memory, each access a round trip again behind the stores), and the weights are read several at a time, as far
// as six blocks per SM leave registers (40: with eight loads in flight and 64 registers, four blocks, 262 x 688 x 7 x 7 NHWC
// took 118 us a round of six, 94 so). Both operands of 512 x 512 x 3 x 3 (NCHW): 47 us value by value, 11.5 staged.
__global__ void __launch_bounds__(256, 6) prep_group_kernel(const PrepJob *__restrict__ jobs, const int *__restrict__ b0,
                                                         int njobs) {
    __shared__ float tile[64][65];
    extern __shared__ int s_b0[];
    tc::pdl_wait();
    tc::pdl_trigger();
    for (int i = threadIdx.x; i < njobs; i += blockDim.x) s_b0[i] = __ldg(b0 + i);
    __syncthreads();
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_b0[mid] <= (int) blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const int t = threadIdx.x;
    __shared__ alignas(16) uint32_t job[sizeof(PrepJob) / 4];
    __shared__ int taps[TC_MAXTAPS];   // the class's filter taps (input-gradient jobs)
    static_assert(sizeof(PrepJob) % 4 == 0, "job copied by words");
    for (int i = t; i < (int) (sizeof(PrepJob) / 4); i += 256) job[i] = __ldg(reinterpret_cast<const uint32_t *>(jobs + lo) + i);
    __syncthreads();
    const PrepJob &J = *reinterpret_cast<const PrepJob *>(job);
    const int lb = blockIdx.x - J.block0;
    switch (J.type) {
        case PREP_FOLD: {
            const int n = lb * 256 + t;
            if (n >= J.kn) return;
            double sc = 1.0, sh = J.bias ? (double) J.bias[n] : 0.0;
            if (J.mean) {
                sc = (double) J.gamma[n] * (double) J.inv_std[n];
                sh = (double) J.beta[n] + (sh - (double) J.mean[n]) * sc;
            }
            J.scale[n] = (float) sc;
            J.shift[n] = (float) sh;
            return;
        }
        case PREP_FWD_TILED: {
            // NHWC-API weights [ci][tap][co] -> out[co][tap*Cp + ci]: one block per (tap, 64 ci x 64 co
            // tile); four independent 16-byte loads per thread along co, a padded shared-memory
            // transpose, 8-byte stores of four BF16 along ci
            const int nci = (J.Cp + 63) / 64, nco = (J.kn + 63) / 64, khw = J.kh * J.kw;
            const int tap = lb / (nci * nco), rem = lb % (nci * nco);
            const int ci0 = (rem % nci) * 64, co0 = (rem / nci) * 64;
            const int cq = (t & 15) * 4, r0 = t >> 4;   // 4 co per thread; rows r0 + 16 i
            const bool vec_in = ((J.kn & 3) == 0) && (((uintptr_t) J.w & 15) == 0);
            const bool vec_out = ((J.Kpad & 3) == 0) && ((J.Cp & 3) == 0) && (((uintptr_t) J.out & 7) == 0);
            float4 v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int ci = ci0 + r0 + 16 * i, co = co0 + cq;
                const float *src = J.w + ((size_t) ci * khw + tap) * J.kn + co;
                if (ci < J.C && co + 4 <= J.kn && vec_in) {
                    v[i] = __ldg(reinterpret_cast<const float4 *>(src));
                } else {
                    float e[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) e[q] = (ci < J.C && co + q < J.kn) ? __ldg(src + q) : 0.0f;
                    v[i] = make_float4(e[0], e[1], e[2], e[3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float *d = &tile[r0 + 16 * i][cq];
                d[0] = v[i].x;
                d[1] = v[i].y;
                d[2] = v[i].z;
                d[3] = v[i].w;
            }
            __syncthreads();
            bf16 *out = (bf16 *) J.out;
            const int cw = (t & 15) * 4, o0 = t >> 4;   // 4 ci per thread; co rows o0 + 16 j
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int co = co0 + o0 + 16 * j, ci = ci0 + cw;
                if (co >= J.kn || ci >= J.Cp) continue;
                bf16 *dst = out + (size_t) co * J.Kpad + (size_t) tap * J.Cp + ci;
                const int cc = o0 + 16 * j;
                if (ci + 4 <= J.Cp && vec_out) {
                    __nv_bfloat162 lo = __floats2bfloat162_rn(tile[cw][cc], tile[cw + 1][cc]);
                    __nv_bfloat162 hi = __floats2bfloat162_rn(tile[cw + 2][cc], tile[cw + 3][cc]);
                    uint2 u;
                    u.x = *reinterpret_cast<uint32_t *>(&lo);
                    u.y = *reinterpret_cast<uint32_t *>(&hi);
                    *reinterpret_cast<uint2 *>(dst) = u;
                } else {
                    for (int q = 0; q < 4 && ci + q < J.Cp; q++) dst[q] = __float2bfloat16_rn(tile[cw + q][cc]);
                }
            }
            return;
        }
        case PREP_FWD_NCHW: {
            // NCHW-API weights [co][ci][tap] -> out[co][tap*Cp + ci]: block = (row co, a chunk of its
            // input channels), the chunk read contiguously into shared memory and written tap by tap
            // (gathering single values from a stride of taps: 60 us for 512 x 512 x 3 x 3 with the
            // input-gradient operand, 8 us staged)
            const int khw = J.kh * J.kw, CH = prep_nchw_channels(khw), Cp = J.Cp, Kpad = J.Kpad, nch = (Cp + CH - 1) / CH;
            const int co = lb / nch, ci0 = (lb % nch) * CH, n = min(CH, Cp - ci0);
            float *buf = &tile[0][0];
            const float *src = J.w + ((size_t) co * J.C + ci0) * khw;
            const int have = max(0, min(n, J.C - ci0)) * khw;
            if (khw == 1) {   // one tap: the row as it is
                bf16 *row = (bf16 *) J.out + (size_t) co * Kpad + ci0;
                const int end = ci0 + n == Cp ? Kpad - ci0 : n;   // with the K padding after the last chunk
                batched<2, float>(end, [&](int i) { return i < have ? __ldg(src + i) : 0.0f; }, [&](int i, float v) { row[i] = __float2bfloat16_rn(v); });
                return;
            }
            if (((uintptr_t) src & 15) == 0 && (have & 3) == 0 && (n * khw & 3) == 0)
                batched<2, float4>(
                    n * khw >> 2,
                    [&](int i) { return 4 * i < have ? __ldg(reinterpret_cast<const float4 *>(src) + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f); },
                    [&](int i, float4 v) {
                        buf[4 * i] = v.x;
                        buf[4 * i + 1] = v.y;
                        buf[4 * i + 2] = v.z;
                        buf[4 * i + 3] = v.w;
                    });
            else
                batched<4, float>(n * khw, [&](int i) { return i < have ? __ldg(src + i) : 0.0f; }, [&](int i, float v) { buf[i] = v; });
            __syncthreads();
            // a warp per tap, two channels per store where the chunk's ends are even
            bf16 *row = (bf16 *) J.out + (size_t) co * Kpad;
            const int lane = t & 31;
            if ((n & 1) == 0 && (ci0 & 1) == 0 && ((uintptr_t) row & 3) == 0) {
                for (int tap = t >> 5; tap < khw; tap += 8)
#pragma unroll 4
                    for (int ci = 2 * lane; ci < n; ci += 64)
                        *reinterpret_cast<__nv_bfloat162 *>(row + tap * Cp + ci0 + ci) =
                            __floats2bfloat162_rn(buf[ci * khw + tap], buf[(ci + 1) * khw + tap]);
            } else {
                for (int tap = t >> 5; tap < khw; tap += 8)
                    for (int ci = lane; ci < n; ci += 32) row[tap * Cp + ci0 + ci] = __float2bfloat16_rn(buf[ci * khw + tap]);
            }
            if (ci0 == 0)
                for (int k = khw * Cp + t; k < Kpad; k += 256) row[k] = __float2bfloat16_rn(0.0f);
            return;
        }
        case PREP_FWD_TAIL: {
            const int kbeg = J.kh * J.kw * J.Cp, width = J.Kpad - kbeg;
            const int i = lb * 256 + t;
            if (i >= J.kn * width) return;
            const int co = i / width;
            ((bf16 *) J.out)[(size_t) co * J.Kpad + kbeg + (i - co * width)] = __float2bfloat16_rn(0.0f);
            return;
        }
        case PREP_DGRAD_NCHW: {
            // NCHW-API weights [co][ci][tap], one class: block = (4 input channels, a run of output channels): the run's
            // 4 x taps values, contiguous per output channel, staged through shared memory (odd pitch) and written along co
            const int khw = J.kh * J.kw, Ktot = J.info.Ktot, knp = J.knp, C = J.C;
            const int run = prep_nchw_run(khw), nrun = (knp + run - 1) / run;
            const int ci0 = lb / nrun * 4, co0 = lb % nrun * run;
            const int nci = min(4, C - ci0), w4 = nci * khw, pitch = (4 * khw) | 1, nco = min(run, knp - co0);
            float *buf = &tile[0][0];
            if (t < khw) taps[t] = J.info.kx[t] * J.kw + J.info.ky[t];
            const float *src = J.w + ((size_t) co0 * C + ci0) * khw;
            const int have = J.kn - co0;
            const int lane = t & 31;
            if ((w4 & 3) == 0 && (C * khw & 3) == 0 && ((uintptr_t) src & 15) == 0) {
                // 16 lanes per output channel
#pragma unroll 2
                for (int co = t >> 4; co < nco; co += 16)
                    for (int k = 4 * (t & 15); k < w4; k += 64) {
                        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        if (co < have) v = __ldg(reinterpret_cast<const float4 *>(src + (size_t) co * C * khw + k));
                        float *d = buf + co * pitch + k;
                        d[0] = v.x;
                        d[1] = v.y;
                        d[2] = v.z;
                        d[3] = v.w;
                    }
            } else {
                // several output channels' values at a time
                const uint32_t inv = 0xFFFFFFFFu / (uint32_t) w4 + 1;   // i / w4 (w4 > 1) by its high product: i * w4 is far below 2^32
                batched<4, float>(
                    nco * w4,
                    [&](int i) {
                        const int co = (int) __umulhi((uint32_t) i, inv);
                        return co < have ? __ldg(src + (size_t) co * C * khw + (i - co * w4)) : 0.0f;
                    },
                    [&](int i, float v) {
                        const int co = (int) __umulhi((uint32_t) i, inv);
                        buf[co * pitch + (i - co * w4)] = v;
                    });
            }
            __syncthreads();
            // a warp per (input channel, tap), two output channels per store
            bf16 *dst = (bf16 *) J.out + (size_t) ci0 * Ktot + co0;
            const bool two = (nco & 1) == 0 && (knp & 1) == 0 && (Ktot & 1) == 0 && ((uintptr_t) dst & 3) == 0;
            for (int q = t >> 5; q < nci * khw; q += 8) {
                const int r = q / khw, g = q - r * khw;
                const float *v = buf + r * khw + taps[g];
                bf16 *o = dst + (size_t) r * Ktot + g * knp;
                if (two)
                    for (int co = 2 * lane; co < nco; co += 64)
                        *reinterpret_cast<__nv_bfloat162 *>(o + co) = __floats2bfloat162_rn(v[co * pitch], v[(co + 1) * pitch]);
                else
                    for (int co = lane; co < nco; co += 32) o[co] = __float2bfloat16_rn(v[co * pitch]);
            }
            if (co0 == 0)   // the K padding after the taps
                for (int r = 0; r < nci; r++)
                    for (int k = khw * knp + t; k < Ktot; k += 256) dst[(size_t) r * Ktot + k] = __float2bfloat16_rn(0.0f);
            return;
        }
        default: {   // PREP_DGRAD: block = (4 input channels, one stride-phase class): the class's
                     // K segment of those rows, taps x knp output channels and the K padding after them
            const int c = lb % J.info.ncls, ci0 = (lb / J.info.ncls) * 4;
            const int beg = J.info.kbeg[c], end = c + 1 < J.info.ncls ? J.info.kbeg[c + 1] : J.info.Ktot;
            const int nt = J.info.ntaps[c];
            if (!J.nchw && (J.kn & 3) == 0 && (J.knp & 3) == 0 && ((beg | end | J.info.Ktot) & 3) == 0 &&
                ((uintptr_t) J.w & 15) == 0 && ((uintptr_t) J.out & 7) == 0) {
                // NHWC-API weights: four consecutive output channels per 16-byte load and 8-byte
                // store; long rows one after the other (to find its row by a division per value took 470 x 664 x 3 x 3 from
                // 15 us to 21 a round of six; 13 so)
                if (t < nt) taps[t] = J.info.kx[J.info.tap0[c] + t] * J.kw + J.info.ky[J.info.tap0[c] + t];
                __syncthreads();
                const int nq = (end - beg) >> 2, khw = J.kh * J.kw, kn = J.kn, knp = J.knp, Ktot = J.info.Ktot;
                const FastDiv dknp = J.dknp;
                const float *w = J.w + (size_t) ci0 * khw * kn;
                bf16 *out = (bf16 *) J.out + (size_t) ci0 * Ktot + beg;
                const int nci = min(4, J.C - ci0);
                auto load = [&](int r, int idx) {
                    const int g = (int) dknp.div((uint32_t) idx), co = idx - g * knp;
                    if (g >= nt || co >= kn) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    return __ldg(reinterpret_cast<const float4 *>(w + ((size_t) r * khw + taps[g]) * kn + co));
                };
                auto store = [&](int r, int idx, float4 v) {
                    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                    uint2 u;
                    u.x = *reinterpret_cast<uint32_t *>(&lo);
                    u.y = *reinterpret_cast<uint32_t *>(&hi);
                    *reinterpret_cast<uint2 *>(out + (size_t) r * Ktot + idx) = u;
                };
                if (nq <= 128) {   // short rows side by side
                    batched<2, float4>(
                        4 * nq, [&](int i) { return (i & 3) < nci ? load(i & 3, i & ~3) : make_float4(0.0f, 0.0f, 0.0f, 0.0f); },
                        [&](int i, float4 v) { if ((i & 3) < nci) store(i & 3, i & ~3, v); });
                } else {
                    for (int r = 0; r < nci; r++)
#pragma unroll 4
                        for (int q = t; q < nq; q += 256) store(r, 4 * q, load(r, 4 * q));
                }
                return;
            }
            for (int r = 0; r < 4; r++) {
                const int ci = ci0 + r;
                if (ci >= J.C) break;
                bf16 *row = (bf16 *) J.out + (size_t) ci * J.info.Ktot + beg;
                for (int idx = t; idx < end - beg; idx += 256) {
                    const int g = (int) J.dknp.div((uint32_t) idx), co = idx - g * J.knp;
                    float v = 0.0f;
                    if (g < nt && co < J.kn) v = wref(J.w, J.nchw, J.C, J.kh, J.kw, J.kn, ci, J.info.kx[J.info.tap0[c] + g], J.info.ky[J.info.tap0[c] + g], co);
                    row[idx] = __float2bfloat16_rn(v);
                }
            }
        }
    }
}

int grid_for(long long n) {
    long long g = (n + 255) / 256;
    return (int) (g > 152 * 32 ? 152 * 32 : (g < 1 ? 1 : g));
}

}  // namespace

cudaError_t prep_pack_fwd(const float *w, int nchw, int C, int kh, int kw, int kn, int Cp, int Kpad, void *out,
                          cudaStream_t st) {
    if (nchw) {
        cg_launch_pdl(pack_fwd_kernel, dim3(grid_for((long long) kn * Kpad)), dim3(256), 0, st, w, nchw, C, kh, kw, kn, Cp, Kpad, (bf16 *) out);
        return cudaGetLastError();
    }
    const int khw = kh * kw;
    dim3 grid((Cp + 31) / 32, (kn + 31) / 32, khw), block(32, 8);
    cg_launch_pdl(pack_fwd_tiled_kernel, grid, block, 0, st, w, C, khw, kn, Cp, Kpad, (bf16 *) out);
    if (Kpad > khw * Cp)
        cg_launch_pdl(pack_fwd_tail_kernel, dim3(grid_for((long long) kn * (Kpad - khw * Cp))), dim3(256), 0, st, kn, khw * Cp, Kpad, (bf16 *) out);
    return cudaGetLastError();
}

cudaError_t prep_pack_dgrad(const float *w, int nchw, int C, int kh, int kw, int kn, int knp,
                            const PackDgradInfo &info, void *out, cudaStream_t st) {
    cg_launch_pdl(pack_dgrad_kernel, dim3(grid_for((long long) C * info.Ktot)), dim3(256), 0, st, w, nchw, C, kh, kw, kn, knp, info, (bf16 *) out);
    return cudaGetLastError();
}

cudaError_t prep_fold(int kn, const float *bias, const float *mean, const float *inv_std, const float *gamma,
                      const float *beta, float *scale, float *shift, cudaStream_t st) {
    cg_launch_pdl(fold_kernel, dim3((kn + 127) / 128), dim3(128), 0, st, kn, bias, mean, inv_std, gamma, beta, scale, shift);
    return cudaGetLastError();
}

cudaError_t prep_to_bf16_nhwc(const float *in, int nchw, int B, int C, int H, int W, int Cp, void *out,
                              cudaStream_t st) {
    const long long HW = (long long) H * W, P = B * HW;
    const bool vin = ((uintptr_t) in & 15) == 0;
    if ((uintptr_t) out & 15 || HW > (1LL << 30) || B > 65535 || Cp > 64 * 65535) {
        cg_launch_pdl(to_bf16_nhwc_kernel, dim3(grid_for(P * Cp)), dim3(256), 0, st, in, nchw, B, C, H, W, Cp, (bf16 *) out);
    } else if (!nchw) {
        cg_launch_pdl(nhwc_to_bf16_kernel, dim3(grid_for(P * (Cp / 8))), dim3(256), 0, st, in, C, Cp, P * (Cp / 8), vin && C == Cp, (uint4 *) out);
    } else if (C <= 8) {
        cg_launch_pdl(nchw_few_to_bf16_kernel, dim3((unsigned) ((HW + 1023) / 1024), (unsigned) B), dim3(256), 0, st, in, C, (int) HW, (uint4 *) out);
    } else {
        const dim3 grid((unsigned) ((HW + 63) / 64), (unsigned) ((Cp + 63) / 64), (unsigned) B);
        cg_launch_pdl(nchw_tiled_to_bf16_kernel, grid, dim3(256), 0, st, in, C, (int) HW, Cp, vin && HW % 4 == 0, (uint4 *) out);
    }
    return cudaGetLastError();
}

cudaError_t prep_fp8_quantize(long long n, int in_bf16, const void *in, void *out, float *scale, unsigned *amax_tmp,
                              cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(amax_tmp, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    const long long na = ((uintptr_t) in & 15) == 0 ? n / 8 : 0, nq = ((uintptr_t) out & 7) == 0 ? na : 0;
    const int ga = (int) std::min<long long>(grid_for(na ? na : n), 152 * 8), gq = nq ? (int) std::min<long long>(grid_for((nq + 3) / 4), 152 * 4) : grid_for(n);
    if (in_bf16) {
        cg_launch_pdl(amax_kernel<true>, dim3(ga), dim3(256), 0, st, in, na, n, amax_tmp);
        cg_launch_pdl(quant_e4m3_kernel<true>, dim3(gq), dim3(256), 0, st, in, nq, n, amax_tmp, (uint8_t *) out, scale);
    } else {
        cg_launch_pdl(amax_kernel<false>, dim3(ga), dim3(256), 0, st, in, na, n, amax_tmp);
        cg_launch_pdl(quant_e4m3_kernel<false>, dim3(gq), dim3(256), 0, st, in, nq, n, amax_tmp, (uint8_t *) out, scale);
    }
    return cudaGetLastError();
}

cudaError_t prep_pack_fp8(const float *w, int nchw, int C, int kh, int kw, int kn, int Cp, int Kpad, void *out,
                          float *wscale, cudaStream_t st) {
    cg_launch_pdl(wscale_kernel, dim3((kn + 127) / 128), dim3(128), 0, st, w, nchw, C * kh * kw, kn, wscale);
    cg_launch_pdl(pack_fp8_kernel, dim3(grid_for((long long) kn * Kpad)), dim3(256), 0, st, w, nchw, C, kh, kw, kn, Cp, Kpad, wscale, (uint8_t *) out);
    return cudaGetLastError();
}

cudaError_t prep_fp8_scales(int kn, const float *scale, const float *shift, const float *wscale, const float *xscale,
                            float *out_scale, float *out_shift, cudaStream_t st) {
    cg_launch_pdl(fp8_scales_kernel, dim3((kn + 127) / 128), dim3(128), 0, st, kn, scale, shift, wscale, xscale, out_scale, out_shift);
    return cudaGetLastError();
}

cudaError_t prep_split(long long n, const float *in, void *hi, void *lo, cudaStream_t st) {
    const long long n8 = (((uintptr_t) in | (uintptr_t) hi | (uintptr_t) lo) & 15) == 0 ? n / 8 : 0;
    cg_launch_pdl(split_kernel, dim3(grid_for(n8 ? n8 : n)), dim3(256), 0, st, in, n8, n, (bf16 *) hi, (bf16 *) lo);
    return cudaGetLastError();
}

cudaError_t prep_pack_split(const float *w, int nchw, int C, int kh, int kw, int kn, int Cp, int Kpad, void *hi,
                            void *lo, cudaStream_t st) {
    cg_launch_pdl(pack_split_kernel, dim3(grid_for((long long) kn * Kpad)), dim3(256), 0, st, w, nchw, C, kh, kw, kn, Cp, Kpad, (bf16 *) hi, (bf16 *) lo);
    return cudaGetLastError();
}

cudaError_t prep_group_launch(const PrepJob *jobs, int njobs, int nblocks, cudaStream_t st) {
    const int *b0 = (const int *) (jobs + njobs);
    static bool attr = false;   // up to 12288 job offsets (48 KB) beside the 16.6 KB transpose tile
    if (!attr) {
        if (cudaError_t e = cudaFuncSetAttribute(prep_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 12288 * (int) sizeof(int)))
            return e;
        attr = true;
    }
    return cg_launch_pdl(prep_group_kernel, dim3(nblocks), dim3(256), sizeof(int) * njobs, st, jobs, b0, njobs);
}
