// Training-mode batch normalisation around the BF16 forward: the convolution's
// epilogue writes, per group of 32 output pixels, the FP32 sum and sum of squares of
// z = acc * scale + shift for each channel (tc_conv.cu / tc_stem.cu); this file
//   * reduces those partials in a fixed order into FP64 per-channel sums (bit-for-bit
//     reproducible: no atomics),
//   * folds the batch mean / biased variance with gamma / beta into the per-channel
//     scale / shift of the normalisation,
//   * applies y = relu?(z * scale + shift) to the BF16 NHWC output.
// The reference's epilogue is inference-style batch norm only (running statistics,
// src/im2row_nhwc.c:279-280); these are the training-step kernels either side of it.
#include <cstring>

#include <numeric>

#include <cuda_bf16.h>

#include "../../include/convgemm_gpu.h"
#include "cg_common.cuh"
#include "cg_internal.h"
#include "tc_host.h"
#include "tc_ptx.cuh"

namespace {

constexpr int BN_CHUNK = CG_STAT_CHUNK;

// Pass 1: block (x = 8 channels, y = a chunk of BN_CHUNK groups) sums its groups for
// its channels in FP64, the 32 thread rows strided over the chunk, then in a fixed
// order across the rows.  part: [ngroups][2][kn] FP32; out: [nchunks][2][kn] FP64 (PLANES = 1: the
// sums alone). FP64 arithmetic bounds it, so blocks are narrow enough for every SM to have some (32
// channels wide, 7168 groups x 64 channels made 56 blocks: 22 us), and the conversions are done on the
// integer pipe (17 us with them on the FP64 pipe, 12 us so).
__device__ __forceinline__ double widen(float f) {   // (double) f
    const uint32_t u = __float_as_uint(f), e = u >> 23 & 255;
    if (e - 1u < 254u) return __hiloint2double((int) ((u & 0x80000000u) | ((u & 0x7FFFFFFFu) >> 3) + 0x38000000u), (int) (u << 29));
    return (u << 1) == 0 ? __hiloint2double((int) u, 0) : (double) f;   // zero; subnormal, infinite, NaN
}
// With one chunk of all groups its sums are the result, and the second kernel is not needed: OUT double writes them like
// the chunk sums, OUT float the first plane's. That leaves one block per 8 channels, so it is for what one chunk holds, and
// up to two chunks of few channels (500 groups of 64 channels with their forward 10.4 us, 10.3 in two passes; 1000 groups 30
// and 17; 375 groups of 256 channels 25 and 19). The column sums, half the loads, have a line of their own.
inline bool one_pass(long long ngroups, int kn) { return ngroups <= BN_CHUNK || (ngroups <= 2 * BN_CHUNK && ngroups * kn <= 36864); }
template <int PLANES, class OUT>
__global__ void __launch_bounds__(256) bn_stats_pass1(const float *__restrict__ part, int ngroups, int chunk, int kn,
        OUT *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    __shared__ double red[PLANES][32][9];
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    const int c = blockIdx.x * 8 + tx;
    const int g1 = min(ngroups, (int) (blockIdx.y + 1) * chunk);
    double s[PLANES] = {};
    if (c < kn)
        for (int g0 = blockIdx.y * chunk; g0 < g1; g0 += BN_CHUNK) {
            float v[PLANES][BN_CHUNK / 32];   // eight groups in flight, added in order
#pragma unroll
            for (int j = 0; j < BN_CHUNK / 32; j++) {
                const int g = g0 + ty + 32 * j;
#pragma unroll
                for (int p = 0; p < PLANES; p++) v[p][j] = g < g1 ? __ldg(part + ((size_t) g * 2 + p) * kn + c) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < BN_CHUNK / 32; j++)
#pragma unroll
                for (int p = 0; p < PLANES; p++) s[p] += widen(v[p][j]);
        }
#pragma unroll
    for (int p = 0; p < PLANES; p++) red[p][ty][tx] = s[p];
    __syncthreads();
    if (ty < PLANES && c < kn) {
        double a = 0.0;
#pragma unroll
        for (int r = 0; r < 32; r++) a += red[ty][r][tx];
        out[(size_t) blockIdx.y * 2 * kn + (size_t) ty * kn + c] = (OUT) a;
    }
}

// Pass 2, block = 32 columns: the chunks in order, eight thread rows strided over them, then the rows in
// order. Returns the total to thread row 0.
__device__ __forceinline__ double chunk_total(const double *__restrict__ chunks, int nchunks, int stride, int i, bool in) {
    __shared__ double red[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double a = 0.0;
    if (in) {
        int j = ty;
        for (; j + 56 < nchunks; j += 64) {   // eight loads in flight, added in order
            double v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = chunks[(size_t) (j + 8 * k) * stride + i];
#pragma unroll
            for (int k = 0; k < 8; k++) a += v[k];
        }
        for (; j < nchunks; j += 8) a += chunks[(size_t) j * stride + i];
    }
    red[ty][tx] = a;
    __syncthreads();
    a = 0.0;
    if (ty == 0)
        for (int r = 0; r < 8; r++) a += red[r][tx];
    return a;
}
// stats[0][c] = sum, stats[1][c] = sum of squares.
__global__ void __launch_bounds__(256) bn_stats_pass2(const double *__restrict__ chunks, int nchunks, int kn, double *__restrict__ stats) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const int i = blockIdx.x * 32 + (threadIdx.x & 31);
    const double a = chunk_total(chunks, nchunks, 2 * kn, i, i < 2 * kn);
    if (threadIdx.x < 32 && i < 2 * kn) stats[i] = a;
}

// Column sums in FP32: out[c] = sum over the chunks of the first statistics plane.
__global__ void __launch_bounds__(256) colsum_pass2_f32(const double *__restrict__ chunks, int nchunks, int kn, float *__restrict__ out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const int c = blockIdx.x * 32 + (threadIdx.x & 31);
    const double a = chunk_total(chunks, nchunks, 2 * kn, c, c < kn);
    if (threadIdx.x < 32 && c < kn) out[c] = (float) a;
}

__global__ void bn_fold_kernel(int kn, const double *__restrict__ stats, double inv_count, const float *gamma,
                               const float *beta, float eps, float *scale, float *shift, float *mean_out,
                               float *var_out) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= kn) return;
    const double mean = stats[c] * inv_count;
    double var = stats[kn + c] * inv_count - mean * mean;
    if (var < 0.0) var = 0.0;
    const double sc = (gamma ? (double) gamma[c] : 1.0) / sqrt(var + (double) eps);
    scale[c] = (float) sc;
    shift[c] = (float) ((beta ? (double) beta[c] : 0.0) - mean * sc);
    if (mean_out) mean_out[c] = (float) mean;
    if (var_out) var_out[c] = (float) var;
}

// y = relu?(z * scale + shift), BF16 NHWC [npix][kn], 8 channels per thread step. HBM-bound: a thread keeps its eight
// channels (the number of threads is a multiple of k8 = kn / 8) and has four loads in flight; with a 64-bit division
// and the tables read at each step, 103 MB in and 103 out took 37 us, 31 so (30 at the rate of a copy).
__global__ void __launch_bounds__(256) bn_apply_kernel(long long n8, int k8, const uint4 *z, const float *__restrict__ scale,
        const float *__restrict__ shift, int relu, uint4 *y) {
    tc::pdl_wait();
    tc::pdl_trigger();
    const long long step = (long long) gridDim.x * blockDim.x;
    long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    const int c0 = (int) (i % k8) * 8;
    float sc[8], sh[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        sc[j] = __ldg(scale + c0 + j);
        sh[j] = __ldg(shift + c0 + j);
    }
    for (; i < n8; i += 4 * step) {
        uint4 u[4];   // z may be y: each thread reads its elements before it writes them
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (i + k * step < n8) u[k] = z[i + k * step];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i + k * step >= n8) break;
            uint32_t w[4] = {u[k].x, u[k].y, u[k].z, u[k].w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(&w[j]);
                float a = fmaf(__bfloat162float(h.x), sc[2 * j], sh[2 * j]);
                float b = fmaf(__bfloat162float(h.y), sc[2 * j + 1], sh[2 * j + 1]);
                if (relu) {
                    a = fmaxf(a, 0.0f);
                    b = fmaxf(b, 0.0f);
                }
                const __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
                w[j] = *reinterpret_cast<const uint32_t *>(&r);
            }
            y[i + k * step] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// dz = bf16(gy * (y > 0) * scale), 8 channels per thread step. One pass over memory (6 bytes per value) and one
// launch for the five of the same expression in tensor operations; the products in their order, so that a NaN or
// an infinity under the mask and the sign of a zero stay what they were.
__global__ void epilogue_grad_kernel(uint32_t n8, uint32_t k8, const uint4 *__restrict__ gy, const uint4 *__restrict__ y,
                                     const float *__restrict__ scale, uint4 *__restrict__ dz) {
    tc::pdl_wait();
    tc::pdl_trigger();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += gridDim.x * blockDim.x) {
        const uint4 ug = gy[i], uy = y ? y[i] : ug;
        const uint32_t wg[4] = {ug.x, ug.y, ug.z, ug.w}, wy[4] = {uy.x, uy.y, uy.z, uy.w};
        const float *sc = scale ? scale + i % k8 * 8 : nullptr;
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const __nv_bfloat162 g = *reinterpret_cast<const __nv_bfloat162 *>(&wg[j]);
            const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162 *>(&wy[j]);
            float a = __bfloat162float(g.x), b = __bfloat162float(g.y);
            if (y) {
                a = __fmul_rn(a, __bfloat162float(v.x) > 0.0f ? 1.0f : 0.0f);
                b = __fmul_rn(b, __bfloat162float(v.y) > 0.0f ? 1.0f : 0.0f);
            }
            if (sc) {
                a = __fmul_rn(a, __ldg(sc + 2 * j));
                b = __fmul_rn(b, __ldg(sc + 2 * j + 1));
            }
            const __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
            o[j] = *reinterpret_cast<const uint32_t *>(&r);
        }
        dz[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// statistics groups of the forward's path for this shape: the small-channel kernel
// groups per (output row, 128-pixel chunk), the general kernel per 32 output pixels
int stat_groups(const cg_shape &s, bool *stem) {
    const ConvGeom g = make_geom(s);
    *stem = tc_stem_applicable(s);
    return *stem ? tc_stem_stat_groups(s) : (int) (((long long) s.b * g.ho * g.wo + 31) / 32);
}

size_t stats_ws_bytes(const cg_shape &s) {
    bool stem;
    const long long ng = stat_groups(s, &stem);
    const long long nchunks = (ng + BN_CHUNK - 1) / BN_CHUNK;
    // FP64 chunk sums first (8-byte aligned), then the FP32 group partials
    return (size_t) (nchunks * 2 * s.kn * 8 + ng * 2 * s.kn * 4);
}

}  // namespace

size_t cg_colsum_ws_bytes(long long ngroups, int kn) {
    const long long nchunks = (ngroups + BN_CHUNK - 1) / BN_CHUNK;
    return (size_t) (nchunks * 2 * kn * 8 + ngroups * 2 * kn * 4);
}

cudaError_t cg_colsum_reduce(void *workspace, int ngroups, int kn, float *out, cudaStream_t st) {
    const int nchunks = (ngroups + BN_CHUNK - 1) / BN_CHUNK;
    double *chunks = (double *) workspace;
    const float *part = (const float *) ((uint8_t *) workspace + (size_t) nchunks * 2 * kn * 8);
    // One pass up to two chunks of groups, of any width: never behind two on 36 input gradients of 263 to 500 groups (392 groups of
    // 256 channels with their 3 x 3: 32.8 us, 34.8 in two; 512 -> 512: 69.6, 71.7). Its blocks are launched during the tail of the
    // kernel that writes the groups where there are few of them or their chains are short; otherwise they keep its last
    // tiles waiting (392 groups of 128 channels from 512: 30.7 us, 20.5 launched plainly; 125 groups of 512: 16.6, 10.7; but
    // 392 of 64: 16.4, 18.4).
    if (ngroups <= 2 * BN_CHUNK) {
        const bool early = kn <= 64 || (ngroups <= BN_CHUNK && kn <= 256);
        cg_launch_ex(early ? CG_PDL_THREAD : CG_PDL_OFF, bn_stats_pass1<1, float>, dim3((kn + 7) / 8), dim3(256), 0, st, part,
                     ngroups, ngroups, kn, out);
        return cudaGetLastError();
    }
    dim3 g1((kn + 7) / 8, nchunks);
    // launched plainly: with its blocks launched during the tail of the kernel that writes the groups, 9 of 10 input
    // gradients took longer by 2 to 5 us (56 x 56, 256 -> 64 1 x 1, batch 64: 64 us, 66; 28 x 28, 128 -> 512: 20.6, 25), none
    // less
    cg_launch_ex(CG_PDL_OFF, bn_stats_pass1<1, double>, g1, dim3(256), 0, st, part, ngroups, BN_CHUNK, kn, chunks);
    cg_launch_pdl(colsum_pass2_f32, dim3((kn + 31) / 32), dim3(256), 0, st, chunks, nchunks, kn, out);
    return cudaGetLastError();
}

extern "C" size_t convgemm_fwd_bf16_stats_workspace_size(const convgemm_shape_t *shape) {
    if (!shape || shape->b < 1 || shape->kn < 1 || shape->c < 1) return 0;
    if (convgemm_bf16_weights_size(shape, CONVGEMM_OPERAND_FWD) == 0) return 0;
    return stats_ws_bytes(cg_from_public(*shape));
}

extern "C" convgemm_status_t convgemm_fwd_bf16_stats(const convgemm_shape_t *shape, const void *x,
        const void *wpacked, void *y, const float *scale,
        const float *shift, int relu, double *stats, void *workspace,
        size_t workspace_bytes, void *stream) {
    const char *fn = "convgemm_fwd_bf16_stats";
    if (!shape || !x || !wpacked || !y || !stats || !workspace)
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "%s: NULL argument", fn);
    const size_t need = convgemm_fwd_bf16_stats_workspace_size(shape);
    if (need == 0) return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "%s: invalid shape", fn);
    if (workspace_bytes < need || ((uintptr_t) workspace & 15))
        return cg_set_error(CONVGEMM_ERROR_WORKSPACE, "%s: workspace needs %zu bytes, 16-byte aligned", fn, need);
    if (shape->kn % 8) return cg_set_error(CONVGEMM_ERROR_NOT_SUPPORTED, "%s: kn must be a multiple of 8", fn);
    const cg_shape s = cg_from_public(*shape);
    bool stem;
    const int ng = stat_groups(s, &stem);
    const int nchunks = (ng + BN_CHUNK - 1) / BN_CHUNK;
    double *chunks = (double *) workspace;
    float *part = (float *) ((uint8_t *) workspace + (size_t) nchunks * 2 * s.kn * 8);
    const cudaStream_t st = (cudaStream_t) stream;
    TcPlan pl;
    tc_plan_fwd(s, pl);
    convgemm_status_t e;
    if (stem) {
        if (((uintptr_t) y & 15) || ((uintptr_t) wpacked & 15) || ((uintptr_t) x & 15))
            return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "%s: tensors must be 16-byte aligned", fn);
        e = tc_stem_run(s, x, wpacked, pl.Ktot, y, scale, shift, relu, st, part);
    } else {
        if (pl.ncls != 1) return cg_set_error(CONVGEMM_ERROR_NOT_SUPPORTED, "%s: forward plan with several classes", fn);
        TcTune t{0, 0};
        tc_tune_get(CONVGEMM_TUNE_FWD, *shape, &t);
        e = tc_run(pl, s, x, wpacked, y, scale, shift, relu, st, 0, nullptr, nullptr, t.bn, t.splits, nullptr, part);
    }
    if (e) return e;
    if (one_pass(ng, s.kn)) {
        cg_launch_pdl(bn_stats_pass1<2, double>, dim3((s.kn + 7) / 8), dim3(256), 0, st, part, ng, ng, s.kn, stats);
    } else {
        dim3 g1((s.kn + 7) / 8, nchunks);
        cg_launch_pdl(bn_stats_pass1<2, double>, g1, dim3(256), 0, st, part, ng, BN_CHUNK, s.kn, chunks);
        cg_launch_pdl(bn_stats_pass2, dim3((2 * s.kn + 31) / 32), dim3(256), 0, st, chunks, nchunks, s.kn, stats);
    }
    return cg_cuda_check(cudaGetLastError(), "batch statistics reduction");
}

extern "C" convgemm_status_t convgemm_bn_stats_fold(int kn, const double *stats, long long count, const float *gamma,
        const float *beta, float eps, float *scale, float *shift,
        float *batch_mean, float *batch_var, void *stream) {
    if (kn < 1 || !stats || count < 1 || !scale || !shift || !(eps >= 0.0f))
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "convgemm_bn_stats_fold: bad arguments");
    cg_launch_pdl(bn_fold_kernel, dim3((kn + 127) / 128), dim3(128), 0, (cudaStream_t) stream, kn, stats, 1.0 / (double) count, gamma, beta,
        eps, scale, shift, batch_mean, batch_var);
    return cg_cuda_check(cudaGetLastError(), "convgemm_bn_stats_fold");
}

extern "C" convgemm_status_t convgemm_bn_apply_bf16(long long npix, int kn, const void *z, const float *scale,
        const float *shift, int relu, void *y, void *stream) {
    if (npix < 1 || kn < 8 || kn % 8 || !z || !scale || !shift || !y)
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "convgemm_bn_apply_bf16: bad arguments (kn % 8 == 0)");
    if (((uintptr_t) z & 15) || ((uintptr_t) y & 15))
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "convgemm_bn_apply_bf16: tensors must be 16-byte aligned");
    const long long n8 = npix * (kn / 8);
    // four steps per thread or a wave of eight blocks per SM, rounded up to whole rows of channels
    const int k8 = kn / 8;
    long long blocks = (n8 + 1023) / 1024;
    if (blocks > 152 * 8) blocks = 152 * 8;
    const int unit = k8 / std::gcd(k8, 256);
    blocks = (blocks + unit - 1) / unit * unit;
    cg_launch_pdl(bn_apply_kernel, dim3((int) blocks), dim3(256), 0, (cudaStream_t) stream, n8, k8, (const uint4 *) z, scale, shift, relu,
        (uint4 *) y);
    return cg_cuda_check(cudaGetLastError(), "convgemm_bn_apply_bf16");
}

extern "C" convgemm_status_t convgemm_epilogue_grad_bf16(long long npix, int kn, const void *gy, const void *y,
        const float *scale, void *dz, void *stream) {
    if (npix < 1 || kn < 8 || kn % 8 || !gy || !dz || npix > ((1LL << 31) - 1) / kn)
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "convgemm_epilogue_grad_bf16: bad arguments (kn %% 8 == 0)");
    if (((uintptr_t) gy & 15) || ((uintptr_t) y & 15) || ((uintptr_t) dz & 15))
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "convgemm_epilogue_grad_bf16: tensors must be 16-byte aligned");
    const uint32_t n8 = (uint32_t) (npix * (kn / 8)), blocks = (n8 + 255) / 256;
    cg_launch_pdl(epilogue_grad_kernel, dim3(blocks < 152 * 16 ? blocks : 152 * 16), dim3(256), 0, (cudaStream_t) stream,
        n8, (uint32_t) kn / 8, (const uint4 *) gy, (const uint4 *) y, scale, (uint4 *) dz);
    return cg_cuda_check(cudaGetLastError(), "convgemm_epilogue_grad_bf16");
}
