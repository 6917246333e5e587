// FP32 plain form of the five convGemm entry points: SIMT FFMA implicit GEMM.
//
// Each output element is one fused multiply-add chain per KC=384 block of the
// reduction, blocks added in increasing order — the arithmetic of the
// reference's loop nests with a BLIS micro-kernel (the KC loop and betaI of
// src/gemm_blis_B3A2C0_orig.c:55-64, src/gemm_blis_B3A2C0.c:64; sxpbyM at
// src/gemm_blis.c:147-161), and the
// reduction index runs in the reference's order k = (c*kh + kx)*kw + ky
// (src/im2row_nhwc.c:163).  Forward and weight gradient therefore reproduce
// the reference's values, not just its tolerance.
//
// One templated kernel serves every operation; an "op" object supplies the
// implicit operands (im2row/im2col gathers straight from the activation
// tensor, never materialised), the block boundaries of the reduction and the
// store.  128-thread CTAs compute 128x128, 64x64 or 128x32 outputs, 16x8 or 8x4
// per thread, in packed pairs of FP32 multiply-adds (fma.rn.f32x2), from reduction
// slices of 16 that asynchronous copies bring into two shared-memory buffers.
// Every gather address splits into a row part (computed once per thread) and a
// reduction-index part, which the CTA tabulates in shared memory 128 indices at a
// time; which taps of a row read inside the image is a bit mask, so a gathered
// element costs a mask test, an address and a copy.  The running sum of
// completed KC blocks lives in shared memory (it is touched once per 384
// reduction steps).
//
// What bounds it: the FMA pipe's issue, 72% active on 56x56 256 -> 256 3x3 (batch
// 32, NCHW): 2.10 ms forward, 2.20 input gradient, 2.21 weight gradient (56, 54, 54
// TFLOP/s of 77 measured for independent scalar multiply-adds), against 2.91, 3.02
// and 2.76 with scalar multiply-adds, 8x8 outputs per thread and slices of 8 staged
// through registers.  That form spent its issue slots on the gather and its operand reads
// on register bank conflicts.  The same packed arithmetic with 8x8 per thread and B stored
// twice in shared memory ran at 28 TFLOP/s, with 16x8 and register staging at 47.
//
// Operands are read in the layout where a tile's column (or a B row) is
// contiguous: k x k NHWC activations through NCHW copies, single-tap NHWC rows
// as 16-byte channel vectors, weights repacked, NCHW weight-gradient operands
// through NHWC copies (see the entry points at the end).  Strided input
// gradients group their rows by stride phase (DgradPhaseOp), so each row runs
// only the taps that reach it.  None of this changes which products are added
// to an output, or in which order.
//
// Block split: when a convolution's tiles leave SMs idle or end in a thin last wave,
// the forward and input gradient run one CTA per (tile, reduction segment): each CTA
// writes the FMA chain of one KC block (input gradient: one KC block of one tap) to a
// scratch plane, and a second kernel adds the planes in order to the same start value
// (0, or dx) and applies the epilogue: the fused form's running sum, the same additions
// in the same order, so bit for bit the same result.
#include <climits>
#include <cmath>
#include <cstdint>
#include <tuple>
#include <type_traits>
#include <map>
#include <mutex>
#include <utility>
#include "cg_common.cuh"

namespace {

constexpr int BK = 16;   // reduction indices per slice
constexpr int KC = 384;
constexpr int OUT = 1 << 29;  // an input offset that puts a gather outside every image

// Which filter taps read inside the image is one bit mask per gathered position: bit kx the filter
// row, bit 16 + ky the filter column (filters up to 15 x 15). A tap reads inside when both its bits are
// set, one logic operation instead of two range tests per element. Bit 15 is never set: an index
// past the reduction range asks for it. Larger filters (BIG) keep the range tests, in every tile shape and with vector
// loads of B as the others: 17 x 17, 64 x 64, 16 -> 64, batch 4 (NHWC) 220 us forward, 1137 input gradient, 299 weight
// gradient (397, 2420, 453 with 128 x 128 tiles and element loads alone).
constexpr int MASK_TAPS = 15;
constexpr int OUT_BIT = 1 << 15;
__device__ __forceinline__ int tap_bits(int kx, int ky) { return 1 << kx | 1 << (16 + ky); }

__device__ __forceinline__ bool in_range(int v, int n) { return (unsigned) v < (unsigned) n; }

// Four consecutive outputs of one row: one 16-byte store where the caller knows p is aligned
// and all four exist, else the ones below `valid`.
__device__ __forceinline__ void store4(float *p, const float (&v)[4], bool vec, int valid) {
    if (vec && valid >= 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (j < valid) p[j] = v[j];
    }
}

// The forward epilogue, operation by operation as the reference does it
// (src/im2row_nhwc.c:276-282, src/im2col_nchw.c:422-431); the gamma/beta step is
// one fused multiply-add, as gcc contracts it in the reference's -Ofast build.
__device__ __forceinline__ float fwd_epilogue(float t, int n, const cg_epi &e) {
    if (e.bias) t = __fadd_rn(t, __ldg(e.bias + n));
    if (e.mean) {
        t = __fmul_rn(__fsub_rn(t, __ldg(e.mean + n)), __ldg(e.inv_std + n));
        t = __fmaf_rn(t, __ldg(e.gamma + n), __ldg(e.beta + n));
    }
    if (e.relu && t < 0.0f) t = 0.0f;
    return t;
}

// ---------------------------------------------------------------- forward
// GEMM rows m = output pixel p = (b*ho + ox)*wo + oy, columns n = output
// channel, reduction r = K index (c, kx, ky).
//
// Every gather is base(row) + delta(r) in both layouts, valid where the input
// position (ix(row) + ox(r), iy(row) + oy(r)) lies inside the image:
//   NHWC  ((b*h + ix)*w + iy)*c + ch = ((b*h + bix)*w + biy)*c + ((kx*vdil)*w + ky*hdil)*c + ch
//   NCHW  ((b*c + ch)*h + ix)*w + iy = ((b*c*h) + bix)*w + biy + (ch*h + kx*vdil)*w + ky*hdil
// The row part is computed once per thread, the r part once per CTA (the
// reduction-index table).
__device__ __forceinline__ int tap_mask(int bix, int biy, const ConvGeom &g) {
    int m = 0;
    for (int kx = 0; kx < g.kh; kx++) m |= in_range(bix + kx * g.vdil, g.h) ? 1 << kx : 0;
    for (int ky = 0; ky < g.kw; ky++) m |= in_range(biy + ky * g.hdil, g.w) ? 1 << (16 + ky) : 0;
    return m;
}

template <bool BIG>
struct FwdOp {
    ConvGeom g;
    int nchw;        // layout of y
    int xl, wl;      // layout of the x the kernel reads (0 NHWC, 1 NCHW) and of w (0 [K][kn], 1 [kn][K])
    int ov;          // y NHWC with 16-byte aligned rows of kn % 4 == 0
    int mv;          // y NCHW, 16-byte aligned, ho*wo % 4 == 0: four rows of one column are one vector
    const float *w, *x;
    float *y;
    cg_epi e;
    FastDiv dwo, dho, dkw, dkh;
    float *ws;   // block split: [K blocks][P][kn] chains, else NULL

    __host__ __device__ int M() const { return (int) g.P; }
    __host__ __device__ int N() const { return g.kn; }

    // p: the row's gather base (may lie outside x; never read unless a tap is valid);
    // a: tap mask (BIG: a, b the input row / column of tap (0, 0))
    struct Row { const float *p; int a, b; };
    __device__ Row row(int m) const {
        uint32_t q, oy, ox, bb;
        dwo.divmod(m < g.P ? m : 0, q, oy);
        dho.divmod(q, bb, ox);
        Row rw;
        const int bix = (int) ox * g.vstr - g.vpad, biy = (int) oy * g.hstr - g.hpad;
        rw.p = x + (xl ? ((long long) bb * g.c * g.h + bix) * g.w + biy
                       : (((long long) bb * g.h + bix) * g.w + biy) * g.c);
        if constexpr (BIG) {
            rw.a = m < g.P ? bix : -OUT;
            rw.b = biy;
        } else {
            rw.a = m < g.P ? tap_mask(bix, biy, g) : 0;
            rw.b = 0;
        }
        return rw;
    }
    struct Col { const float *p; int valid; };
    __device__ Col col(int n) const { return Col{w + (wl ? (long long) n * g.K : (long long) n), n < g.kn}; }
    struct alignas(16) REnt { int delta, a, b, bd; };
    __device__ REnt rent(int r, int rend) const {
        uint32_t q, ky, kx, c;
        dkw.divmod(r < rend ? r : 0, q, ky);
        dkh.divmod(q, c, kx);
        REnt t;
        const int offx = (int) kx * g.vdil, offy = (int) ky * g.hdil;
        t.delta = xl ? ((int) c * g.h + offx) * g.w + offy : (offx * g.w + offy) * g.c + (int) c;
        if constexpr (BIG) {
            t.a = r < rend ? offx : -OUT;
            t.b = offy;
        } else {
            t.a = r < rend ? tap_bits((int) kx, (int) ky) : OUT_BIT;
            t.b = 0;
        }
        t.bd = r < rend ? (wl ? r : r * g.kn) : -1;
        return t;
    }
    __device__ const float *asrc(const Row &rw, const REnt &t) const { return rw.p + t.delta; }
    __device__ bool ain(const Row &rw, const REnt &t) const {
        bool in;
        if constexpr (BIG) in = in_range(rw.a + t.a, g.h) && in_range(rw.b + t.b, g.w);
        else in = (~rw.a & t.a) == 0;
        return in;
    }
    // Single-tap NHWC: the row's reduction indices are its input pixel's channels, contiguous.
    __device__ const float *vrow(const Row &rw) const { return (~rw.a & tap_bits(0, 0)) == 0 ? rw.p : nullptr; }
    __device__ bool bin(const Col &cl, long long bd) const { return cl.valid && bd >= 0; }
    __device__ const float *bbase() const { return w; }   // 16-byte aligned where B is read as vectors
    __host__ __device__ int segments() const { return (g.K + KC - 1) / KC; }
    bool phased() const { return false; }
    __host__ __device__ long long rlen() const { return g.K; }
    __device__ void range(int m0, int z, int &rbeg, int &rend) const {
        if (ws) {
            rbeg = z * KC;
            rend = min(g.K, rbeg + KC);
        } else {
            rbeg = 0;
            rend = g.K;
        }
    }
    __device__ int next_fold(int r, int rend) const {
        int nf = (r / KC + 1) * KC;
        return nf >= rend ? INT_MAX : nf;
    }
    __device__ bool starts() const { return false; }
    __device__ float s_init(int m, int n) const { return 0.0f; }
    __device__ float s_start(int m, int n) const { return 0.0f; }
    __device__ int zcount(int m, int nz) const { return nz; }
    __device__ void finish_z4(int z, int m, int n, const float (&s)[4]) const {
        if (m >= (int) g.P) return;
        if (ws) return store4(ws + ((size_t) z * g.P + m) * g.kn + n, s, g.kn % 4 == 0, g.kn - n);
        finish_n4(m, n, s);
    }
    __device__ void finish_n4(int m, int n, const float (&s)[4]) const {
        if (!ov) {
#pragma unroll
            for (int j = 0; j < 4; j++) finish(m, n + j, s[j]);
            return;
        }
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = n + j < g.kn ? fwd_epilogue(s[j], n + j, e) : 0.0f;
        store4(y + (size_t) m * g.kn + n, v, true, g.kn - n);
    }
    // NCHW y: rows m .. m + 3 (m % 4 == 0) of column n
    __device__ bool by_rows() const { return mv && !ws; }
    __device__ bool by_column() const { return nchw && !ws; }
    __device__ void finish_m4(int m, int n, const float (&s)[4]) const {
        if (m >= (int) g.P || n >= g.kn) return;
        uint32_t q, oy, ox, bb;
        dwo.divmod(m, q, oy);
        dho.divmod(q, bb, ox);
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = fwd_epilogue(s[i], n, e);
        store4(y + ((size_t) bb * g.kn + n) * g.ho * g.wo + (size_t) ox * g.wo + oy, v, true, 4);
    }
    // NCHW y: channel 0 of row m, or NULL past the last
    __device__ float *out_row(int m) const {
        if (m >= (int) g.P) return nullptr;
        uint32_t q, oy, ox, bb;
        dwo.divmod(m, q, oy);
        dho.divmod(q, bb, ox);
        return y + ((size_t) bb * g.kn * g.ho + ox) * g.wo + oy;
    }
    __device__ void put(float *row, int n, float s) const {
        if (row && n < g.kn) row[(size_t) n * g.ho * g.wo] = fwd_epilogue(s, n, e);
    }
    __device__ void finish(int m, int n, float s) const {
        if (m >= (int) g.P || n >= g.kn) return;
        float v = fwd_epilogue(s, n, e);
        if (nchw) {
            uint32_t q, oy, ox, bb;
            dwo.divmod(m, q, oy);
            dho.divmod(q, bb, ox);
            y[(((size_t) bb * g.kn + n) * g.ho + ox) * g.wo + oy] = v;
        } else {
            y[(size_t) m * g.kn + n] = v;
        }
    }
};

// --------------------------------------------------------- weight gradient
// Rows m = K index, columns n = output channel, reduction r = output pixel.
// One CTA per (tile, KC block of pixels): it writes that block's partial to
// the workspace, and wgrad_reduce adds the blocks in increasing order.  The
// gather of x is the forward's with the roles swapped: the tap part comes from
// the row, the pixel part from the reduction-index table.
template <bool BIG>
struct WgradOp {
    ConvGeom g;
    int xl, yl;  // layout of the x and dy the kernel reads (0 NHWC, 1 NCHW)
    const float *dy, *x;
    float *ws;   // [nblocks][K][kn]
    int ov;      // ws 16-byte aligned, kn % 4 == 0
    FastDiv dwo, dho, dkw, dkh;

    __host__ __device__ int M() const { return g.K; }
    __host__ __device__ int N() const { return g.kn; }

    struct Row { int delta, a, b; };
    __device__ Row row(int m) const {
        uint32_t q, ky, kx, c;
        dkw.divmod(m < g.K ? m : 0, q, ky);
        dkh.divmod(q, c, kx);
        Row rw;
        const int offx = (int) kx * g.vdil, offy = (int) ky * g.hdil;
        rw.delta = xl ? ((int) c * g.h + offx) * g.w + offy : (offx * g.w + offy) * g.c + (int) c;
        if constexpr (BIG) {
            rw.a = m < g.K ? offx : -OUT;
            rw.b = offy;
        } else {
            rw.a = m < g.K ? tap_bits((int) kx, (int) ky) : OUT_BIT;
            rw.b = 0;
        }
        return rw;
    }
    struct Col { const float *p; int valid; };
    __device__ Col col(int n) const {
        return Col{dy + (yl ? (long long) n * g.ho * g.wo : (long long) n), n < g.kn};
    }
    struct REnt { long long base, bd; int a, b; };
    __device__ REnt rent(int r, int rend) const {
        uint32_t q, oy, ox, bb;
        dwo.divmod(r < rend ? r : 0, q, oy);
        dho.divmod(q, bb, ox);
        REnt t;
        const int bix = (int) ox * g.vstr - g.vpad, biy = (int) oy * g.hstr - g.hpad;
        t.base = xl ? ((long long) bb * g.c * g.h + bix) * g.w + biy
                      : (((long long) bb * g.h + bix) * g.w + biy) * g.c;
        if constexpr (BIG) {
            t.a = r < rend ? bix : -OUT;
            t.b = biy;
        } else {
            t.a = r < rend ? tap_mask(bix, biy, g) : 0;
            t.b = 0;
        }
        const long long hw = (long long) g.ho * g.wo;
        t.bd = r < rend ? (yl ? (long long) bb * g.kn * hw + ((long long) ox * g.wo + oy) : (long long) r * g.kn)
                        : -1;
        return t;
    }
    __device__ const float *asrc(const Row &rw, const REnt &t) const { return x + (t.base + rw.delta); }
    __device__ bool ain(const Row &rw, const REnt &t) const {
        bool in;
        if constexpr (BIG) in = in_range(t.a + rw.a, g.h) && in_range(t.b + rw.b, g.w);
        else in = (~t.a & rw.a) == 0;
        return in;
    }
    __device__ const float *vrow(const Row &) const { return nullptr; }
    __device__ bool bin(const Col &cl, long long bd) const { return cl.valid && bd >= 0; }
    __device__ const float *bbase() const { return dy; }   // 16-byte aligned where B is read as vectors
    __device__ bool by_rows() const { return false; }
    __device__ bool by_column() const { return false; }
    __device__ void finish_m4(int, int, const float (&)[4]) const {}
    __device__ float *out_row(int) const { return nullptr; }
    __device__ void put(float *, int, float) const {}
    __device__ void range(int m0, int z, int &rbeg, int &rend) const {
        rbeg = z * KC;
        rend = min((long long) (z + 1) * KC, g.P);
    }
    __device__ int next_fold(int r, int rend) const { return INT_MAX; }
    __device__ bool starts() const { return false; }
    __device__ float s_init(int m, int n) const { return 0.0f; }
    __device__ void finish_z4(int z, int m, int n, const float (&s)[4]) const {
        if (m < g.K) store4(ws + ((size_t) z * g.K + m) * g.kn + n, s, ov, g.kn - n);
    }
};

// ---------------------------------------------------------- input gradient
// Gather form: rows m = input pixel (b, ih, iw), columns n = input channel,
// reduction r = tap*kn + l over taps (kx, ky) and output channels l.  A tap
// contributes where (ih + vpad - kx*vdil) is a non-negative multiple of the
// stride below ho (same for iy).  Each (tap, KC block of l) partial is added
// to the running value in a fixed order; the reference adds the same partials
// with `omp atomic` in thread order (src/im2row_nhwc.c:252).
//
// With ih + vpad = vstr*xd + xm and kx*vdil = vstr*exd + exm (0 <= xm, exm < vstr),
// the tap reads output row xd - exd exactly when xm == exm, so the table holds
// (exd, exm) per r and the rows hold (xd, xm): no division per element.
// The taps whose output row / column exists for input pixel (ih, iw), as a tap mask.
__device__ __forceinline__ int reach_mask(int ih, int iw, const ConvGeom &g) {
    int m = 0;
    for (int kx = 0; kx < g.kh; kx++) {
        const int t = ih + g.vpad - kx * g.vdil;
        m |= t >= 0 && t % g.vstr == 0 && t / g.vstr < g.ho ? 1 << kx : 0;
    }
    for (int ky = 0; ky < g.kw; ky++) {
        const int t = iw + g.hpad - ky * g.hdil;
        m |= t >= 0 && t % g.hstr == 0 && t / g.hstr < g.wo ? 1 << (16 + ky) : 0;
    }
    return m;
}

template <bool BIG>
struct DgradOp {
    ConvGeom g;
    int nchw, accumulate;   // layout of dx; dx += result
    int yl;                 // layout of the dy the kernel reads (0 NHWC, 1 NCHW)
    int wl;                 // layout of w: 0 NHWC [c][tap][kn], 1 NCHW [kn][c][tap], 2 packed [tap][kn][c]
    int ov;                 // dx NHWC with 16-byte aligned rows of c % 4 == 0
    int mv;                 // dx NCHW, 16-byte aligned, h*w % 4 == 0: four rows of one column are one vector
    const float *w, *dy;
    float *dx;
    FastDiv dw_, dh_, dkn, dkw, dvs, dhs;
    float *ws;   // block split: [segment][b*h*w][c] chains (segment = tap, KC block of kn), else NULL

    __host__ __device__ int M() const { return g.b * g.h * g.w; }
    __host__ __device__ int N() const { return g.c; }

    // a: mask of the taps that reach the pixel (BIG: a, b the output row / column of tap (0, 0), cls the
    // stride phase)
    struct Row { const float *p; int a, b, cls; };
    __device__ Row row(int m) const {
        const bool valid = m < M();
        uint32_t q, iw, ih, bb, xd, xm, yd, ym;
        dw_.divmod(valid ? m : 0, q, iw);
        dh_.divmod(q, bb, ih);
        dvs.divmod(ih + g.vpad, xd, xm);
        dhs.divmod(iw + g.hpad, yd, ym);
        Row rw;
        rw.p = dy + (yl ? ((long long) bb * g.kn * g.ho + xd) * g.wo + yd
                        : (((long long) bb * g.ho + xd) * g.wo + yd) * g.kn);
        if constexpr (BIG) {
            rw.a = valid ? (int) xd : -OUT;
            rw.b = (int) yd;
            rw.cls = (int) (xm | (ym << 16));
        } else {
            rw.a = valid ? reach_mask((int) ih, (int) iw, g) : 0;
            rw.b = rw.cls = 0;
        }
        return rw;
    }
    struct Col { const float *p; int valid; };
    __device__ Col col(int n) const {
        const long long b = wl == 2 ? n : wl == 1 ? (long long) n * g.kh * g.kw : (long long) n * g.kh * g.kw * g.kn;
        return Col{w + b, n < g.c};
    }
    struct alignas(16) REntM { int delta, a, b, bd; };
    struct alignas(16) REntB { int delta, a, b, bd, cls, pad[3]; };
    using REnt = std::conditional_t<BIG, REntB, REntM>;
    __device__ REnt rent(int r, int rend) const {
        uint32_t tap, l, kx, ky, exd, exm, eyd, eym;
        dkn.divmod(r < rend ? r : 0, tap, l);
        dkw.divmod(tap, kx, ky);
        dvs.divmod(kx * g.vdil, exd, exm);
        dhs.divmod(ky * g.hdil, eyd, eym);
        REnt t;
        t.delta = yl ? ((int) l * g.ho - (int) exd) * g.wo - (int) eyd
                     : (int) l - ((int) exd * g.wo + (int) eyd) * g.kn;
        if constexpr (BIG) {
            t.a = r < rend ? -(int) exd : -OUT;
            t.b = -(int) eyd;
            t.cls = (int) (exm | (eym << 16));
        } else {
            t.a = r < rend ? tap_bits((int) kx, (int) ky) : OUT_BIT;
            t.b = 0;
        }
        t.bd = r < rend ? (wl == 2 ? r * g.c : wl == 1 ? (int) l * g.K + (int) tap : r) : -1;
        return t;
    }
    __device__ const float *asrc(const Row &rw, const REnt &t) const { return rw.p + t.delta; }
    __device__ bool ain(const Row &rw, const REnt &t) const {
        bool in;
        if constexpr (BIG) in = rw.cls == t.cls && in_range(rw.a + t.a, g.ho) && in_range(rw.b + t.b, g.wo);
        else in = (~rw.a & t.a) == 0;
        return in;
    }
    // Single-tap NHWC: the row's reduction indices are its output pixel's channels, contiguous.
    __device__ const float *vrow(const Row &rw) const { return (~rw.a & tap_bits(0, 0)) == 0 ? rw.p : nullptr; }
    __device__ bool bin(const Col &cl, long long bd) const { return cl.valid && bd >= 0; }
    __device__ const float *bbase() const { return w; }   // 16-byte aligned where B is read as vectors
    __host__ __device__ int segments() const { return g.kh * g.kw * ((g.kn + KC - 1) / KC); }
    bool phased() const { return false; }
    __host__ __device__ long long rlen() const { return (long long) g.kh * g.kw * g.kn; }
    __device__ void range(int m0, int z, int &rbeg, int &rend) const {
        if (ws) {
            const int nch = (g.kn + KC - 1) / KC, tap = z / nch, j = z - tap * nch;
            rbeg = tap * g.kn + j * KC;
            rend = tap * g.kn + min(g.kn, (j + 1) * KC);
        } else {
            rbeg = 0;
            rend = g.kh * g.kw * g.kn;
        }
    }
    __device__ int next_fold(int r, int rend) const {
        uint32_t tap, l;
        dkn.divmod(r, tap, l);
        int nf = r - (int) l + min(g.kn, (int) (l / KC + 1) * KC);
        return nf >= rend ? INT_MAX : nf;
    }
    __device__ size_t out_index(int m, int n) const {
        if (!nchw) return (size_t) m * g.c + n;
        uint32_t q, iw, ih, bb;
        dw_.divmod(m, q, iw);
        dh_.divmod(q, bb, ih);
        return (((size_t) bb * g.c + n) * g.h + ih) * g.w + iw;
    }
    __device__ bool starts() const { return accumulate && !ws; }   // split: the reduction starts from dx
    __device__ float s_init(int m, int n) const { return m < M() && n < g.c ? dx[out_index(m, n)] : 0.0f; }
    __device__ float s_start(int m, int n) const {
        if (!accumulate || m >= M() || n >= g.c) return 0.0f;
        return dx[out_index(m, n)];
    }
    __device__ int zcount(int m, int nz) const { return nz; }
    __device__ void finish_z4(int z, int m, int n, const float (&s)[4]) const {
        if (m >= M()) return;
        if (ws) return store4(ws + ((size_t) z * M() + m) * g.c + n, s, g.c % 4 == 0, g.c - n);
        finish_n4(m, n, s);
    }
    __device__ void finish_n4(int m, int n, const float (&s)[4]) const {
        if (ov) return store4(dx + (size_t) m * g.c + n, s, true, g.c - n);
#pragma unroll
        for (int j = 0; j < 4; j++) finish(m, n + j, s[j]);
    }
    // NCHW dx: rows m .. m + 3 (m % 4 == 0) of column n
    __device__ bool by_rows() const { return mv && !ws; }
    __device__ bool by_column() const { return nchw && !ws; }
    __device__ void finish_m4(int m, int n, const float (&s)[4]) const {
        if (m < M() && n < g.c) store4(dx + out_index(m, n), s, true, 4);
    }
    __device__ float *out_row(int m) const { return m < M() ? dx + out_index(m, 0) : nullptr; }   // NCHW dx: channel 0
    __device__ void put(float *row, int n, float s) const {
        if (row && n < g.c) row[(size_t) n * g.h * g.w] = s;
    }
    __device__ void finish(int m, int n, float s) const {
        if (m >= M() || n >= g.c) return;
        dx[out_index(m, n)] = s;
    }
};


// ------------------------------------------- input gradient, strided layers
// The gather form above runs every tap for every input pixel, although with strides
// (sv, sh) a pixel of stride phase (xm, ym) = ((ih + vpad) % sv, (iw + hpad) % sh) is
// reached only by the taps of the same phase.  Here the GEMM rows are the input pixels
// grouped by phase (each phase padded to a multiple of 256 rows, so no tile straddles
// two), and a phase's reduction runs over its own taps only, in increasing tap order:
// the segments (tap, KC block of kn) of a pixel are those of the gather form minus the
// ones whose products are all zero, added in the same order.
constexpr int DG_MAXCLS = 16, DG_MAXTAPS = 64;
struct DgPhase {
    int mbeg, rows;   // first (padded) GEMM row, pixels of this phase
    int ih0, iw0;     // first input row / column of this phase
    int rbeg, ntaps;  // reduction indices [rbeg, rbeg + ntaps*kn), taps tap0 .. tap0 + ntaps - 1
    int tap0;
    FastDiv dwc, dhc; // phase columns and rows per image
};
template <bool BIG>
struct DgradPhaseOp {
    ConvGeom g;
    int nchw, accumulate, yl, wl, ov;   // as in DgradOp
    const float *w, *dy;
    float *dx;
    FastDiv dkn, dvs, dhs;
    int ncls, mpad, nkb;            // phases, padded rows, KC blocks per tap
    DgPhase ph[DG_MAXCLS];
    unsigned char taps[DG_MAXTAPS]; // tap indices kx*kw + ky grouped by phase
    float *ws;

    __host__ __device__ int M() const { return mpad; }
    __host__ __device__ int N() const { return g.c; }
    __device__ int phase_of_m(int m) const {
        int c = 0;
        for (int i = 1; i < ncls; i++) c = m >= ph[i].mbeg ? i : c;
        return c;
    }
    __device__ int phase_of_r(int r) const {
        int c = 0;
        for (int i = 1; i < ncls; i++) c = r >= ph[i].rbeg && ph[i].ntaps ? i : c;
        return c;
    }
    // GEMM row -> input pixel (b, ih, iw), or false for padding rows
    __device__ bool pixel(int m, uint32_t &bb, int &ih, int &iw) const {
        const DgPhase &p = ph[phase_of_m(m)];
        const int loc = m - p.mbeg;
        uint32_t q, tw, th;
        p.dwc.divmod(loc < p.rows ? loc : 0, q, tw);
        p.dhc.divmod(q, bb, th);
        ih = p.ih0 + (int) th * g.vstr;
        iw = p.iw0 + (int) tw * g.hstr;
        return loc < p.rows;
    }

    struct Row { const float *p; int a, b; };
    __device__ Row row(int m) const {
        uint32_t bb;
        int ih, iw;
        const bool valid = pixel(m, bb, ih, iw);
        const int xd = (ih + g.vpad) / g.vstr, yd = (iw + g.hpad) / g.hstr;   // exact for this phase
        Row rw;
        rw.p = dy + (yl ? ((long long) bb * g.kn * g.ho + xd) * g.wo + yd
                        : (((long long) bb * g.ho + xd) * g.wo + yd) * g.kn);
        if constexpr (BIG) {
            rw.a = valid ? xd : -OUT;
            rw.b = yd;
        } else {
            rw.a = valid ? reach_mask(ih, iw, g) : 0;
            rw.b = 0;
        }
        return rw;
    }
    __device__ const float *vrow(const Row &rw) const { return (~rw.a & tap_bits(0, 0)) == 0 ? rw.p : nullptr; }
    struct Col { const float *p; int valid; };
    __device__ Col col(int n) const {
        const long long b = wl == 2 ? n : wl == 1 ? (long long) n * g.kh * g.kw : (long long) n * g.kh * g.kw * g.kn;
        return Col{w + b, n < g.c};
    }
    struct alignas(16) REnt { int delta, a, b, bd; };
    __device__ REnt rent(int r, int rend) const {
        const DgPhase &p = ph[phase_of_r(r)];
        uint32_t j, l;
        dkn.divmod(r < rend ? r - p.rbeg : 0, j, l);
        const int tap = p.ntaps > 0 ? taps[p.tap0 + min((int) j, p.ntaps - 1)] : 0;
        const int kx = tap / g.kw, ky = tap - kx * g.kw;
        const int exd = kx * g.vdil / g.vstr, eyd = ky * g.hdil / g.hstr;
        REnt t;
        t.delta = yl ? ((int) l * g.ho - exd) * g.wo - eyd : (int) l - (exd * g.wo + eyd) * g.kn;
        if constexpr (BIG) {
            t.a = r < rend ? -exd : -OUT;
            t.b = -eyd;
        } else {
            t.a = r < rend ? tap_bits(kx, ky) : OUT_BIT;
            t.b = 0;
        }
        const int rg = tap * g.kn + (int) l;   // reduction index of the gather form
        t.bd = r < rend ? (wl == 2 ? rg * g.c : wl == 1 ? (int) l * g.K + tap : rg) : -1;
        return t;
    }
    __device__ const float *asrc(const Row &rw, const REnt &t) const { return rw.p + t.delta; }
    __device__ bool ain(const Row &rw, const REnt &t) const {
        bool in;
        if constexpr (BIG) in = in_range(rw.a + t.a, g.ho) && in_range(rw.b + t.b, g.wo);
        else in = (~rw.a & t.a) == 0;
        return in;
    }
    __device__ bool bin(const Col &cl, long long bd) const { return cl.valid && bd >= 0; }
    __device__ const float *bbase() const { return w; }   // 16-byte aligned where B is read as vectors
    __device__ bool by_rows() const { return false; }
    __device__ bool by_column() const { return nchw && !ws; }
    __device__ void finish_m4(int, int, const float (&)[4]) const {}
    bool phased() const { return true; }
    __host__ __device__ int segments() const {
        int nt = 0;
        for (int i = 0; i < ncls; i++) nt = ph[i].ntaps > nt ? ph[i].ntaps : nt;
        return nt * nkb;
    }
    __host__ __device__ long long rlen() const { return (long long) segments() * min(g.kn, KC); }
    __device__ void range(int m0, int z, int &rbeg, int &rend) const {
        const DgPhase &p = ph[phase_of_m(m0)];
        if (ws) {
            const int j = z / nkb, kb = z - j * nkb;
            if (j >= p.ntaps) {
                rbeg = rend = p.rbeg;
                return;
            }
            rbeg = p.rbeg + j * g.kn + kb * KC;
            rend = p.rbeg + j * g.kn + min(g.kn, (kb + 1) * KC);
        } else {
            rbeg = p.rbeg;
            rend = p.rbeg + p.ntaps * g.kn;
        }
    }
    __device__ int next_fold(int r, int rend) const {
        const DgPhase &p = ph[phase_of_r(r)];
        uint32_t j, l;
        dkn.divmod(r - p.rbeg, j, l);
        int nf = r - (int) l + min(g.kn, (int) (l / KC + 1) * KC);
        return nf >= rend ? INT_MAX : nf;
    }
    __device__ int zcount(int m, int nz) const { return ph[phase_of_m(m)].ntaps * nkb; }
    __device__ bool out_index(int m, int n, size_t &o) const {
        uint32_t bb;
        int ih, iw;
        if (!pixel(m, bb, ih, iw) || n >= g.c) return false;
        o = nchw ? (((size_t) bb * g.c + n) * g.h + ih) * g.w + iw : (((size_t) bb * g.h + ih) * g.w + iw) * g.c + n;
        return true;
    }
    __device__ float s_start(int m, int n) const {
        size_t o;
        return accumulate && out_index(m, n, o) ? dx[o] : 0.0f;
    }
    __device__ bool starts() const { return accumulate && !ws; }
    __device__ float s_init(int m, int n) const { return s_start(m, n); }
    __device__ void finish_z4(int z, int m, int n, const float (&s)[4]) const {
        if (ws) {
            if (z < zcount(m, 0)) store4(ws + ((size_t) z * mpad + m) * g.c + n, s, g.c % 4 == 0, g.c - n);
            return;
        }
        finish_n4(m, n, s);
    }
    __device__ void finish_n4(int m, int n, const float (&s)[4]) const {
        size_t o;
        if (!out_index(m, n, o)) return;
        if (!nchw) return store4(dx + o, s, ov, g.c - n);
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (n + j < g.c) dx[o + (size_t) j * g.h * g.w] = s[j];
    }
    __device__ float *out_row(int m) const {   // NCHW dx: channel 0
        size_t o;
        return out_index(m, 0, o) ? dx + o : nullptr;
    }
    __device__ void put(float *row, int n, float s) const {
        if (row && n < g.c) row[(size_t) n * g.h * g.w] = s;
    }
    __device__ void finish(int m, int n, float s) const {
        size_t o;
        if (out_index(m, n, o)) dx[o] = s;
    }
};

// Tiles of BM x BN outputs per 128-thread CTA, TM x TN per thread. Large thread tiles need fewer
// shared-memory loads per multiply-add: 16 x 8 (two CTAs per SM) runs the bare inner loop at 66-69 of
// 77 TFLOP/s, 8 x 8 at 61-64, 8 x 4 at 59-62. 128 x 128 tiles for large problems; 64 x 64 where those would
// leave SMs idle, compute padding columns or have short reductions (four CTAs per SM hide each other's
// start and end); 128 x 32 for operations with at most 32 columns.
template <int BM_, int BN_, int TM_, int TN_, int CTAS_>
struct Tile {
    static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_;
    static constexpr int NT = (BM / TM) * (BN / TN);       // threads
    static constexpr int CTAS = CTAS_;                     // resident per SM (register bound)
    static constexpr int TX = BN / TN;                     // compute threads along n
    static_assert(TX % 8 == 0 && TM % 4 == 0 && TN % 4 == 0, "warps cover 4 x 8 threads, threads runs of 4");
    static_assert(BM % 32 == 0 && BN % 32 == 0 && BK % (NT / 32) == 0, "loader: whole warps per reduction index");
    static constexpr size_t S_BYTES = sizeof(float) * BM * BN;   // running sum of completed KC blocks
};
using TileSquare = Tile<128, 128, 16, 8, 2>;
using TileSmall = Tile<64, 64, 8, 4, 4>;
using TileNarrow = Tile<128, 32, 8, 4, 4>;

// d = a * b + d on two FP32 lanes: each lane is the scalar fused multiply-add's result.
__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long both(float v) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
}
// Asynchronous copies into shared memory; `in` false: zeros, and the source is not read. It has to lie on the copy's
// own grid (4 or 16 bytes) all the same.
__device__ __forceinline__ void copy4(uint32_t dst, const float *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy16(uint32_t dst, const float *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ float lane_of(unsigned long long v, int i) {
    return __uint_as_float((uint32_t) (i ? v >> 32 : v));
}

// VEC (single-tap NHWC operations): the reduction indices of an A row are consecutive
// channels of one pixel, so each thread loads whole 4-index quads of its rows as 16-byte
// vectors instead of gathering element by element down a column.
// BV (B read from a layout with the tile's columns contiguous, N % 4 == 0, 16-byte aligned):
// each B row of a slice is loaded as BN/4 16-byte vectors.
//
// Otherwise warp w gathers the reduction indices w, w + 4 of a slice for rows / columns lane, lane + 32,
// ...: one table entry per index serves all of them, and each element costs a mask test, an address
// and a load.
//
// The inner product runs on packed pairs (fma.rn.f32x2: rows i, i + 1 of one column): operand
// registers of scalar multiply-adds collide in their banks (55 of 77 TFLOP/s for an 8 x 8 outer
// product held in registers, 70 packed), and half the issue slots are left for the loads.
template <class Op, class T, bool VEC, bool BV>
__global__ void __launch_bounds__(T::NT, T::CTAS) fp32_igemm_kernel(const __grid_constant__ Op op) {
    constexpr int NT = T::NT, TM = T::TM, TN = T::TN, NW = NT / 32;
    constexpr int PITCH = T::BM + (VEC ? 4 : 0);   // VEC stores columns of As: spread over the banks
    __shared__ __align__(16) float As[2][BK][PITCH];
    __shared__ __align__(16) float Bs[2][BK][T::BN];
    // Reduction-index table: the r part of every gather, for two chunks of NT
    // consecutive r; chunk c + 1 is filled while the slices of chunk c run.
    __shared__ typename Op::REnt Rt[2][NT];
    extern __shared__ float Ssm[];  // [TM * TN][NT], running sum of completed KC blocks
    constexpr int SLICES = NT / BK;  // slices per table chunk

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int m0 = blockIdx.x * T::BM;
    const int n0 = blockIdx.y * T::BN;
    const int z = blockIdx.z;
    int rbeg, rend;
    op.range(m0, z, rbeg, rend);
    // Pixels of a stride phase that no tap reaches: an accumulating call leaves them as they are (56 x 56, 256 -> 512 1 x 1
    // stride 2, batch 64: 848 -> 477 us; 256 -> 128: 530 -> 180)
    if (op.starts() && rbeg >= rend) return;
    Rt[0][tid] = op.rent(rbeg + tid, rend);
    Rt[1][tid] = op.rent(rbeg + NT + tid, rend);

    // loader mapping (see above)
    constexpr int KPW = BK / NW;                                // reduction indices per warp and slice
    constexpr int AR = T::BM / 32, BC = T::BN / 32;             // rows / columns per lane
    constexpr int QA = BK / 4, VI = QA * T::BM / NT;            // VEC: quads per row, quads per thread
    constexpr int QB = T::BN / 4, BI = BK * QB / NT;            // BV: quads per B row, per thread
    static_assert(!VEC || NT % QA == 0, "VEC: a thread keeps its quad");
    static_assert(!BV || (NT % QB == 0 && BI >= 1), "BV: a thread keeps its columns");
    typename Op::Row arow[VEC ? 1 : AR];
    const float *vsrc[VEC ? VI : 1];
    if constexpr (VEC) {
#pragma unroll
        for (int i = 0; i < VI; i++) vsrc[i] = op.vrow(op.row(m0 + (tid + NT * i) / QA));
    } else {
#pragma unroll
        for (int i = 0; i < AR; i++) arow[i] = op.row(m0 + lane + 32 * i);
    }
    typename Op::Col bcol[BV ? 1 : BC];
    if constexpr (BV) {
        bcol[0] = op.col(n0 + 4 * (tid % QB));
    } else {
#pragma unroll
        for (int i = 0; i < BC; i++) bcol[i] = op.col(n0 + lane + 32 * i);
    }
    float4 ra[VEC ? VI : 1];
    const uint32_t sA = (uint32_t) __cvta_generic_to_shared(&As[0][0][0]);
    const uint32_t sB = (uint32_t) __cvta_generic_to_shared(&Bs[0][0][0]);

    // compute mapping: a warp covers 4 x 8 threads; rows {ty*4 + i%4 + i/4 * BM/GM}, columns likewise
    constexpr int WX = T::TX / 8, GM = TM / 4, GN = TN / 4;
    const int tx = warp % WX * 8 + lane % 8, ty = warp / WX * 4 + lane / 8;
    auto mrow = [&](int i) { return m0 + (i / 4) * (T::BM / GM) + ty * 4 + i % 4; };
    auto ncol = [&](int j) { return n0 + (j / 4) * (T::BN / GN) + tx * 4 + j % 4; };

    // The running sum starts at 0 without being written (none = true), or at dx when accumulating. Loops
    // over it are rolled: unrolled 128 times they are tens of KB of code run once per CTA, and
    // short reductions then spend their time on instruction fetches.
    bool none = !op.starts();
    if (!none) {   // eight loads in flight (one by one, a 64 x 64 tile's 32 per thread took 9 us)
#pragma unroll 1
        for (int e = 0; e < TM * TN; e += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = op.s_init(mrow((e + j) / TN), ncol((e + j) % TN));
#pragma unroll
            for (int j = 0; j < 8; j++) Ssm[(e + j) * NT + tid] = v[j];
        }
    }

    unsigned long long acc[TM / 2][TN];   // rows 2i, 2i + 1
#pragma unroll
    for (int i = 0; i < TM / 2; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0ull;

    auto fold = [&]() {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) {
                float *s = &Ssm[(i * TN + j) * NT + tid];
                *s = __fadd_rn(none ? 0.0f : *s, lane_of(acc[i / 2][j], i & 1));
            }
        none = false;
#pragma unroll
        for (int i = 0; i < TM / 2; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) acc[i][j] = 0ull;
    };

    // slice t into buffer t & 1: asynchronous copies (VEC: the A quads through registers, stored by
    // vstore after the current slice's arithmetic)
    auto load = [&](int t) {
        const int rr = t * BK;   // slices never straddle a chunk: NT % BK == 0
        const typename Op::REnt *rt = Rt[(rr / NT) & 1] + rr % NT;
        const uint32_t a0 = sA + (t & 1) * (uint32_t) sizeof(As[0]), b0 = sB + (t & 1) * (uint32_t) sizeof(Bs[0]);
        if constexpr (VEC) {
            const int r = rbeg + rr + 4 * (tid % QA);
#pragma unroll
            for (int i = 0; i < VI; i++) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (const float *src = vsrc[i]) {
                    if (r + 3 < rend) {
                        v = __ldg(reinterpret_cast<const float4 *>(src + r));
                    } else {
                        if (r < rend) v.x = __ldg(src + r);
                        if (r + 1 < rend) v.y = __ldg(src + r + 1);
                        if (r + 2 < rend) v.z = __ldg(src + r + 2);
                    }
                }
                ra[i] = v;
            }
        } else {
#pragma unroll
            for (int k = 0; k < KPW; k++) {
                const typename Op::REnt e = rt[warp + NW * k];
#pragma unroll
                for (int i = 0; i < AR; i++)
                    copy4(a0 + 4 * ((warp + NW * k) * PITCH + lane + 32 * i), op.asrc(arow[i], e), op.ain(arow[i], e));
            }
        }
        if constexpr (BV) {
#pragma unroll
            for (int i = 0; i < BI; i++) {
                const int kk = (tid + NT * i) / QB;
                const auto bd = rt[kk].bd;   // -1 past the range
                const bool in = op.bin(bcol[0], bd);
                copy16(b0 + 4 * (kk * T::BN + 4 * (tid % QB)), in ? bcol[0].p + bd : op.bbase(), in);
            }
        } else {
#pragma unroll
            for (int k = 0; k < KPW; k++) {
                const auto bd = rt[warp + NW * k].bd;
#pragma unroll
                for (int i = 0; i < BC; i++)
                    copy4(b0 + 4 * ((warp + NW * k) * T::BN + lane + 32 * i), bcol[i].p + bd, op.bin(bcol[i], bd));
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto vstore = [&](int t) {
        if constexpr (VEC) {
#pragma unroll
            for (int i = 0; i < VI; i++) {
                const int row = (tid + NT * i) / QA, k0 = 4 * (tid % QA);
                As[t & 1][k0][row] = ra[i].x;
                As[t & 1][k0 + 1][row] = ra[i].y;
                As[t & 1][k0 + 2][row] = ra[i].z;
                As[t & 1][k0 + 3][row] = ra[i].w;
            }
        }
    };
    auto arrived = [&]() { asm volatile("cp.async.wait_group 0;" ::: "memory"); };
    auto step = [&](int buf, int kk) {
        unsigned long long av[TM / 2];
        float bv[TN];
#pragma unroll
        for (int q = 0; q < GM; q++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(&As[buf][kk][q * (T::BM / GM) + ty * 4]);
            av[2 * q] = v.x;
            av[2 * q + 1] = v.y;
        }
#pragma unroll
        for (int q = 0; q < GN; q++) {
            const float4 v = *reinterpret_cast<const float4 *>(&Bs[buf][kk][q * (T::BN / GN) + tx * 4]);
            bv[4 * q] = v.x;
            bv[4 * q + 1] = v.y;
            bv[4 * q + 2] = v.z;
            bv[4 * q + 3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const unsigned long long bb = both(bv[j]);
#pragma unroll
            for (int i = 0; i < TM / 2; i++) fma2(acc[i][j], av[i], bb);
        }
    };

    const int ntiles = (rend - rbeg + BK - 1) / BK;
    int next_fold = op.next_fold(rbeg, rend);
    __syncthreads();
    load(0);
    vstore(0);
    arrived();
    __syncthreads();
    for (int t = 0; t < ntiles; t++) {
        const int buf = t & 1;
        if (t > 0 && t % SLICES == 0) {
            // chunk c + 1 replaces chunk c - 1, whose last reader (the loads of that chunk's last
            // slice, issued one slice earlier) is behind two barriers
            const int c = t / SLICES + 1;
            Rt[c & 1][tid] = op.rent(rbeg + c * NT + tid, rend);
        }
        if (t + 1 < ntiles) load(t + 1);   // its buffer's readers are behind the last barrier
        const int r0 = rbeg + t * BK;
        if (next_fold >= r0 + BK) {
#pragma unroll
            for (int kk = 0; kk < BK; kk++) step(buf, kk);
        } else {
#pragma unroll 1
            for (int kk = 0; kk < BK; kk++) {
                if (r0 + kk == next_fold) {
                    fold();
                    next_fold = op.next_fold(r0 + kk, rend);
                }
                step(buf, kk);
            }
        }
        if (t + 1 < ntiles) vstore(t + 1);
        arrived();
        __syncthreads();
    }
    if (ntiles > 0) {
        fold();
    } else if (none) {   // an empty range leaves the start value as it is
#pragma unroll 1
        for (int e = 0; e < TM * TN; e++) Ssm[e * NT + tid] = 0.0f;
    }

    if (op.by_rows()) {
#pragma unroll 1
        for (int e = 0; e < GM * TN; e++) {   // rows mrow(4g) .. mrow(4g) + 3 are consecutive
            const int g = e / TN, j = e % TN;
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = Ssm[((4 * g + i) * TN + j) * NT + tid];
            op.finish_m4(mrow(4 * g), ncol(j), v);
        }
        return;
    }
    if (op.by_column()) {   // NCHW rows that are no vectors: a warp stores 32 rows of one column at a time
        __syncthreads();
        constexpr int RG = T::BM / GM, CG = T::BN / GN;   // rows / columns between a thread's runs of four
#pragma unroll 1
        for (int rb = 0; rb < T::BM / 32; rb++) {
            const int row = 32 * rb + lane, i = row / RG * 4 + row % 4, ry = row % RG / 4;
            float *out = op.out_row(m0 + row);   // the row's place is found once
#pragma unroll 4
            for (int col = warp; col < T::BN; col += NW) {
                const int j = col / CG * 4 + col % 4, cx = col % CG / 4;
                const int t = (ry / 4 * WX + cx / 8) * 32 + ry % 4 * 8 + cx % 8;   // the thread that holds it
                op.put(out, n0 + col, Ssm[(i * TN + j) * NT + t]);
            }
        }
        return;
    }
#pragma unroll 1
    for (int e = 0; e < TM * GN; e++) {   // columns ncol(4q) .. ncol(4q) + 3 are consecutive
        const int i = e / GN, q = e % GN;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = Ssm[(i * TN + q * 4 + j) * NT + tid];
        op.finish_z4(z, mrow(i), ncol(4 * q), v);
    }
}

// Block split: out(m, n) = finish(((start + ws[0]) + ws[1]) + ...), the planes in segment order
// (start: 0, or dx for the accumulating input gradient).
template <class Op>
__global__ void fp32_split_reduce_kernel(const __grid_constant__ Op op, int nz, int M, int N) {
    const long long total = (long long) M * N;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x) {
        const int m = (int) (i / N), n = (int) (i % N);
        float s = op.s_start(m, n);
        const int nzr = op.zcount(m, nz);
        int z = 0;
        for (; z + 8 <= nzr; z += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = op.ws[(size_t) (z + j) * total + i];
#pragma unroll
            for (int j = 0; j < 8; j++) s = __fadd_rn(s, v[j]);
        }
        for (; z < nzr; z++) s = __fadd_rn(s, op.ws[(size_t) z * total + i]);
        op.finish(m, n, s);
    }
}
// The same for N % 4 == 0: four neighbouring columns per thread, 16-byte plane reads (the planes are
// 16-byte aligned).
template <class Op>
__global__ void fp32_split_reduce4_kernel(const __grid_constant__ Op op, int nz, int M, int N) {
    const long long total = (long long) M * N / 4;
    const float4 *ws = reinterpret_cast<const float4 *>(op.ws);
    const int N4 = N / 4;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x) {
        const int m = (int) (i / N4), n = 4 * (int) (i % N4);
        float s[4];
#pragma unroll
        for (int c = 0; c < 4; c++) s[c] = op.s_start(m, n + c);
        const int nzr = op.zcount(m, nz);
        auto add = [&](const float4 &v) {
            s[0] = __fadd_rn(s[0], v.x);
            s[1] = __fadd_rn(s[1], v.y);
            s[2] = __fadd_rn(s[2], v.z);
            s[3] = __fadd_rn(s[3], v.w);
        };
        int z = 0;
        for (; z + 4 <= nzr; z += 4) {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = ws[(size_t) (z + j) * total + i];
#pragma unroll
            for (int j = 0; j < 4; j++) add(v[j]);
        }
        for (; z < nzr; z++) add(ws[(size_t) z * total + i]);
        op.finish_n4(m, n, s);
    }
}

// dW(m, n) = ((ws[0] + ws[1]) + ws[2]) + ... : the reference's block order.
__global__ void wgrad_reduce_kernel(const float *__restrict__ ws, float *__restrict__ dw, int K, int kn,
                                    int nblocks, int nchw) {
    const long long total = (long long) K * kn;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < total;
         i += (long long) gridDim.x * blockDim.x) {
        // loads eight blocks ahead, adds strictly in block order
        float s = ws[i];
        int z = 1;
        for (; z + 8 <= nblocks; z += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = ws[(size_t) (z + j) * total + i];
#pragma unroll
            for (int j = 0; j < 8; j++) s = __fadd_rn(s, v[j]);
        }
        for (; z < nblocks; z++) s = __fadd_rn(s, ws[(size_t) z * total + i]);
        const int m = (int) (i / kn), n = (int) (i % kn);
        dw[nchw ? ((size_t) n * K + m) : (size_t) i] = s;
    }
}

template <class Op, class T, bool VEC, bool BV>
cudaError_t launch_tile(const Op &op, int gz, cudaStream_t st) {
    static bool attr_set = false;  // per template instance; harmless if set twice
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(fp32_igemm_kernel<Op, T, VEC, BV>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int) T::S_BYTES);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    dim3 grid((op.M() + T::BM - 1) / T::BM, (op.N() + T::BN - 1) / T::BN, gz);
    if (grid.x == 0 || grid.y == 0) return cudaSuccess;
    fp32_igemm_kernel<Op, T, VEC, BV><<<grid, T::NT, T::S_BYTES, st>>>(op); cg_note_launch();
    return cudaGetLastError();
}

enum { TILE_SQUARE, TILE_SMALL, TILE_NARROW };

template <class Op, bool VEC, bool BV>
cudaError_t launch_shape(const Op &op, int tile, int gz, cudaStream_t st) {
    return tile == TILE_SMALL ? launch_tile<Op, TileSmall, VEC, BV>(op, gz, st)
           : tile == TILE_NARROW ? launch_tile<Op, TileNarrow, VEC, BV>(op, gz, st)
                                 : launch_tile<Op, TileSquare, VEC, BV>(op, gz, st);
}

// vec: A rows as channel vectors (single-tap NHWC forward / input gradient), taken together
// with bv (B rows as 16-byte vectors), which the same layouts allow.
template <template <bool> class Op, bool BIG>
cudaError_t launch(const Op<BIG> &op, int tile, int gz, bool vec, bool bv, cudaStream_t st) {
    if constexpr (!BIG && !std::is_same<Op<false>, WgradOp<false>>::value) {   // (a filter beyond the tap masks has many taps)
        if (vec && bv) return launch_shape<Op<BIG>, true, true>(op, tile, gz, st);
    }
    return bv ? launch_shape<Op<BIG>, false, true>(op, tile, gz, st)
              : launch_shape<Op<BIG>, false, false>(op, tile, gz, st);
}
inline bool big_filter(const cg_shape &s) { return s.kh > MASK_TAPS || s.kw > MASK_TAPS; }

inline bool aligned16(const void *p) { return ((uintptr_t) p & 15) == 0; }

// Gathers add 32-bit offsets within one image and within the weights.
inline bool offsets_fit(const ConvGeom &g) {
    const long long lim = INT_MAX / 2;
    return (long long) g.c * g.h * g.w < lim && (long long) g.kn * g.ho * g.wo < lim &&
           (long long) g.K * g.kn < lim;
}

// Library-owned scratch, one grow-only buffer per (device, stream, purpose): a CUDA graph
// that captured a buffer keeps using it, so buffers are never freed or reused for another
// stream.  Purposes: the block split's planes, an operand copy in the kernel's gather layout
// (activation; a second one where a call copies two), a repacked weight tensor.
enum { SLOT_SPLIT = 0, SLOT_ACT = 1, SLOT_WGT = 2, SLOT_ACT2 = 3 };
constexpr size_t SLOT_MAX[4] = {(size_t) 256 << 20, (size_t) 4 << 30, (size_t) 256 << 20, (size_t) 4 << 30};
std::mutex g_scratch_mu;
std::map<std::tuple<int, cudaStream_t, int>, std::pair<float *, size_t>> g_scratch;

float *scratch(int slot, size_t bytes, cudaStream_t st) {
    if (bytes == 0 || bytes > SLOT_MAX[slot]) return nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    auto &e = g_scratch[std::make_tuple(dev, st, slot)];
    if (e.second >= bytes) return e.first;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return nullptr;   // no allocation under capture: the form without scratch runs instead
    }
    size_t want = e.second ? e.second : ((size_t) 32 << 20);
    while (want < bytes) want *= 2;
    if (want > SLOT_MAX[slot]) want = SLOT_MAX[slot];
    float *p = nullptr;
    if (cudaMalloc(&p, want) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    e = {p, want};   // the previous buffer stays allocated for graphs that captured it
    return p;
}

// dst[b][c][r] = src[b][r][c] through 64 x 64 shared-memory tiles, both sides coalesced: sixteen loads in
// flight per thread, as 16-byte vectors where the layout allows (C or R a multiple of 4 and the
// pointer aligned).
__global__ void __launch_bounds__(256) transpose_kernel(const float *__restrict__ src, float *__restrict__ dst, int R, int C,
                                                        int vr, int vw) {
    __shared__ float t[64][65];
    const size_t off = (size_t) blockIdx.z * R * C;
    const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64, tid = threadIdx.x;
    src += off;
    dst += off;
    if (vr) {
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int r = r0 + tid / 16 + 16 * k, c = c0 + 4 * (tid % 16);
            if (r < R && c < C) v[k] = __ldg(reinterpret_cast<const float4 *>(src + (size_t) r * C + c));
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
            const int r = r0 + tid / 64 + 4 * k, c = c0 + tid % 64;
            if (r < R && c < C) v[k] = __ldg(src + (size_t) r * C + c);
        }
#pragma unroll
        for (int k = 0; k < 16; k++) t[tid / 64 + 4 * k][tid % 64] = v[k];
    }
    __syncthreads();
    if (vw) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int c = tid / 16 + 16 * k, r = 4 * (tid % 16);
            if (c0 + c < C && r0 + r < R)
                *reinterpret_cast<float4 *>(dst + (size_t) (c0 + c) * R + r0 + r) =
                    make_float4(t[r][c], t[r + 1][c], t[r + 2][c], t[r + 3][c]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int c = tid / 64 + 4 * k, r = tid % 64;
            if (c0 + c < C && r0 + r < R) dst[(size_t) (c0 + c) * R + r0 + r] = t[r][c];
        }
    }
}

// A transposed copy of src ([batch][R][C] -> [batch][C][R]) in the given scratch slot, or NULL
// when there is no room (or the grid would not fit); the caller then reads src as it is.
const float *transposed(int slot, const float *src, long long batch, long long R, long long C, cudaStream_t st) {
    const long long gy = (R + 63) / 64, gx = (C + 63) / 64;
    if (batch < 1 || batch > 65535 || gy > 65535 || gx > INT_MAX) return nullptr;
    float *dst = scratch(slot, sizeof(float) * (size_t) (batch * R * C), st);
    if (!dst) return nullptr;
    transpose_kernel<<<dim3((unsigned) gx, (unsigned) gy, (unsigned) batch), 256, 0, st>>>(
        src, dst, (int) R, (int) C, C % 4 == 0 && aligned16(src), R % 4 == 0);
    cg_note_launch();
    if (cudaGetLastError() != cudaSuccess) return nullptr;
    return dst;
}

inline int num_sms() {
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 152;
}

// Estimated seconds of n tiles of R reduction steps each on the SM with the most of them. It runs `ctas`
// at a time; fewer resident CTAs leave latencies uncovered, so they run at eff[resident - 1] of the FMA
// rate. A tile's start and end cost about `ov` more steps and `begin` microseconds a round, adding a segment to the
// running sum `fold`, the rows of a stride-phase tile, whose places are found one by one, `phase`. Fitted to 20 shapes
// (0.01 to 118 GFLOP) with each tile forced, the microseconds to 170 forwards and input gradients with every tile, fused
// and split (0.5% off the best on average; 5% for input gradients without them: 14 x 14, 34 -> 22 5 x 5 stride 2, batch 34
// fused 55 us, split 41). 128 x 128 takes 2.10 ms where 64 x 64 takes 2.35 (56 x 56, 256 -> 256, 3 x 3, batch 32),
// 223 us against 206 (56 x 56, 64 -> 256, 1 x 1, batch 64), 68 us against 28 (28 x 28, 64 -> 64, batch 8).
struct TileCost {
    int bm, bn, ctas, ov;
    double eff[4];
    double begin, fold, phase;
};
constexpr TileCost TILE_COST[3] = {{128, 128, 2, 60, {0.58, 0.74, 0, 0}, 1.9, 1.7, 37.0},
                                   {64, 64, 4, 40, {0.38, 0.50, 0.57, 0.63}, 0.7, 1.0, 12.0},
                                   {128, 32, 4, 40, {0.38, 0.50, 0.57, 0.63}, 2.3, 1.1, 13.0}};

inline double tile_time(const TileCost &c, long long n, double R, int segs, bool phased, int sms) {
    const long long per_sm = (n + sms - 1) / sms;
    const double one = (double) c.bm * c.bn * (R + c.ov) / 128 / 2.0e9;   // 128 multiply-adds per cycle, about 2 GHz
    const long long rounds = per_sm / c.ctas, rest = per_sm % c.ctas;
    const double adds = (double) (rounds + (rest > 0)) * (c.begin + c.fold * (segs - 1) + (phased ? c.phase : 0.0)) * 1e-6;
    return one * (rounds * c.ctas / c.eff[c.ctas - 1] + (rest ? rest / c.eff[rest - 1] : 0.0)) + adds;
}

// The cheapest tile shape for M x N outputs, nz chains of `segs` segments, R steps in all, per output; *cost: its estimate.
inline int pick_tile(long long M, long long N, int nz, double R, int segs, bool phased, double *cost) {
    const int sms = num_sms();
    int best = TILE_SQUARE;
    *cost = -1.0;
    for (int t = 0; t < 3; t++) {
        if (t == TILE_NARROW && N > 32) continue;
        const TileCost &c = TILE_COST[t];
        const double v = tile_time(c, ((M + c.bm - 1) / c.bm) * ((N + c.bn - 1) / c.bn) * nz, R, segs, phased, sms);
        if (*cost < 0 || v < *cost) {
            *cost = v;
            best = t;
        }
    }
    return best;
}

// The tile shape, and whether to run one CTA per reduction segment: the split pays when
// the fused grid leaves SMs idle or ends in a thin last wave, weighed against the planes it
// writes and reads back (2 x bytes at about 4 TB/s, plus the reduction's launch).
template <class Op>
cudaError_t launch_split_or_fused(Op op, int M, int N, bool vec, bool bv, cudaStream_t st) {
    const int nz = op.segments();
    const size_t bytes = sizeof(float) * (size_t) nz * (size_t) M * (size_t) N;
    const double R = (double) op.rlen();
    op.ws = nullptr;
    double cost;
    int tile = pick_tile(M, N, 1, R, nz, op.phased(), &cost);
    if (nz > 1) {
        double c2;
        const int t2 = pick_tile(M, N, nz, R / nz, 1, false, &c2);
        if (c2 + 2.0 * (double) bytes / 4e12 + 10e-6 < cost) {
            op.ws = scratch(SLOT_SPLIT, bytes, st);
            if (op.ws) tile = t2;
        }
    }
    if (!op.ws) return launch(op, tile, 1, vec, bv, st);
    cudaError_t e = launch(op, tile, nz, vec, bv, st);
    if (e != cudaSuccess) return e;
    const long long total = (long long) M * N;
    const bool v4 = N % 4 == 0;
    const int blocks = (int) std::min<long long>((total / (v4 ? 4 : 1) + 255) / 256, (long long) num_sms() * 16);
    if (v4) fp32_split_reduce4_kernel<Op><<<blocks, 256, 0, st>>>(op, nz, M, N);
    else fp32_split_reduce_kernel<Op><<<blocks, 256, 0, st>>>(op, nz, M, N);
    cg_note_launch();
    return cudaGetLastError();
}

// A call's launches (operand copies, the kernel, the plane reduction) are enqueued under one
// lock: the copies live in per-stream scratch, so two host threads enqueueing on the same
// stream must not interleave one call's copy between another call's copy and its kernel.
std::mutex g_call_mu;

}  // namespace

namespace {

// Operand layouts the kernel reads (the arithmetic and its order do not depend on them):
// a k x k NHWC forward reads x from an NCHW copy (a column of A, 128 output pixels at one
// reduction index, is then 128 consecutive floats instead of 128 pixels c floats apart);
// a single-tap NHWC forward reads x rows as 16-byte channel vectors; an NCHW forward reads
// its weights as [K][kn] (a row of B contiguous).
template <bool BIG>
cudaError_t fwd_call(int nchw, const cg_shape &s, const float *w, const float *x, float *y, const cg_epi &e,
                     cudaStream_t st) {
    FwdOp<BIG> op;
    op.g = make_geom(s);
    if (!offsets_fit(op.g)) return cudaErrorNotSupported;
    op.nchw = nchw;
    op.xl = op.wl = nchw;
    op.w = w;
    op.x = x;
    op.y = y;
    op.e = e;
    op.dwo = FastDiv(op.g.wo);
    op.dho = FastDiv(op.g.ho);
    op.dkw = FastDiv(s.kw);
    op.dkh = FastDiv(s.kh);
    op.ws = nullptr;
    bool vec = false;
    if (!nchw) {
        if (s.kh == 1 && s.kw == 1) {
            vec = s.c % 4 == 0 && aligned16(x);
        } else if (const float *xt = transposed(SLOT_ACT, x, s.b, (long long) s.h * s.w, s.c, st)) {
            op.x = xt;
            op.xl = 1;
        }
    } else if (const float *wt = transposed(SLOT_WGT, w, 1, s.kn, op.g.K, st)) {
        op.w = wt;
        op.wl = 0;
    }
    op.mv = nchw && (op.g.ho * op.g.wo) % 4 == 0 && aligned16(y);
    op.ov = !nchw && s.kn % 4 == 0 && aligned16(y);
    const bool bv = op.wl == 0 && s.kn % 4 == 0 && aligned16(op.w);
    return launch_split_or_fused(op, (int) op.g.P, op.g.kn, vec, bv, st);
}

template <bool BIG>
cudaError_t wgrad_call(int nchw, const cg_shape &s, const float *dy, const float *x, float *dw, float *ws,
                       cudaStream_t st) {
    WgradOp<BIG> op;
    op.g = make_geom(s);
    if (!offsets_fit(op.g)) return cudaErrorNotSupported;
    op.xl = op.yl = nchw;
    op.dy = dy;
    op.x = x;
    op.ws = ws;
    op.dwo = FastDiv(op.g.wo);
    op.dho = FastDiv(op.g.ho);
    op.dkw = FastDiv(s.kw);
    op.dkh = FastDiv(s.kh);
    if (nchw) {
        // NCHW dy strides the tile's columns (output channels) by ho*wo: read an NHWC copy, and
        // for a single tap, whose rows are input channels, an NHWC copy of x as well
        if (const float *t = transposed(SLOT_ACT, dy, s.b, s.kn, (long long) op.g.ho * op.g.wo, st)) {
            op.dy = t;
            op.yl = 0;
        }
        if (s.kh * s.kw == 1)
            if (const float *t = transposed(SLOT_ACT2, x, s.b, s.c, (long long) s.h * s.w, st)) {
                op.x = t;
                op.xl = 0;
            }
    }
    const int nblocks = (int) ((op.g.P + KC - 1) / KC);
    double cost;
    const int tile = pick_tile(op.g.K, s.kn, nblocks, KC, 1, false, &cost);
    op.ov = s.kn % 4 == 0 && aligned16(ws);
    cudaError_t e = launch(op, tile, nblocks, false, op.yl == 0 && s.kn % 4 == 0 && aligned16(op.dy), st);
    if (e != cudaSuccess) return e;
    const long long total = (long long) op.g.K * op.g.kn;
    int blocks = (int) std::min<long long>((total + 255) / 256, 152LL * 16);
    wgrad_reduce_kernel<<<blocks, 256, 0, st>>>(ws, dw, op.g.K, op.g.kn, nblocks, nchw); cg_note_launch();
    return cudaGetLastError();
}

// Operand layouts as in the forward: a k x k NHWC input gradient reads dy from an NCHW copy,
// a single-tap NHWC one reads dy rows as channel vectors, and the weights are read as
// [tap][kn][c] (a row of B, consecutive input channels at one (tap, output channel), contiguous).
template <bool BIG>
cudaError_t dgrad_call(int nchw, const cg_shape &s, const float *w, const float *dy, float *dx, int accumulate,
                       cudaStream_t st) {
    DgradOp<BIG> op;
    op.g = make_geom(s);
    if (!offsets_fit(op.g)) return cudaErrorNotSupported;
    op.nchw = nchw;
    op.accumulate = accumulate;
    op.yl = op.wl = nchw;
    op.w = w;
    op.dy = dy;
    op.dx = dx;
    op.dw_ = FastDiv(s.w);
    op.dh_ = FastDiv(s.h);
    op.dkn = FastDiv(s.kn);
    op.dkw = FastDiv(s.kw);
    op.dvs = FastDiv(s.vstride);
    op.dhs = FastDiv(s.hstride);
    op.ws = nullptr;
    const int taps = s.kh * s.kw;
    const bool phased = (s.vstride > 1 || s.hstride > 1) && s.vstride * s.hstride <= DG_MAXCLS && taps <= DG_MAXTAPS;
    bool vec = false;
    if (!nchw) {
        if (taps == 1) {
            vec = s.kn % 4 == 0 && aligned16(dy);
        } else if (const float *t = transposed(SLOT_ACT, dy, s.b, (long long) op.g.ho * op.g.wo, s.kn, st)) {
            op.dy = t;
            op.yl = 1;
        }
    }
    // NHWC w is [c][tap*kn], NCHW w is [kn*c][tap]; both transpose to [tap][kn][c]
    const float *wt = nullptr;
    if (!nchw) wt = transposed(SLOT_WGT, w, 1, s.c, (long long) taps * s.kn, st);
    else if (taps > 1) wt = transposed(SLOT_WGT, w, 1, (long long) s.kn * s.c, taps, st);
    if (wt) {
        op.w = wt;
        op.wl = 2;
    } else if (nchw && taps == 1) {
        op.wl = 2;   // [kn][c] is [tap][kn][c] already
    }
    op.mv = nchw && (s.h * s.w) % 4 == 0 && aligned16(dx);
    op.ov = !nchw && s.c % 4 == 0 && aligned16(dx);
    const bool bv = op.wl == 2 && s.c % 4 == 0 && aligned16(op.w);
    if (!phased) return launch_split_or_fused(op, op.M(), op.g.c, vec, bv, st);

    DgradPhaseOp<BIG> po;
    po.g = op.g;
    po.nchw = nchw;
    po.accumulate = accumulate;
    po.yl = op.yl;
    po.wl = op.wl;
    po.ov = op.ov;
    po.w = op.w;
    po.dy = op.dy;
    po.dx = dx;
    po.dkn = FastDiv(s.kn);
    po.nkb = (s.kn + KC - 1) / KC;
    po.ws = nullptr;
    long long m = 0;
    int r = 0, t0 = 0, c = 0;
    for (int xm = 0; xm < s.vstride; xm++)
        for (int ym = 0; ym < s.hstride; ym++, c++) {
            DgPhase &p = po.ph[c];
            p.ih0 = ((xm - s.vpad) % s.vstride + s.vstride) % s.vstride;
            p.iw0 = ((ym - s.hpad) % s.hstride + s.hstride) % s.hstride;
            const int hc = p.ih0 < s.h ? (s.h - p.ih0 + s.vstride - 1) / s.vstride : 0;
            const int wc = p.iw0 < s.w ? (s.w - p.iw0 + s.hstride - 1) / s.hstride : 0;
            p.rows = s.b * hc * wc;
            p.dhc = FastDiv(hc > 0 ? hc : 1);
            p.dwc = FastDiv(wc > 0 ? wc : 1);
            p.mbeg = (int) m;
            p.rbeg = r;
            p.tap0 = t0;
            p.ntaps = 0;
            for (int kx = 0; kx < s.kh; kx++)
                for (int ky = 0; ky < s.kw; ky++)
                    if ((kx * s.vdil) % s.vstride == xm && (ky * s.hdil) % s.hstride == ym)
                        po.taps[t0 + p.ntaps++] = (unsigned char) (kx * s.kw + ky);
            t0 += p.ntaps;
            r += p.ntaps * s.kn;
            m += ((long long) p.rows + 255) / 256 * 256;
        }
    if (m > INT_MAX / 2) return cudaErrorNotSupported;
    po.ncls = c;
    po.mpad = (int) m;
    return launch_split_or_fused(po, po.mpad, s.c, vec && taps == 1, bv, st);
}

}  // namespace

cudaError_t cg_fp32_fwd(int nchw, const cg_shape &s, const float *w, const float *x, float *y,
                        const cg_epi &e, cudaStream_t st) {
    std::lock_guard<std::mutex> call_lock(g_call_mu);
    return big_filter(s) ? fwd_call<true>(nchw, s, w, x, y, e, st) : fwd_call<false>(nchw, s, w, x, y, e, st);
}

size_t cg_fp32_wgrad_ws_bytes(const cg_shape &s) {
    ConvGeom g = make_geom(s);
    long long nblocks = (g.P + KC - 1) / KC;
    return sizeof(float) * (size_t) nblocks * (size_t) g.K * (size_t) g.kn;
}

cudaError_t cg_fp32_wgrad(int nchw, const cg_shape &s, const float *dy, const float *x, float *dw, float *ws,
                          cudaStream_t st) {
    std::lock_guard<std::mutex> call_lock(g_call_mu);
    return big_filter(s) ? wgrad_call<true>(nchw, s, dy, x, dw, ws, st) : wgrad_call<false>(nchw, s, dy, x, dw, ws, st);
}

cudaError_t cg_fp32_dgrad(int nchw, const cg_shape &s, const float *w, const float *dy, float *dx, int accumulate,
                          cudaStream_t st) {
    std::lock_guard<std::mutex> call_lock(g_call_mu);
    return big_filter(s) ? dgrad_call<true>(nchw, s, w, dy, dx, accumulate, st)
                         : dgrad_call<false>(nchw, s, w, dy, dx, accumulate, st);
}
