// BF16 tensor-core implicit-GEMM convolution (sm_103a, tcgen05 + TMEM + TMA).
//
// One kernel serves the forward pass (sconvGemmNHWC 'N', src/convGemm.c:65-70)
// and the input gradient (sconvGemmNHWC_back, src/convGemm.c:82-97), which it
// computes in gather form: every input-gradient pixel collects the taps that
// reach it, so there is no col2im/row2im scatter (src/im2row_nhwc.c:231-267)
// and no atomics.  A stride > 1 input gradient is split into stride-phase
// classes (pixels with the same (ih + pad) mod stride see the same taps), each
// a dense implicit GEMM of its own; their tiles share one launch.
//
// GEMM view of one class: D[m, n] = sum_k A[m, k] * B[n, k]
//   m = output pixel of the class (128 per tile),
//   n = output channel (BN per tile, in TMEM columns),
//   k = tap * Cin + ci over the class's taps (64 per pipeline stage).
// A comes straight from the NHWC activation into the 128-byte-swizzled K-major
// layout the tensor core reads: by im2col-mode TMA (128 pixels x 64 channels of
// one tap per load, out-of-range taps and channels zero-filled), or by 16-byte
// cp.async gathers, zero-filled for padding, where channels are so few that
// whole K blocks per tap would mostly be zeros — no im2row buffer exists
// anywhere.  B is the packed weight matrix [Cout][K] loaded by TMA (as
// (channel, tap, Cout) boxes where a tap's last K block is partly zeros).  The
// FP32 accumulator lives in TMEM.
//
// The kernel is persistent: each CTA walks tiles blockIdx.x, +gridDim.x, ... (launches of few tiles: a
// cluster of 2 or 4 CTAs per tile, see TcConvParams::split)
// with two to four TMEM accumulators, so the epilogue of one tile runs while the
// MMAs of the next accumulate.  Warp roles (288 threads, 384 with EW = 8):
//   warps 0-3   load A and B (warp 0 by TMA; or all four warps gathering A);
//               stage ring of STAGES;
//   warps 4-    epilogue (EW = 4 or 8 warps): TMEM -> registers (tcgen05.ld),
//               scale/shift/ReLU, BF16, then either a 128-byte-swizzled
//               shared-memory tile and a TMA store (pixels contiguous in the
//               output), or whole rows (the strided pixels of a class);
//   warp 8 / 1  allocates TMEM, issues tcgen05.mma and the commits.
// The producer and MMA loops run by whole warps, an elected lane issuing each
// instruction, so that its operands are in uniform registers: issued by a single
// thread, every operand was moved there first, and that, not the tensor core or the
// loads, bounded the short K blocks (64-wide tiles 0.27 us per block, 0.18 so).
// What bounds it now: the tensor core at its operand-read rate on long reductions,
// the loads of x on short ones, and waves of tiles that do not fill the SMs.
#include <cuda_bf16.h>

#include "cg_common.cuh"
#include "tc_conv.h"
#include "tc_epi.cuh"
#include "tc_ptx.cuh"

namespace {

using bf16 = __nv_bfloat16;

// What the epilogue does beside scale, shift and ReLU (BF16 forms): nothing; masking by the activation of a ReLU (and
// adding the output's old values first); column sums of its output, masked when a mask is given (input
// gradient); column sums of its output and of the squares (forward); adding the output's old values, which take
// the mask's place in the parameters and its way into the staging buffer.
constexpr int EXTRA_NONE = 0, EXTRA_MASK = 1, EXTRA_SUMS = 2, EXTRA_STATS = 3, EXTRA_ACC = 4;

// Operand forms of the kernel.
constexpr int MODE_BF16 = 0;  // BF16 x BF16, kind::f16
constexpr int MODE_FP8 = 1;   // E4M3 x E4M3, kind::f8f6f4 (64-byte K rows, 64-byte swizzle)
constexpr int MODE_X3 = 2;    // 3xBF16: hi*hi + hi*lo + lo*hi into one accumulator, FP32 output
constexpr int MODE_FP8W = 3;  // E4M3 with 128-channel K blocks: 128-byte K rows, 128-byte swizzle

// KB 64-deep K blocks per pipeline stage: one full barrier and one MMA commit
// cover KB blocks (a barrier round trip costs ~400 cycles, a 128 x 64 x 64 block
// of BF16 MMAs ~150).
// MT 128-row M tiles share every weight tile: each K block loads MT activation
// tiles and one weight tile and issues MT MMAs into MT accumulators, which cuts
// the shared-memory bytes per FLOP (the operand delivery from L2 bounds the kernel).
// EW epilogue warps: 4 (one per TMEM lane quarter), or 8 (two per quarter, taking
// alternate 64-column chunks) for short-K tiles, whose time goes to the epilogue's
// latency chain (TMEM load, scale/shift, convert, staging) rather than the MMAs.
template <int BN, int STAGES, int KB = 1, int MODE = MODE_BF16, int MT = 1, int EW = 4>
struct TcCfg {
    static constexpr int BM = 128, BK = MODE == MODE_FP8W ? 128 : 64;   // K elements per block
    static constexpr int ROWB = MODE == MODE_FP8 ? 64 : 128;  // bytes of one K row of a block
    static constexpr int NOPS = MODE == MODE_X3 ? 2 : 1;      // hi / lo copies of each operand
    static constexpr uint32_t A_TILE = BM * ROWB;
    static constexpr uint32_t B_TILE = BN * ROWB;
    static constexpr uint32_t A_BLOCK = NOPS * A_TILE;
    static constexpr uint32_t B_BLOCK = NOPS * B_TILE;
    static constexpr uint32_t A_BYTES = KB * MT * A_BLOCK;
    static constexpr uint32_t B_BYTES = KB * B_BLOCK;
    static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr uint32_t SBO = 8 * ROWB;                  // 8-row swizzle atom
    static constexpr uint32_t LAYOUT = ROWB == 128 ? 2 : 4;    // SWIZZLE_128B / SWIZZLE_64B
    static constexpr bool OUTF32 = MODE == MODE_X3;
    static constexpr int CW = OUTF32 ? 32 : 64;                // output columns per 128-byte staging row
    static constexpr uint32_t EPI_BYTES = EW * 32 * 128;       // one 32-row x 128-byte chunk per epilogue warp
    // cp.async groups in flight per producer thread; the other STAGES - LAG slots let the
    // MMA run ahead of the arrivals (LAG = STAGES - 1 would lock the two in step)
    static constexpr int LAG = STAGES / 2;
    // shared tables: tap offsets, the class table, scale/shift (whole vectors up to 1024 channels)
    static constexpr size_t BAR_BYTES = 512;                   // mbarriers
    static constexpr size_t TAB_BYTES = TC_TAPTAB * 4 + TC_MAXCLS * 128 + 2 * 1024 * 4;
    // output staging buffers: two when they fit beside the stage ring, else one
    static constexpr int EPI_BUFS =
        (1024 + (size_t) STAGES * STAGE_BYTES + 2 * EPI_BYTES + BAR_BYTES + TAB_BYTES <= 232448) ? 2 : 1;
    static constexpr size_t SMEM = 1024 + (size_t) STAGES * STAGE_BYTES + EPI_BUFS * EPI_BYTES + BAR_BYTES + TAB_BYTES;
    static_assert(SMEM <= 232448, "shared memory above the 227 KB per-block limit");
    static_assert(EW == 4 || EW == 8, "four or eight epilogue warps");
    static_assert(BN != 64 || MT != 1 || (size_t) STAGES * STAGE_BYTES >= 3 * 128 * BN * 4, "a split tile's shares in the ring");
    // warps: 0 producer (0-3 on the cp.async path), 4..4+EW-1 epilogue, the MMA issuer in
    // warp 8 (EW = 4) or in the otherwise idle warp 1 (EW = 8)
    static constexpr int THREADS = EW == 8 ? 384 : 288;
    static constexpr int MMA_WARP = EW == 8 ? 1 : 8;
    static constexpr int NCH = BN / CW;   // output chunks of one accumulator
    // TMEM: MT accumulators of BN columns, double-buffered when 512 columns allow (four buffers
    // for tiles of <= 128 columns)
    static constexpr int ACC_BUFS = BN * MT <= 128 ? 4 : (2 * BN * MT <= 512 ? 2 : 1);
    static constexpr uint32_t TMEM_COLS = ACC_BUFS * BN * MT;
};

__device__ __forceinline__ uint64_t op_desc(uint32_t saddr, uint32_t sbo, uint32_t layout) {
    uint64_t d = tc::sw128_desc(saddr, 16, sbo);
    d &= ~((uint64_t) 7 << 61);
    return d | ((uint64_t) layout << 61);
}

// 0xFFFF in each half where the BF16 value is positive (not zero, not NaN).
__device__ __forceinline__ uint32_t positive_mask(uint32_t v) {
    return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162 *>(&v), __floats2bfloat162_rn(0.0f, 0.0f));
}

// A chunk of the warp's 32 accumulator rows: 64 columns as fragments (tc_epi.cuh), 32 columns of an FP32 output as a row per
// lane, whose 16-byte staging stores meet no bank twice as often as need be (8-byte ones of fragments do: 3xBF16, 54 x 54,
// 64 -> 256 1 x 1, batch 15: 15.1 us as fragments, 14.2 so).
template <bool F32>
__device__ __forceinline__ void acc_load(uint32_t ta, uint32_t (&v)[F32 ? 1 : 2][32]) {
    if constexpr (F32) {
        tc::tmem_ld_32x32b_x32(ta, v[0]);
        tc::tmem_ld_wait();
    } else {
        tc::frag_load(ta, v);
    }
}

template <int N>
__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"((uint64_t) map),
                 "r"(src), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

struct Tile {
    int cls, m0, n0;
};

// The scalars of a class, copied to shared memory at kernel start (reading the
// kernel parameters with a runtime class index would cost generic-memory loads
// on every tile).
struct ClsS {
    int Hg, Wg, oy0, ox0, osy, osx, isy, isx, iby, ibx, tap0, ntaps, kbeg, ktiles, tile0, lo_y, lo_x, mint_y, mint_x, gbase;
    FastDiv dwg, dhg;
};
static_assert(sizeof(ClsS) <= 128, "class table entry");

__device__ __forceinline__ Tile decode_tile(const ClsS *cls, int ncls, int ntiles, int bn, int t, int mt = 1) {
    int c = 0;
    while (c + 1 < ncls && t >= cls[c + 1].tile0) c++;
    const int local = t - cls[c].tile0;
    Tile tl;
    tl.cls = c;
    tl.m0 = (local / ntiles) * 128 * mt;
    tl.n0 = (local % ntiles) * bn;
    return tl;
}

template <int BN, int STAGES, int KB, bool IM2C, int MODE, int MT, int EW, int EXTRA>
__global__ void __launch_bounds__(EW == 8 ? 384 : 288, 1)
    tc_conv_kernel(const __grid_constant__ TcConvParams p, const __grid_constant__ CUtensorMap wmap,
                   const __grid_constant__ CUtensorMap omap, const __grid_constant__ TcMaps amaps) {
    using C = TcCfg<BN, STAGES, KB, MODE, MT, EW>;
    static_assert(EW == 4 || IM2C, "eight epilogue warps: im2col path");
    static_assert(EXTRA == EXTRA_NONE || (MODE == MODE_BF16 && C::EPI_BUFS == 2), "masks and sums: BF16, two staging buffers");
    // items of a tile: (accumulator mt, 64-column chunk). Eight warps: the two warps of a TMEM lane quarter
    // take alternate items, or alternate tiles where a tile has one item (each tile's accumulator is then
    // released by four warps)
    constexpr bool ALT = EW == 8 && MT * C::NCH == 1;
    constexpr int STEP = ALT ? 1 : EW / 4, TSTEP = ALT ? 2 : 1;
    // A tile covers p.nn <= BN output channels (a multiple of 16): the width that divides the channels into
    // equal tiles, so that 192 or 272 channels do not pay for 256 and 512. The last of its nch 64-column
    // chunks starts at nn - 64 and repeats columns of the one before (same values, stored twice).
    const int nn = p.nn, nch = (nn + C::CW - 1) / C::CW, NIT = MT * nch;
    auto chunk_col = [&](int chunk) { return max(0, min(chunk * C::CW, nn - C::CW)); };
    static_assert(IM2C || (KB == 1 && MODE == MODE_BF16), "the cp.async gather fills one BF16 K block per stage");
    static_assert(MT == 1 || (IM2C && MODE == MODE_BF16), "two M tiles per weight tile: BF16 im2col path only");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = (uint8_t *) (((uintptr_t) smem_raw + 1023) & ~(uintptr_t) 1023);
    uint8_t *epi_smem = base + STAGES * C::STAGE_BYTES;
    uint64_t *full = (uint64_t *) (epi_smem + C::EPI_BUFS * C::EPI_BYTES);
    uint64_t *empty = full + STAGES;
    uint64_t *acc_full = empty + STAGES;
    uint64_t *acc_empty = acc_full + 4;
    uint32_t *tmem_holder = (uint32_t *) (acc_empty + 4);
    uint64_t *mask_full = acc_empty + 5;   // [epilogue warp][staging buffer]
    static_assert((2 * STAGES + 9 + 2 * EW) * 8 <= C::BAR_BYTES, "mbarriers");
    // per-class tap offsets (packed y:16 | x:16) and the tile's epilogue scale/shift, in shared
    // memory: indexing the kernel parameters with runtime values would go through slow generic loads
    int32_t *tap_tab = (int32_t *) (epi_smem + C::EPI_BUFS * C::EPI_BYTES + C::BAR_BYTES);
    ClsS *cls_tab = (ClsS *) (tap_tab + TC_TAPTAB);
    float *sc_tab = (float *) (cls_tab + TC_MAXCLS);   // [1024]: all channels, or the tile's BN
    float *sh_tab = sc_tab + 1024;
    const bool sc_all = p.Cout <= 1024;              // whole scale/shift vectors fit

    const int warp = tc::w::warp_index(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            // im2col: the one expect_tx arrival; gather: 128 producer threads + the expect_tx
            tc::mbar_init(&full[s], IM2C ? 1 : 128 + 1);
            tc::mbar_init(&empty[s], 1);
        }
        if (EXTRA == EXTRA_MASK || EXTRA == EXTRA_SUMS || EXTRA == EXTRA_ACC)
            for (int b = 0; b < 2 * EW; b++) tc::mbar_init(&mask_full[b], 1);
        for (int b = 0; b < C::ACC_BUFS; b++) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], ALT ? 128 : 32 * EW);
        }
        tc::fence_mbar_init();
        tc::prefetch_tmap(&wmap);
        if (p.epi_tma) tc::prefetch_tmap(&omap);
        if (IM2C)
            for (int c = 0; c < p.ncls; c++) {
                tc::prefetch_tmap(&amaps.a[c]);
                if (MODE == MODE_X3) tc::prefetch_tmap(&amaps.b[c]);
            }
        if (MODE == MODE_X3) tc::prefetch_tmap(&amaps.wlo);
    }
    for (int i = threadIdx.x; i < TC_MAXTAPS; i += blockDim.x)
        tap_tab[i] = ((int32_t) p.toy[i] << 16) | ((int32_t) p.tox[i] & 0xFFFF);
    if (threadIdx.x < (unsigned) p.ncls) {
        const TcClass &c = p.cls[threadIdx.x];
        ClsS &d = cls_tab[threadIdx.x];
        d.Hg = c.Hg; d.Wg = c.Wg; d.oy0 = c.oy0; d.ox0 = c.ox0; d.osy = c.osy; d.osx = c.osx;
        d.isy = c.isy; d.isx = c.isx; d.iby = c.iby; d.ibx = c.ibx; d.tap0 = c.tap0; d.ntaps = c.ntaps; d.kbeg = c.kbeg;
        d.ktiles = c.ktiles; d.tile0 = c.tile0; d.lo_y = c.lo_y; d.lo_x = c.lo_x; d.mint_y = c.mint_y;
        d.mint_x = c.mint_x; d.gbase = c.gbase; d.dwg = c.dwg; d.dhg = c.dhg;
    }
    // everything above touched only shared memory and kernel parameters; the next kernel may
    // launch once every CTA has started its last tile (pdl_trigger in the producer loop), so
    // its waiting CTAs do not hold SMs that work on other streams could use
    tc::pdl_wait();
    if (sc_all)
        for (int n = threadIdx.x; n < p.Cout; n += blockDim.x) {
            sc_tab[n] = p.scale ? __ldg(p.scale + n) : 1.0f;
            sh_tab[n] = p.shift ? __ldg(p.shift + n) : 0.0f;
        }
    if (warp == C::MMA_WARP) {
        tc::tmem_alloc(tmem_holder, C::TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_holder;
    bool ok = true;
    // split reductions: CTA `krank` of the tile's cluster takes its share of the K blocks
    constexpr bool SPLITS = IM2C && MT == 1 && BN == 64;
    const int split = SPLITS ? p.split : 1, krank = split > 1 ? (int) blockIdx.x % split : 0;
    const int cta = split > 1 ? (int) blockIdx.x / split : (int) blockIdx.x;   // the first tile
    bool met = false;   // this thread has passed the cluster's two meetings

    if (IM2C && warp < 4 && warp != C::MMA_WARP) {
        // ------------------------------------------------ producer: one warp, im2col TMA for A, TMA for B
        if (warp == 0) {
            uint32_t it = 0;
            const uint32_t b_bytes = (uint32_t) (C::NOPS * nn * C::ROWB);
            for (int tile = cta; tile < p.ntiles_total && ok; tile += gridDim.x) {
                if (tile + (int) gridDim.x >= p.ntiles_total) tc::pdl_trigger();   // this CTA's last tile
                const Tile tl = decode_tile(cls_tab, p.ncls, p.ntiles, nn, tile, MT);
                const ClsS &cl = cls_tab[tl.cls];
                const int32_t *taps = tap_tab + cl.tap0;
                const int ktiles = __shfl_sync(0xFFFFFFFFu, cl.ktiles, 0), kbeg = cl.kbeg, mint_y = cl.mint_y, mint_x = cl.mint_x;
                int h0[MT], w0[MT], bb0[MT];   // im2col start of each M tile (beyond the class: zero-filled)
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    uint32_t q, jw, j, b;
                    cl.dwg.divmod(tl.m0 + mt * 128, q, jw);
                    cl.dhg.divmod(q, b, j);
                    h0[mt] = (int) j * cl.isy + cl.lo_y;
                    w0[mt] = (int) jw * cl.isx + cl.lo_x;
                    bb0[mt] = (int) b;
                }
                const CUtensorMap *am = &amaps.a[tl.cls];
                int tap = 0, ci0 = 0;   // k = tap*Cin + ci0, walked incrementally
                int k0 = 0, k1 = ktiles;
                if (split > 1) {
                    const int cpb = (p.Cin + C::BK - 1) / C::BK;
                    k0 = ktiles * krank / split;
                    k1 = ktiles * (krank + 1) / split;
                    tap = k0 / cpb;
                    ci0 = (k0 - tap * cpb) * C::BK;
                }
                for (int kt = k0; kt < k1; kt += KB, it++) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (it >= (uint32_t) STAGES && !(ok = tc::w::mbar_wait(&empty[s], ph ^ 1, p.err, 1))) break;
                    const int nkb = min(KB, k1 - kt);
                    const uint32_t sa = tc::smem_u32(base + s * C::STAGE_BYTES);
                    tc::w::mbar_arrive_expect_tx(&full[s], nkb * (MT * C::A_BLOCK + b_bytes));
                    for (int kb = 0; kb < nkb; kb++) {
                        const int32_t to = taps[tap];
                        const uint16_t offy = (uint16_t) ((to >> 16) - mint_y);
                        const uint16_t offx = (uint16_t) ((int32_t) (int16_t) (to & 0xFFFF) - mint_x);
                        const uint32_t ab = sa + kb * MT * C::A_BLOCK, bb = sa + C::A_BYTES + kb * C::B_BLOCK;
                        const int kcol = kbeg + (kt + kb) * C::BK;
#pragma unroll
                        for (int mt = 0; mt < MT; mt++)
                            tc::w::tma_load_im2col_4d(ab + mt * C::A_BLOCK, am, ci0, w0[mt], h0[mt], bb0[mt], offx, offy,
                                                   &full[s]);
                        if (MODE == MODE_BF16 && p.wtail) tc::w::tma_load_3d(bb, &amaps.b[tl.cls], ci0, tap, tl.n0, &full[s]);
                        else tc::w::tma_load_2d(bb, &wmap, kcol, tl.n0, &full[s]);
                        if (MODE == MODE_X3) {
                            tc::w::tma_load_im2col_4d(ab + C::A_TILE, &amaps.b[tl.cls], ci0, w0[0], h0[0], bb0[0], offx,
                                                   offy, &full[s]);
                            tc::w::tma_load_2d(bb + C::B_TILE, &amaps.wlo, kcol, tl.n0, &full[s]);
                        }
                        ci0 += C::BK;
                        if (ci0 >= p.Cin) {
                            ci0 = 0;
                            tap++;
                        }
                    }
                }
            }
        }
    } else if (!IM2C && warp < 4) {
        // ------------------------------------------------ producers: gather A, TMA B
        const int t = threadIdx.x;
        const int piece = t & 7;   // 16-byte piece of the 128-byte K row
        const int r0 = t >> 3;     // rows r0 + 16*i
        uint32_t it = 0;
        for (int tile = blockIdx.x; tile < p.ntiles_total && ok; tile += gridDim.x) {
            if (t == 0 && tile + (int) gridDim.x >= p.ntiles_total) tc::pdl_trigger();   // this CTA's last tile
            const Tile tl = decode_tile(cls_tab, p.ncls, p.ntiles, nn, tile);
            const ClsS &cl = cls_tab[tl.cls];
            const int32_t *taps = tap_tab + cl.tap0;
            const int M = p.B * cl.Hg * cl.Wg;
            int rb[8], ry[8], rx[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int m = tl.m0 + r0 + 16 * i;
                if (m < M) {
                    uint32_t q, jw, j, b;
                    cl.dwg.divmod(m, q, jw);
                    cl.dhg.divmod(q, b, j);
                    rb[i] = b;
                    ry[i] = (int) j * cl.isy + cl.iby;
                    rx[i] = (int) jw * cl.isx + cl.ibx;
                } else {
                    rb[i] = -1;
                    ry[i] = rx[i] = 0;
                }
            }
            for (int kt = 0; kt < cl.ktiles; kt++, it++) {
                const int s = it % STAGES;
                const uint32_t ph = (it / STAGES) & 1;
                if (it >= (uint32_t) STAGES) ok = tc::mbar_wait(&empty[s], ph ^ 1, p.err, 1);
                if (!ok) break;
                const int k = kt * C::BK + piece * 8;
                uint32_t tap, ci;
                p.dcin.divmod(k, tap, ci);
                const bool kval = (int) tap < cl.ntaps;
                const int32_t to = kval ? taps[tap] : 0;
                const int oy = to >> 16, ox = (int32_t) (int16_t) (to & 0xFFFF);
                const uint32_t sA = tc::smem_u32(base + s * C::STAGE_BYTES);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int r = r0 + 16 * i;
                    const int iy = ry[i] + oy, ix = rx[i] + ox;
                    const bool v =
                        kval && rb[i] >= 0 && (unsigned) iy < (unsigned) p.Hin && (unsigned) ix < (unsigned) p.Win;
                    const bf16 *src = v ? p.in + ((((size_t) rb[i] * p.Hin + iy) * p.Win + ix) * p.Cin + ci) : p.in;
                    tc::cp_async_16(sA + r * 128 + ((piece ^ (r & 7)) << 4), src, v ? 16u : 0u);
                }
                tc::cp_async_commit();
                if (t == 0) {
                    tc::mbar_arrive_expect_tx(&full[s], (uint32_t) (nn * C::ROWB));
                    tc::tma_load_2d(tc::smem_u32(base + s * C::STAGE_BYTES + C::A_BYTES), &wmap,
                                    cl.kbeg + kt * C::BK, tl.n0, &full[s]);
                }
                if (it >= (uint32_t) C::LAG) {
                    tc::cp_async_wait<C::LAG>();
                    tc::fence_proxy_async_smem();
                    tc::mbar_arrive(&full[(it - C::LAG) % STAGES]);
                }
            }
        }
        tc::cp_async_wait<0>();
        tc::fence_proxy_async_smem();
        if (ok)
            for (uint32_t j = (it > (uint32_t) C::LAG ? it - C::LAG : 0); j < it; j++) tc::mbar_arrive(&full[j % STAGES]);
    } else if (warp >= 4 && warp < 4 + EW) {
        // ------------------------------------------------ epilogue
        const int ew = (warp - 4) & 3;    // TMEM lane quarter (a warp reads lanes 32 * (warp % 4) ..)
        const int half = (warp - 4) >> 2; // EW = 8: which alternate items (ALT: tiles) this warp takes
        const int row = ew * 32 + lane;   // tile row = TMEM lane
        const int et = threadIdx.x - 128; // 0 .. 32 * EW - 1
        uint8_t *const stg_warp = epi_smem + (warp - 4) * 4096;   // this warp's 32 x 128-byte staging
        const int first_item = ALT ? 0 : half;
        const bool affine = p.scale || p.shift;
        uint32_t lt = ALT ? half : 0;     // local tile count
        int ebuf = 0;                     // staging buffer toggle
        // The mask's (or the output's old) 32 x 64 values of an item, loaded into the staging buffer the item will use: by TMA, or where
        // the rows are scattered (stride-phase classes) by 16-byte pieces, eight lanes to a row. (Read by
        // their own lanes, one cache line of another row per lane, the masked form of 56 x 56, 256 -> 64 took 60 us,
        // 27 without a mask.) The load is issued during the item before, off the critical path. Returns whether
        // the mask_full barrier will tell of its arrival.
        uint64_t *const mbar = mask_full + 2 * (warp - 4);
        auto prefetch_mask = [&](int tile, int item, int buf) {
            const Tile tl = decode_tile(cls_tab, p.ncls, p.ntiles, nn, tile, MT);
            const ClsS &cl = cls_tab[tl.cls];
            const int M = p.B * cl.Hg * cl.Wg;
            const int r0 = tl.m0 + (item / nch) * 128 + ew * 32, nb = tl.n0 + chunk_col(item % nch);
            const uint32_t dst = tc::smem_u32(stg_warp + buf * C::EPI_BYTES);
            if (p.epi_tma) {
                if (r0 >= M || nb >= p.Cout) return false;
                if (lane == 0) {
                    tc::mbar_arrive_expect_tx(&mbar[buf], 4096);
                    tc::tma_load_2d(dst, &amaps.mask, nb, r0, &mbar[buf]);
                }
                return true;
            }
            int pix = r0 + lane;
            uint32_t q, jw, j, b;
            cl.dwg.divmod(pix < M ? pix : 0, q, jw);
            cl.dhg.divmod(q, b, j);
            pix = ((int) b * p.Hout + cl.oy0 + cl.osy * (int) j) * p.Wout + cl.ox0 + cl.osx * (int) jw;
            const int ch = lane & 7;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int r = i * 4 + (lane >> 3);
                const int px = __shfl_sync(0xFFFFFFFFu, pix, r);
                const bool v = r0 + r < M && nb + ch * 8 < p.Cout;
                const __nv_bfloat16 *src = v ? p.mask + ((size_t) px * p.Cout + nb + ch * 8) : p.mask;
                tc::cp_async_16(dst + r * 128 + ((ch ^ (r & 7)) << 4), src, v ? 16u : 0u);
            }
            tc::cp_async_commit();
            return false;
        };
        constexpr bool MASKED = EXTRA == EXTRA_MASK || EXTRA == EXTRA_SUMS || EXTRA == EXTRA_ACC;
        bool by_tma = false;       // this item's mask arrives at mbar[ebuf]
        uint32_t mphase = 0;       // bit b: parity of the next arrival at mbar[b]
        if constexpr (MASKED) {
            const int t0 = cta + (int) (lt * gridDim.x);
            if (p.mask && t0 < p.ntiles_total && first_item < NIT && krank == 0) by_tma = prefetch_mask(t0, first_item, 0);
        }
        for (int tile = cta + (int) (lt * gridDim.x); tile < p.ntiles_total && ok; tile += TSTEP * gridDim.x, lt += TSTEP) {
            const Tile tl = decode_tile(cls_tab, p.ncls, p.ntiles, nn, tile, MT);
            const ClsS &cl = cls_tab[tl.cls];
            const int M = p.B * cl.Hg * cl.Wg;
            const int buf = lt % C::ACC_BUFS;
            const float *scp = sc_tab, *shp = sh_tab;
            if (sc_all) {
                scp += tl.n0;
                shp += tl.n0;
            } else {
                // this tile's scale/shift (the previous tile's readers passed the barrier below;
                // ALT: the two groups of warps keep their own copies)
                float *sc = sc_tab + (ALT ? half * 64 : 0), *sh = sh_tab + (ALT ? half * 64 : 0);
                if (ALT) tc::named_bar_sync(1 + half, 128);
                else epi_bar<32 * EW>();
                for (int j = ALT ? (et & 127) : et; j < BN; j += ALT ? 128 : 32 * EW) {
                    const int n = min(tl.n0 + j, p.Cout - 1);
                    sc[j] = p.scale ? __ldg(p.scale + n) : 1.0f;
                    sh[j] = p.shift ? __ldg(p.shift + n) : 0.0f;
                }
                if (ALT) tc::named_bar_sync(1 + half, 128);
                else epi_bar<32 * EW>();
                scp = sc;
                shp = sh;
            }
            ok = tc::mbar_wait(&acc_full[buf], (lt / C::ACC_BUFS) & 1, p.err, 3);
            tc::tc_fence_after();
            if constexpr (SPLITS) {
                if (split > 1) {
                    // the tile's only pass: the other CTAs' accumulators go to the first one's ring, which nothing uses
                    // any more, as [chunk][warp][four registers][lane]
                    met = true;
                    tc::cluster_meet();
                    if (krank > 0) {
                        const uint32_t dst = tc::mapa_shared(tc::smem_u32(base) + (uint32_t) ((krank - 1) * C::NCH * 4 * C::CW * 128), 0);
                        for (int ch = 0; ch < nch && ok; ch++) {
                            uint32_t v[C::CW / 32][32];
                            acc_load<C::OUTF32>(tmem + ((uint32_t) (ew * 32) << 16) + (uint32_t) (buf * BN + chunk_col(ch)), v);
#pragma unroll
                            for (int j = 0; j < C::CW / 4; j++) {
                                const uint32_t *w = &v[j / 8][j % 8 * 4];
                                asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                                                 dst + (uint32_t) (((ch * 4 + ew) * (C::CW / 4) + j) * 512 + lane * 16)),
                                             "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                                             : "memory");
                            }
                        }
                    }
                    tc::cluster_meet();
                    if (krank > 0) break;
                }
            }
            if (!ok) break;
            if (first_item >= NIT) {   // nothing for this warp in the tile: its share of the buffer is free
                tc::tc_fence_before();
                tc::mbar_arrive(&acc_empty[buf]);
            }
#pragma unroll 1
            for (int item = first_item; item < NIT; item += STEP) {
                const int mt = item / nch, c0 = chunk_col(item % nch);
                const int m0 = tl.m0 + mt * 128;   // this accumulator's first output row
                const int m = m0 + row;
                uint8_t *orow = nullptr;   // this row of the output (BF16, or FP32 for MODE_X3)
                if (!p.epi_tma && m < M) {
                    uint32_t q, jw, j, b;
                    cl.dwg.divmod(m, q, jw);
                    cl.dhg.divmod(q, b, j);
                    const int oy = cl.oy0 + cl.osy * (int) j, ox = cl.ox0 + cl.osx * (int) jw;
                    orow = (uint8_t *) p.out +
                           ((((size_t) b * p.Hout + oy) * p.Wout + ox) * p.Cout) * (C::OUTF32 ? 4 : 2);
                }
                constexpr int NQ = C::CW / 8;
                uint32_t v[C::CW / 32][32];
                acc_load<C::OUTF32>(tmem + ((uint32_t) (ew * 32) << 16) + (uint32_t) ((buf * MT + mt) * BN + c0), v);
                if constexpr (SPLITS) {
                    for (int o = 0; o < split - 1; o++) {   // the other shares of the sum, in order
                        const uint8_t *src = base + o * C::NCH * 4 * C::CW * 128 + (item * 4 + ew) * (C::CW / 4) * 512 + lane * 16;
#pragma unroll
                        for (int j = 0; j < C::CW / 4; j++) {
                            const uint4 u = *reinterpret_cast<const uint4 *>(src + j * 512);
                            uint32_t *w = &v[j / 8][j % 8 * 4];
                            w[0] = __float_as_uint(__uint_as_float(w[0]) + __uint_as_float(u.x));
                            w[1] = __float_as_uint(__uint_as_float(w[1]) + __uint_as_float(u.y));
                            w[2] = __float_as_uint(__uint_as_float(w[2]) + __uint_as_float(u.z));
                            w[3] = __float_as_uint(__uint_as_float(w[3]) + __uint_as_float(u.w));
                        }
                    }
                }
                if (item + STEP >= NIT) {
                    // this warp's last read of the accumulator: its share of the TMEM buffer
                    // goes back to the MMA warp
                    tc::tc_fence_before();
                    tc::mbar_arrive(&acc_empty[buf]);
                }
                const int nb = tl.n0 + c0;
                bool next_by_tma = false;
                if constexpr (MASKED) {
                    if (p.mask) {
                        if (by_tma) {
                            if (!(ok = tc::mbar_wait(&mbar[ebuf], mphase >> ebuf & 1, p.err, 5))) break;
                            mphase ^= 1u << ebuf;
                        } else {
                            tc::cp_async_wait<0>();
                        }
                        __syncwarp();
                        // the next item's mask goes to the other buffer, once the store of the item before
                        // this one has read it
                        int nt = tile, ni = item + STEP;
                        if (ni >= NIT) {
                            ni = first_item;
                            nt += TSTEP * gridDim.x;
                        }
                        if (nt < p.ntiles_total) {
                            if (lane == 0) bulk_wait_read<0>();
                            __syncwarp();
                            next_by_tma = prefetch_mask(nt, ni, ebuf ^ 1);
                        }
                    }
                }
                if constexpr (EXTRA == EXTRA_SUMS) {
                    if (p.mask) {   // rows past M arrived as zeros, which keep nothing
                        uint8_t *stg = stg_warp + ebuf * C::EPI_BYTES;
#pragma unroll
                        for (int q = 0; q < 8; q++)
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const uint32_t w = positive_mask(*reinterpret_cast<const uint32_t *>(tc::frag_word(stg, q, k)));
                                v[k >> 1][4 * q + 2 * (k & 1)] &= __byte_perm(w, 0, 0x1010);
                                v[k >> 1][4 * q + 2 * (k & 1) + 1] &= __byte_perm(w, 0, 0x3232);
                            }
                    }
                }
                if constexpr (EXTRA == EXTRA_ACC) {
                    // accumulate (the reference's dx += ...): add the output's old values in FP32
                    uint8_t *stg = stg_warp + ebuf * C::EPI_BYTES;
#pragma unroll
                    for (int q = 0; q < NQ; q++)
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const uint32_t old = *reinterpret_cast<const uint32_t *>(tc::frag_word(stg, q, k));
                            uint32_t *w = &v[k >> 1][4 * q + 2 * (k & 1)];
                            w[0] = __float_as_uint(__uint_as_float(w[0]) + __uint_as_float(old << 16));
                            w[1] = __float_as_uint(__uint_as_float(w[1]) + __uint_as_float(old & 0xFFFF0000u));
                        }
                }
                if (EXTRA == EXTRA_MASK && p.accum == TC_ACCUM_DIRECT) {
                    // the same beside a mask, which has the staging buffer: from the output
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int mr = m0 + ew * 32 + (lane >> 2) + 8 * k;
                        size_t pix = (size_t) mr;
                        if (!p.epi_tma) {
                            uint32_t q, jw, j, b;
                            cl.dwg.divmod(mr < M ? mr : 0, q, jw);
                            cl.dhg.divmod(q, b, j);
                            pix = ((size_t) b * p.Hout + cl.oy0 + cl.osy * (int) j) * p.Wout + cl.ox0 + cl.osx * (int) jw;
                        }
                        const int col = nb + 2 * (lane & 3);
                        const uint32_t *old = reinterpret_cast<const uint32_t *>(p.out + pix * p.Cout + col);
                        uint32_t ow[NQ];
#pragma unroll
                        for (int q = 0; q < NQ; q++) ow[q] = mr < M && col + 8 * q < p.Cout ? old[4 * q] : 0u;
#pragma unroll
                        for (int q = 0; q < NQ; q++) {
                            uint32_t *w = &v[k >> 1][4 * q + 2 * (k & 1)];
                            w[0] = __float_as_uint(__uint_as_float(w[0]) + __uint_as_float(ow[q] << 16));
                            w[1] = __float_as_uint(__uint_as_float(w[1]) + __uint_as_float(ow[q] & 0xFFFF0000u));
                        }
                    }
                }
                if constexpr (C::OUTF32) {
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        float4 sc = make_float4(1.0f, 1.0f, 1.0f, 1.0f), sh = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        if (affine) {
                            sc = *reinterpret_cast<const float4 *>(scp + c0 + 4 * j);
                            sh = *reinterpret_cast<const float4 *>(shp + c0 + 4 * j);
                        }
                        uint32_t *w = &v[0][4 * j];
                        w[0] = __float_as_uint(fmaf(__uint_as_float(w[0]), sc.x, sh.x));
                        w[1] = __float_as_uint(fmaf(__uint_as_float(w[1]), sc.y, sh.y));
                        w[2] = __float_as_uint(fmaf(__uint_as_float(w[2]), sc.z, sh.z));
                        w[3] = __float_as_uint(fmaf(__uint_as_float(w[3]), sc.w, sh.w));
                    }
                } else {
                    tc::frag_affine(v, affine, scp + c0, shp + c0);
                }
                if constexpr (EXTRA == EXTRA_SUMS || EXTRA == EXTRA_STATS) {
                    // Column sums of this item's 64 columns over the warp's 32 rows, to group
                    // gbase + m0 / 32 + ew of the class (the classes' groups are concatenated): the forward's
                    // batch-norm sums of z and z^2, or the sums of the masked input gradient (the bias
                    // gradient of the layer that produced the mask).
                    const int rows = M - (m0 + ew * 32);
                    if (rows > 0) {
                        if (rows < 32) tc::frag_clear_rows(v, rows);
                        float2 sum, sq;
                        tc::frag_col_sums<EXTRA == EXTRA_STATS>(v, sum, sq);
                        float *part = p.stats + (size_t) (cl.gbase + (m0 >> 5) + ew) * 2 * p.Cout + nb + 2 * lane;
                        if (nb + 2 * lane < p.Cout) {   // Cout is a multiple of 8
                            *reinterpret_cast<float2 *>(part) = sum;
                            if (EXTRA == EXTRA_STATS) *reinterpret_cast<float2 *>(part + p.Cout) = sq;
                        }
                    }
                }
                uint32_t pk[32];   // 128 bytes of each of the 32 rows, over the warp
                if constexpr (C::OUTF32) {
#pragma unroll
                    for (int j = 0; j < 32; j++) pk[j] = p.relu ? __float_as_uint(fmaxf(__uint_as_float(v[0][j]), 0.0f)) : v[0][j];
                } else {
                    tc::frag_pack(v, p.relu != 0, pk);
                }
                if constexpr (EXTRA == EXTRA_MASK) {
                    // ReLU backward: the outputs where the mask is positive; each word of the mask lies where the
                    // word of the output goes
                    uint8_t *stg = stg_warp + ebuf * C::EPI_BYTES;
#pragma unroll
                    for (int q = 0; q < 8; q++)
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            pk[4 * q + k] &= positive_mask(*reinterpret_cast<const uint32_t *>(tc::frag_word(stg, q, k)));
                }
                // to the staging buffer of the warp
                auto stage = [&](uint8_t *stg) {
                    if constexpr (C::OUTF32) {
#pragma unroll
                        for (int q = 0; q < 8; q++)
                            *reinterpret_cast<uint4 *>(stg + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                                make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
                    } else {
                        tc::frag_stage(stg, pk);
                    }
                };
                by_tma = next_by_tma;
                if (p.epi_tma) {
                    // each warp stages its 32 rows (4 KB) and stores them with its own TMA
                    // store: no barrier across the epilogue warps (out-of-range rows/columns
                    // are clipped by the store)
                    if (lane == 0) {
                        if (C::EPI_BUFS == 2) bulk_wait_read<1>();
                        else bulk_wait_read<0>();
                    }
                    __syncwarp();
                    uint8_t *stg = stg_warp + ebuf * C::EPI_BYTES;
                    stage(stg);
                    tc::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (nb < p.Cout && m0 + ew * 32 < M) tma_store_2d(&omap, tc::smem_u32(stg), nb, m0 + ew * 32);
                        bulk_commit();   // a group per item, so that waiting for all but the last frees the other buffer
                    }
                } else if (!C::OUTF32) {
                    // rows scattered over the output (stride-phase classes): staged through this warp's
                    // buffer, then each store instruction writes four whole 128-byte rows (eight lanes
                    // per row, Cout a multiple of their 8 channels) instead of 16 bytes of 32 rows
                    uint8_t *stg = stg_warp + ebuf * C::EPI_BYTES;
                    if (lane == 0 && C::EPI_BUFS == 2) bulk_wait_read<1>();
                    else if (lane == 0) bulk_wait_read<0>();
                    __syncwarp();
                    stage(stg);
                    __syncwarp();
                    const unsigned long long my = (unsigned long long) (orow ? orow + (size_t) nb * 2 : nullptr);
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const int r = q * 4 + (lane >> 3), ch = lane & 7;
                        const unsigned long long dst = __shfl_sync(0xFFFFFFFFu, my, r);
                        const uint4 u = *reinterpret_cast<const uint4 *>(stg + r * 128 + ((ch ^ (r & 7)) << 4));
                        if (dst && nb + ch * 8 < p.Cout) *reinterpret_cast<uint4 *>((uint8_t *) dst + ch * 16) = u;
                    }
                    __syncwarp();
                } else {
                    // FP32 rows that TMA cannot store (an output off the 16-byte grid)
                    uint8_t *stg = stg_warp + ebuf * C::EPI_BYTES;
                    __syncwarp();
                    stage(stg);
                    __syncwarp();
                    if (orow) {
                        float *o = reinterpret_cast<float *>(orow) + nb;
#pragma unroll 1
                        for (int q = 0; q < 8; q++) {
                            const float4 u = *reinterpret_cast<const float4 *>(stg + lane * 128 + ((q ^ (lane & 7)) << 4));
                            const float e[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                            for (int j = 0; j < 4; j++)
                                if (nb + 4 * q + j < p.Cout) o[4 * q + j] = e[j];
                        }
                    }
                }
                if (C::EPI_BUFS == 2) ebuf ^= 1;
            }
        }
        if (lane == 0) bulk_wait_all();
    } else {
        // ------------------------------------------------ MMA issuer
        {
            constexpr bool F8 = MODE == MODE_FP8 || MODE == MODE_FP8W;
            const uint32_t idesc = (F8 ? tc::idesc_e4m3(128, 0) : tc::idesc_bf16(128, 0, 0, 0)) | (uint32_t) (nn >> 3) << 17;
            uint32_t it = 0, lt = 0;
            for (int tile = cta; tile < p.ntiles_total && ok; tile += gridDim.x, lt++) {
                const Tile tl = decode_tile(cls_tab, p.ncls, p.ntiles, nn, tile, MT);
                int KT = __shfl_sync(0xFFFFFFFFu, cls_tab[tl.cls].ktiles, 0);   // warp-uniform loop bounds
                if (split > 1) KT = KT * (krank + 1) / split - KT * krank / split;
                const int buf = lt % C::ACC_BUFS;
                if (lt >= (uint32_t) C::ACC_BUFS) {
                    ok = tc::w::mbar_wait(&acc_empty[buf], ((lt / C::ACC_BUFS) - 1) & 1, p.err, 4);
                    if (!ok) break;
                    tc::tc_fence_after();
                }
                const uint32_t dt = tmem + (uint32_t) (buf * MT * BN);
                for (int kt = 0; kt < KT; kt += KB, it++) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!tc::w::mbar_wait(&full[s], ph, p.err, 2)) {
                        ok = false;
                        break;
                    }
                    tc::tc_fence_after();
                    const int nkb = min(KB, KT - kt);
                    const uint32_t a0 = tc::smem_u32(base + s * C::STAGE_BYTES);
                    // descriptors built once per stage; an offset of d bytes adds d / 16 to the
                    // start field (the stage stays below 256 KB, so the field never carries)
                    const uint64_t ad0 = op_desc(a0, C::SBO, C::LAYOUT);
                    const uint64_t bd0 = ad0 + (C::A_BYTES >> 4);
#pragma unroll
                    for (int kb = 0; kb < KB; kb++) {
                        if (kb >= nkb) break;
                        // each MMA consumes 32 bytes of every K row: 16 BF16 or 32 E4M3 elements
#pragma unroll
                        for (int k = 0; k < C::ROWB / 32; k++) {
                            const uint32_t acc = (kt | kb | k) != 0;
                            const uint64_t bd = bd0 + ((kb * C::B_BLOCK + k * 32) >> 4);
#pragma unroll
                            for (int mt = 0; mt < MT; mt++) {
                                const uint64_t ad = ad0 + (((kb * MT + mt) * C::A_BLOCK + k * 32) >> 4);
                                const uint32_t dtm = dt + (uint32_t) (mt * BN);
                                if (F8) {
                                    tc::w::mma_f8(dtm, ad, bd, idesc, acc);
                                } else {
                                    tc::w::mma_f16(dtm, ad, bd, idesc, acc);
                                    if (MODE == MODE_X3) {
                                        const uint64_t adl = ad + (C::A_TILE >> 4);
                                        const uint64_t bdl = bd + (C::B_TILE >> 4);
                                        tc::w::mma_f16(dtm, ad, bdl, idesc, 1);   // hi * lo
                                        tc::w::mma_f16(dtm, adl, bd, idesc, 1);   // lo * hi
                                    }
                                }
                            }
                        }
                    }
                    tc::w::mma_commit(&empty[s]);
                }
                tc::w::mma_commit(&acc_full[buf]);
            }
        }
        __syncwarp();
    }
    if (split > 1 && !met) {   // the threads without a share in the exchange
        tc::cluster_meet();
        tc::cluster_meet();
    }

    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (warp == C::MMA_WARP) tc::tmem_dealloc(tmem, C::TMEM_COLS);
}

template <int BN, int STAGES, int KB, bool IM2C, int MODE, int MT = 1, int EW = 4, int EXTRA = EXTRA_NONE>
cudaError_t launch_bn(const TcConvParams &p, const CUtensorMap &wmap, const CUtensorMap &omap, const TcMaps &amaps,
                      int grid, cudaStream_t st) {
    using C = TcCfg<BN, STAGES, KB, MODE, MT, EW>;
    auto kern = tc_conv_kernel<BN, STAGES, KB, IM2C, MODE, MT, EW, EXTRA>;
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) C::SMEM);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    if (p.split > 1) return cg_launch_pdl_cluster(p.split, kern, dim3(grid), dim3(C::THREADS), C::SMEM, st, p, wmap, omap, amaps);
    return cg_launch_pdl(kern, dim3(grid), dim3(C::THREADS), C::SMEM, st, p, wmap, omap, amaps);
}

}  // namespace

// Stage shapes (~192 KB of ring each).  BF16 im2col: BN=64 4 stages of 2 K blocks,
// BN=128 3 x 2, BN=256 3 x 1 with two output staging buffers (its tiles are often
// single-block 1x1 layers bound by the output stores).  FP8 blocks are half the bytes,
// 3xBF16 blocks twice.
int tc_conv_stages(int bn, int im2col, int mt, int ew, int kb1) {
    if (!im2col) return bn == 64 ? 8 : (bn == 128 ? 6 : 4);
    if (ew == 8) return mt == 2 ? 3 : (bn == 128 ? 4 : 3);
    if (mt == 2) return bn == 256 ? 3 : 4;
    if (kb1 && bn != 256) return bn == 64 ? 8 : 6;
    return bn == 64 ? 4 : 3;
}

namespace {
// The forms with a mask or column sums: one M tile, eight epilogue warps (four beside the gathers), two
// staging buffers.
template <int EXTRA>
cudaError_t launch_extra(const TcConvParams &p, const CUtensorMap &wmap, const CUtensorMap &omap, const TcMaps &amaps,
                         int grid, cudaStream_t st) {
    if (p.mode != MODE_BF16 || p.mt != 1 || p.ew != (p.im2col ? 8 : 4)) return cudaErrorInvalidValue;
    if (p.im2col) {
        switch (p.bn) {
            case 64: return launch_bn<64, 3, 2, true, MODE_BF16, 1, 8, EXTRA>(p, wmap, omap, amaps, grid, st);
            case 128: return launch_bn<128, 4, 1, true, MODE_BF16, 1, 8, EXTRA>(p, wmap, omap, amaps, grid, st);
            case 256: return launch_bn<256, 3, 1, true, MODE_BF16, 1, 8, EXTRA>(p, wmap, omap, amaps, grid, st);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (p.bn) {
        case 64: return launch_bn<64, 6, 1, false, MODE_BF16, 1, 4, EXTRA>(p, wmap, omap, amaps, grid, st);
        case 128: return launch_bn<128, 5, 1, false, MODE_BF16, 1, 4, EXTRA>(p, wmap, omap, amaps, grid, st);
        case 256: return launch_bn<256, 3, 1, false, MODE_BF16, 1, 4, EXTRA>(p, wmap, omap, amaps, grid, st);
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace

cudaError_t tc_conv_launch(const TcConvParams &p, const CUtensorMap &wmap, const CUtensorMap &omap,
                           const TcMaps &amaps, int grid, cudaStream_t st) {
    if (p.mode == MODE_FP8) {
        switch (p.bn) {
            case 64: return launch_bn<64, 4, 4, true, MODE_FP8>(p, wmap, omap, amaps, grid, st);
            case 128: return launch_bn<128, 3, 4, true, MODE_FP8>(p, wmap, omap, amaps, grid, st);
            case 256: return launch_bn<256, 3, 2, true, MODE_FP8>(p, wmap, omap, amaps, grid, st);
            default: return cudaErrorInvalidValue;
        }
    }
    if (p.mode == MODE_FP8W) {   // 128-channel blocks: 16 KB per 128-row block, as BF16
        switch (p.bn) {
            case 64: return launch_bn<64, 4, 2, true, MODE_FP8W>(p, wmap, omap, amaps, grid, st);
            case 128: return launch_bn<128, 3, 2, true, MODE_FP8W>(p, wmap, omap, amaps, grid, st);
            case 256: return launch_bn<256, 3, 1, true, MODE_FP8W>(p, wmap, omap, amaps, grid, st);
            default: return cudaErrorInvalidValue;
        }
    }
    if (p.mode == MODE_X3) {
        switch (p.bn) {
            case 64: return launch_bn<64, 4, 1, true, MODE_X3>(p, wmap, omap, amaps, grid, st);
            case 128: return launch_bn<128, 3, 1, true, MODE_X3>(p, wmap, omap, amaps, grid, st);
            case 256: return launch_bn<256, 2, 1, true, MODE_X3>(p, wmap, omap, amaps, grid, st);
            default: return cudaErrorInvalidValue;
        }
    }
    if (p.stats && p.sums_only) return launch_extra<EXTRA_SUMS>(p, wmap, omap, amaps, grid, st);
    if (p.stats) return launch_extra<EXTRA_STATS>(p, wmap, omap, amaps, grid, st);
    if (p.accum == TC_ACCUM_STAGED) return launch_extra<EXTRA_ACC>(p, wmap, omap, amaps, grid, st);
    if (p.mask) return launch_extra<EXTRA_MASK>(p, wmap, omap, amaps, grid, st);
    if (p.im2col && p.ew == 8) {
        // eight epilogue warps (short-K tiles): one K block per stage, two staging buffers
        if (p.mt == 2) {
            switch (p.bn) {
                case 64: return launch_bn<64, 3, 1, true, MODE_BF16, 2, 8>(p, wmap, omap, amaps, grid, st);
                case 128: return launch_bn<128, 3, 1, true, MODE_BF16, 2, 8>(p, wmap, omap, amaps, grid, st);
                default: return cudaErrorInvalidValue;
            }
        }
        switch (p.bn) {
            case 128: return launch_bn<128, 4, 1, true, MODE_BF16, 1, 8>(p, wmap, omap, amaps, grid, st);
            case 256: return launch_bn<256, 3, 1, true, MODE_BF16, 1, 8>(p, wmap, omap, amaps, grid, st);
            default: return cudaErrorInvalidValue;
        }
    }
    if (p.im2col && p.mt == 2) {
        // two M tiles per weight tile: 40 / 48 / 64 KB per K block
        switch (p.bn) {
            case 64: return launch_bn<64, 4, 1, true, MODE_BF16, 2>(p, wmap, omap, amaps, grid, st);
            case 128: return launch_bn<128, 4, 1, true, MODE_BF16, 2>(p, wmap, omap, amaps, grid, st);
            case 256: return launch_bn<256, 3, 1, true, MODE_BF16, 2>(p, wmap, omap, amaps, grid, st);
            default: return cudaErrorInvalidValue;
        }
    }
    if (p.mt != 1) return cudaErrorInvalidValue;
    if (p.im2col && p.kb1) {
        switch (p.bn) {
            case 64: return launch_bn<64, 8, 1, true, MODE_BF16>(p, wmap, omap, amaps, grid, st);
            case 128: return launch_bn<128, 6, 1, true, MODE_BF16>(p, wmap, omap, amaps, grid, st);
            default: break;   // 256-wide tiles keep their three one-block stages
        }
    }
    if (p.im2col) {
        switch (p.bn) {
            case 64: return launch_bn<64, 4, 2, true, MODE_BF16>(p, wmap, omap, amaps, grid, st);
            case 128: return launch_bn<128, 3, 2, true, MODE_BF16>(p, wmap, omap, amaps, grid, st);
            case 256: return launch_bn<256, 3, 1, true, MODE_BF16>(p, wmap, omap, amaps, grid, st);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (p.bn) {
        case 64: return launch_bn<64, 8, 1, false, MODE_BF16>(p, wmap, omap, amaps, grid, st);
        case 128: return launch_bn<128, 6, 1, false, MODE_BF16>(p, wmap, omap, amaps, grid, st);
        case 256: return launch_bn<256, 4, 1, false, MODE_BF16>(p, wmap, omap, amaps, grid, st);
        default: return cudaErrorInvalidValue;
    }
}
