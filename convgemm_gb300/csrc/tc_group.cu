// Persistent grouped BF16 forward convolution: many convolutions of uneven
// shapes (each an sconvGemmNHWC('N'), src/convGemm.c:65-70) in ONE launch.
//
// A device-resident problem table holds, for every convolution, its im2col
// tensor map (activations), weight and output tensor maps, geometry, tile
// width and epilogue.  The tiles of all problems are numbered consecutively
// (problem-major; inside a problem, pixel tiles x channel tiles with the
// channel tile fastest); persistent CTAs walk them blockIdx.x, +gridDim.x, ...
// The tile width is a per-problem runtime value: at most 64 / 128 / 256 output
// channels (chosen per shape by the autotuner), divided into equal tiles of whole
// 16-column MMA widths, so that 272 channels make two tiles of 144 and not two of
// 256.  Shared memory and TMEM are sized for 256 and the MMA instruction
// descriptor carries N, so one launch mixes tile shapes.
//
// Warp roles as in tc_conv.cu's form with eight epilogue warps: warp 0 issues the
// im2col TMA for the activations and the tiled TMA for the weights, warp 1 owns
// TMEM and issues tcgen05.mma, warps 4-11 drain TMEM through the fused
// scale/shift/ReLU epilogue and TMA-store BF16 (the two warps of a lane quarter
// take alternate 64-column chunks).  Each role keeps its problem's fields in
// registers while its tiles stay in one problem.  Channels that are not a multiple
// of 64 are read as 64-channel boxes whose tail TMA zero-fills; the packed weights
// carry zeros there.
//
// What bounds it: the tensor cores at the power-limited clock on the long
// reductions, and padding: 16 k channels fill whole 64-channel blocks.
#include <algorithm>
#include <cstring>
#include <vector>
#include <cuda_bf16.h>

#include "../../include/convgemm_gpu.h"
#include "cg_common.cuh"
#include "prep.h"
#include "tc_host.h"
#include "tc_epi.cuh"
#include "tc_ptx.cuh"

namespace {

using bf16 = __nv_bfloat16;

struct alignas(64) GroupProblem {
    CUtensorMap amap;   // im2col map of x: 128 pixels x 64 channels per load
    CUtensorMap wmap;   // packed weights [kn][taps * c64]: box 64 x nn
    CUtensorMap omap;   // y as [pixels][kn]: box 64 x 32 (one epilogue warp's rows)
    int tile0, tile_end, count, ntiles_n, nn, M;   // count: convolutions in the table; nn: channels per tile
    int ktiles, cpb, isy, isx, lo_y, lo_x, Cout, relu;
    uint32_t idesc;
    FastDiv dwg, dhg;
    const float *scale, *shift;
    int32_t taps[TC_MAXTAPS];   // (offy << 16) | offx of each tap
};

constexpr int GBN = 256;
constexpr int GEW = 8;
constexpr int GTHREADS = 32 * (4 + GEW);
constexpr uint32_t A_BYTES = 128 * 128;
// The ring's 192 KB hold four, six or eight stages by the width of the problem's tiles (up to 256, 128, 64
// channels), so that narrow tiles have as many bytes in flight as wide ones: 22 convolutions led by 5 x 5, 400 -> 96
// took 472 us with three stages for all widths, 347 so. The table lists the problems by ring class, and the producer
// lets the ring run empty between two classes.
constexpr uint32_t RING_BYTES = 192 * 1024;
constexpr int GCLS = 3, GMAXSTAGES = 8;
__host__ __device__ constexpr int ring_class(int nn) { return nn > 128 ? 0 : (nn > 64 ? 1 : 2); }
__host__ __device__ constexpr int ring_stages(int c) { return 4 + 2 * c; }
__host__ __device__ constexpr uint32_t ring_stage_bytes(int c) { return A_BYTES + (c == 0 ? 256u : (c == 1 ? 128u : 64u)) * 128u; }
static_assert(ring_stages(0) * ring_stage_bytes(0) <= RING_BYTES && ring_stages(1) * ring_stage_bytes(1) <= RING_BYTES &&
                  ring_stages(2) * ring_stage_bytes(2) <= RING_BYTES && ring_stages(GCLS - 1) <= GMAXSTAGES,
              "ring");
constexpr uint32_t EPI_BYTES = GEW * 4096;   // one 32 x 64 staging chunk per epilogue warp
constexpr size_t GSMEM = RING_BYTES + EPI_BYTES + 512 + 2 * GBN * 4;
static_assert(GSMEM <= 232448, "shared memory above the 227 KB per-block limit");

__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, %0;" ::"n"(32 * GEW) : "memory"); }

// The problem of a tile and its tile range; true when it changed.
__device__ __forceinline__ bool advance(const GroupProblem *probs, int nprob, int tile, int &pi, int &end) {
    if (pi >= 0 && tile < end) return false;
    do {
        pi++;
        end = __ldg(&probs[pi].tile_end);
    } while (tile >= end && pi + 1 < nprob);
    return true;
}

__global__ void __launch_bounds__(GTHREADS, 1)
    tc_group_kernel(const GroupProblem *__restrict__ probs, int nprob, int total, int *err) {
    extern __shared__ __align__(1024) uint8_t base[];
    uint8_t *epi = base + RING_BYTES;
    uint64_t *full = (uint64_t *) (epi + EPI_BYTES);    // [ring class][stage]
    uint64_t *empty = full + GCLS * GMAXSTAGES;
    uint64_t *acc_full = empty + GCLS * GMAXSTAGES;
    uint64_t *acc_empty = acc_full + 2;
    uint32_t *tmem_holder = (uint32_t *) (acc_empty + 2);
    static_assert((2 * GCLS * GMAXSTAGES + 5) * 8 <= 512, "mbarriers");
    float *sc_tab = (float *) (epi + EPI_BYTES + 512);
    float *sh_tab = sc_tab + GBN;

    const int warp = tc::w::warp_index(), lane = threadIdx.x & 31;
    tc::pdl_wait();   // pdl_trigger: when the producer starts this CTA's last tile
    // a table prepared for another count (or tiles that would not lie on the swizzle's 1024-byte grid): run nothing
    if (__ldg(&probs[0].count) != nprob || (tc::smem_u32(base) & 1023)) {
        if (threadIdx.x == 0) atomicCAS(err, 0, 25);
        return;
    }
    total = min(total, __ldg(&probs[nprob - 1].tile_end));
    if (threadIdx.x == 0) {
        for (int s = 0; s < GCLS * GMAXSTAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], 32 * GEW);
        }
        tc::fence_mbar_init();
    }
    if (warp == 1) {
        tc::tmem_alloc(tmem_holder, 2 * GBN);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_holder;
    bool ok = true;
    int pi = -1, pend = 0;

    if (warp == 0) {
        // ---------------------------------------------- producer
        uint32_t it = 0, ph = 0, tx_bytes = 0;   // K blocks of this ring class so far, parity of the ring's turn
        int rc = -1, S = 1, s = 0;                // ring class, its stages, the next stage
        uint64_t *fullc = full, *emptyc = empty;
        const GroupProblem *P = nullptr;
        int tile0 = 0, ntn = 1, nn = 0, ktiles = 0, cpb = 1, isy = 0, isx = 0, lo_y = 0, lo_x = 0;
        FastDiv dwg, dhg;
        for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
            if (tile + (int) gridDim.x >= total) tc::pdl_trigger();   // this CTA's last tile
            if (advance(probs, nprob, tile, pi, pend)) {
                P = probs + pi;
                tile0 = __ldg(&P->tile0);
                ntn = __ldg(&P->ntiles_n);
                nn = __ldg(&P->nn);
                ktiles = __shfl_sync(0xFFFFFFFFu, __ldg(&P->ktiles), 0);   // warp-uniform loop bounds
                cpb = __ldg(&P->cpb);
                isy = __ldg(&P->isy);
                isx = __ldg(&P->isx);
                lo_y = __ldg(&P->lo_y);
                lo_x = __ldg(&P->lo_x);
                dwg = P->dwg;
                dhg = P->dhg;
                tx_bytes = A_BYTES + (uint32_t) nn * 128;
                const int c = __shfl_sync(0xFFFFFFFFu, ring_class(nn), 0);
                if (c != rc) {
                    for (uint32_t j = it > (uint32_t) S ? it - S : 0; j < it && ok; j++)
                        ok = tc::w::mbar_wait(&emptyc[j % S], (j / S) & 1, err, 21);
                    if (!ok) break;
                    rc = c;
                    S = ring_stages(c);
                    fullc = full + c * GMAXSTAGES;
                    emptyc = empty + c * GMAXSTAGES;
                    it = ph = 0;
                    s = 0;
                }
            }
            const int local = tile - tile0, mt = local / ntn, n0 = (local - mt * ntn) * nn;
            uint32_t q, jw, j, b;
            dwg.divmod(mt * 128, q, jw);
            dhg.divmod(q, b, j);
            const int h0 = (int) j * isy + lo_y, w0 = (int) jw * isx + lo_x;
            int tap = 0, cc = 0;
            int32_t to = __ldg(&P->taps[0]), to_next = __ldg(&P->taps[1]);   // the next tap's offsets, loaded ahead
            for (int kt = 0; kt < ktiles; kt++, it++) {
                if (it >= (uint32_t) S && !(ok = tc::w::mbar_wait(&emptyc[s], ph ^ 1, err, 21))) break;
                const uint32_t sa = tc::smem_u32(base + s * ring_stage_bytes(rc));
                tc::w::mbar_arrive_expect_tx(&fullc[s], tx_bytes);
                tc::w::tma_load_im2col_4d(sa, &P->amap, cc * 64, w0, h0, (int) b, (uint16_t) (to & 0xFFFF),
                                          (uint16_t) (to >> 16), &fullc[s]);
                tc::w::tma_load_2d(sa + A_BYTES, &P->wmap, kt * 64, n0, &fullc[s]);
                if (++s == S) {
                    s = 0;
                    ph ^= 1;
                }
                if (++cc == cpb) {
                    cc = 0;
                    tap++;
                    to = to_next;
                    to_next = __ldg(&P->taps[min(tap + 1, TC_MAXTAPS - 1)]);
                }
            }
        }
    } else if (warp >= 4) {
        // -------------------------------------------------- epilogue
        const int ew = (warp - 4) & 3, half = (warp - 4) >> 2, et = threadIdx.x - 128;
        uint32_t lt = 0;
        uint8_t *stg = epi + (warp - 4) * 4096;
        const GroupProblem *P = nullptr;
        int tile0 = 0, ntn = 1, nn = 0, Cout = 0, relu = 0, M = 0;
        const float *scale = nullptr, *shift = nullptr;
        for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x, lt++) {
            if (advance(probs, nprob, tile, pi, pend)) {
                P = probs + pi;
                tile0 = __ldg(&P->tile0);
                ntn = __ldg(&P->ntiles_n);
                nn = __ldg(&P->nn);
                Cout = __ldg(&P->Cout);
                relu = __ldg(&P->relu);
                M = __ldg(&P->M);
                scale = P->scale;
                shift = P->shift;
            }
            const int local = tile - tile0, mt = local / ntn, m0 = mt * 128, n0 = (local - mt * ntn) * nn;
            const int nch = (nn + 63) / 64;
            epi_bar();   // the previous tile's readers of the tables are done
            if (et < nn) {
                const int n = min(n0 + et, Cout - 1);
                sc_tab[et] = scale ? __ldg(scale + n) : 1.0f;
                sh_tab[et] = shift ? __ldg(shift + n) : 0.0f;
            }
            epi_bar();
            const int buf = lt & 1;
            ok = tc::mbar_wait(&acc_full[buf], (lt >> 1) & 1, err, 23);
            if (!ok) break;
            tc::tc_fence_after();
            if (half >= nch) {   // one chunk: the other four warps take it
                tc::tc_fence_before();
                tc::mbar_arrive(&acc_empty[buf]);
            }
#pragma unroll 1
            for (int ch = half; ch < nch; ch += 2) {
                const int c0 = max(0, min(ch * 64, nn - 64));   // the last chunk repeats columns of the one before
                uint32_t v[2][32];
                tc::frag_load(tmem + ((uint32_t) (ew * 32) << 16) + (uint32_t) (buf * GBN + c0), v);
                if (ch + 2 >= nch) {
                    tc::tc_fence_before();
                    tc::mbar_arrive(&acc_empty[buf]);
                }
                tc::frag_affine(v, scale || shift, sc_tab + c0, sh_tab + c0);
                uint32_t pk[32];
                tc::frag_pack(v, relu != 0, pk);
                // each warp stages its 32 rows and stores them itself: no barrier across warps
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncwarp();
                tc::frag_stage(stg, pk);
                tc::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (n0 + c0 < Cout && m0 + ew * 32 < M)
                        asm volatile(
                            "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                                (uint64_t) &P->omap),
                            "r"(tc::smem_u32(stg)), "r"(n0 + c0), "r"(m0 + ew * 32)
                            : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else if (warp == 1) {
        // -------------------------------------------------- MMA issuer
        uint32_t ph = 0, lt = 0, idesc = 0;
        int ktiles = 0, rc = -1, S = 1, s = 0;
        uint64_t *fullc = full, *emptyc = empty;
        for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x, lt++) {
            if (advance(probs, nprob, tile, pi, pend)) {
                ktiles = __shfl_sync(0xFFFFFFFFu, __ldg(&probs[pi].ktiles), 0);
                idesc = __shfl_sync(0xFFFFFFFFu, __ldg(&probs[pi].idesc), 0);
                const int c = __shfl_sync(0xFFFFFFFFu, ring_class(__ldg(&probs[pi].nn)), 0);
                if (c != rc) {
                    rc = c;
                    S = ring_stages(c);
                    fullc = full + c * GMAXSTAGES;
                    emptyc = empty + c * GMAXSTAGES;
                    ph = 0;
                    s = 0;
                }
            }
            const int buf = lt & 1;
            if (lt >= 2) {
                ok = tc::w::mbar_wait(&acc_empty[buf], ((lt >> 1) - 1) & 1, err, 24);
                if (!ok) break;
                tc::tc_fence_after();
            }
            const uint32_t dt = tmem + (uint32_t) (buf * GBN);
            for (int kt = 0; kt < ktiles; kt++) {
                if (!tc::w::mbar_wait(&fullc[s], ph, err, 22)) {
                    ok = false;
                    break;
                }
                tc::tc_fence_after();
                // descriptors built once per stage; a 32-byte K step adds 2 to the start field
                const uint64_t ad = tc::sw128_desc(tc::smem_u32(base + s * ring_stage_bytes(rc)), 16, 1024);
                const uint64_t bd = ad + (A_BYTES >> 4);
#pragma unroll
                for (int k = 0; k < 4; k++) tc::w::mma_f16(dt, ad + 2 * k, bd + 2 * k, idesc, (kt | k) != 0);
                tc::w::mma_commit(&emptyc[s]);
                if (++s == S) {
                    s = 0;
                    ph ^= 1;
                }
            }
            tc::w::mma_commit(&acc_full[buf]);
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (warp == 1) tc::tmem_dealloc(tmem, 2 * GBN);
}

inline int rup(int v, int m) { return (v + m - 1) / m * m; }

convgemm_status_t check_group_shape(const convgemm_shape_t &s, const char *fn) {
    if (s.b < 1 || s.h < 1 || s.w < 1 || s.c < 1 || s.kn < 1 || s.kh < 1 || s.kw < 1 || s.vstride < 1 ||
        s.hstride < 1 || s.vdil < 1 || s.hdil < 1 || s.vpad < 0 || s.hpad < 0 ||
        s.h + 2LL * s.vpad - (long long) s.vdil * (s.kh - 1) < 1 ||
        s.w + 2LL * s.hpad - (long long) s.hdil * (s.kw - 1) < 1)
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "%s: invalid geometry", fn);
    if (s.c % 8 || s.kn % 8 || s.kh * s.kw > TC_MAXTAPS || s.vstride > 8 || s.hstride > 8)
        return cg_set_error(CONVGEMM_ERROR_NOT_SUPPORTED, "%s: needs c %% 8 == 0, kn %% 8 == 0, <= 49 taps, strides <= 8",
                            fn);
    return CONVGEMM_SUCCESS;
}

}  // namespace

extern "C" size_t convgemm_group_weights_size(const convgemm_shape_t *shape) {
    if (!shape || check_group_shape(*shape, "convgemm_group_weights_size")) return 0;
    return (size_t) shape->kn * (size_t) (shape->kh * shape->kw * rup(shape->c, 64)) * 2;
}

extern "C" convgemm_status_t convgemm_group_pack_weights(convgemm_layout_t layout, const convgemm_shape_t *shape,
                                                         const float *weights, void *packed, void *stream) {
    if (!shape || !weights || !packed)
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "convgemm_group_pack_weights: NULL");
    if (convgemm_status_t e = check_group_shape(*shape, "convgemm_group_pack_weights")) return e;
    const convgemm_shape_t &s = *shape;
    const int c64 = rup(s.c, 64);
    return cg_cuda_check(prep_pack_fwd(weights, layout == CONVGEMM_NCHW, s.c, s.kh, s.kw, s.kn, c64, s.kh * s.kw * c64,
                                       packed, (cudaStream_t) stream),
                         "pack grouped weights");
}

extern "C" size_t convgemm_group_table_size(int n) { return n > 0 ? (size_t) n * sizeof(GroupProblem) : 0; }

extern "C" convgemm_status_t convgemm_group_prepare(int n, const convgemm_group_conv_t *convs, void *table,
                                                    size_t table_bytes, int *total_tiles) {
    const char *fn = "convgemm_group_prepare";
    if (n < 1 || !convs || !table || !total_tiles)
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "%s: bad arguments", fn);
    if (table_bytes < convgemm_group_table_size(n) || ((uintptr_t) table & 63))
        return cg_set_error(CONVGEMM_ERROR_WORKSPACE, "%s: table needs %zu bytes, 64-byte aligned", fn,
                            convgemm_group_table_size(n));
    // Tiles go to the persistent CTAs round-robin, so the table lists the
    // convolutions of a ring class (below) by decreasing K length (the cost of one of
    // their tiles): every CTA then gets a similar mix of long and short tiles.
    std::vector<int> order(n);
    for (int i = 0; i < n; i++) order[i] = i;
    auto klen = [&](int i) {
        const convgemm_shape_t &s = convs[i].shape;
        return (long long) s.kh * s.kw * rup(s.c > 0 ? s.c : 1, 64);
    };
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return klen(a) > klen(b); });
    // width where the caller names none: 256 channels, or 128 / 64 by the channel count where tiles that wide
    // would not give every SM two
    long long wide = 0;
    for (int i = 0; i < n; i++) {
        const convgemm_shape_t &s = convs[i].shape;
        if (check_group_shape(s, fn)) continue;   // reported below
        wide += (make_geom(cg_from_public(s)).P + 127) / 128 * ((s.kn + 255) / 256);
    }
    const bool wide_ok = wide >= 2LL * tc_num_sms();
    // equal tiles of whole 16-column widths; two tiles never share a 64-column chunk
    auto tile_width = [&](const convgemm_group_conv_t &cv) {
        const int kn = cv.shape.kn > 0 ? cv.shape.kn : 8;
        const int bn = cv.bn == 64 || cv.bn == 128 || cv.bn == 256 ? cv.bn : (kn >= 256 || wide_ok ? 256 : (kn > 64 ? 128 : 64));
        const int ntn = (kn + bn - 1) / bn, nn = rup((kn + ntn - 1) / ntn, 16);
        return nn < 64 && ntn > 1 ? 64 : nn;
    };
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return ring_class(tile_width(convs[a])) < ring_class(tile_width(convs[b])); });
    std::vector<GroupProblem> host(n);
    int t0 = 0;
    for (int oi = 0; oi < n; oi++) {
        const int i = order[oi];
        const convgemm_group_conv_t &cv = convs[i];
        if (convgemm_status_t e = check_group_shape(cv.shape, fn)) return e;
        if (!cv.x || !cv.w || !cv.y) return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "%s: conv %d has a NULL tensor", fn, i);
        const cg_shape s = cg_from_public(cv.shape);
        const ConvGeom g = make_geom(s);
        const int nn = tile_width(cv), ntn = (s.kn + nn - 1) / nn;
        const int c64 = rup(s.c, 64);
        GroupProblem &P = host[oi];
        memset(&P, 0, sizeof(P));
        const int lo_y = -s.vpad, lo_x = -s.hpad;
        const int up_y = lo_y + (g.ho - 1) * s.vstride - (s.h - 1), up_x = lo_x + (g.wo - 1) * s.hstride - (s.w - 1);
        if (lo_y < -128 || lo_x < -128 || up_y < -128 || up_y > 127 || up_x < -128 || up_x > 127)
            return cg_set_error(CONVGEMM_ERROR_NOT_SUPPORTED, "%s: conv %d: padding outside the im2col box range", fn, i);
        if (convgemm_status_t e = tc_make_im2col_map(&P.amap, cv.x, s.b, s.h, s.w, s.c, lo_y, lo_x, up_y, up_x,
                                                     s.vstride, s.hstride, 128, 2))
            return e;
        if (convgemm_status_t e = tc_make_map_2d(&P.wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, cv.w, s.kn,
                                                 s.kh * s.kw * c64, 64, nn))
            return e;
        if (convgemm_status_t e = tc_make_map_2d(&P.omap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, cv.y, g.P, s.kn, 64, 32))
            return e;
        if (g.P > (1LL << 31) - 256 || (long long) s.b * s.h * s.w * c64 > (1LL << 31) - 1)
            return cg_set_error(CONVGEMM_ERROR_NOT_SUPPORTED, "%s: conv %d has more than 2^31 elements", fn, i);
        P.tile0 = t0;
        P.count = n;
        P.ntiles_n = ntn;
        P.nn = nn;
        P.M = (int) g.P;
        P.cpb = c64 / 64;
        P.ktiles = s.kh * s.kw * P.cpb;
        P.isy = s.vstride;
        P.isx = s.hstride;
        P.lo_y = lo_y;
        P.lo_x = lo_x;
        P.Cout = s.kn;
        P.relu = cv.relu;
        P.idesc = tc::idesc_bf16(128, nn, 0, 0);
        P.dwg = FastDiv(g.wo);
        P.dhg = FastDiv(g.ho);
        P.scale = cv.scale;
        P.shift = cv.shift;
        for (int kx = 0; kx < s.kh; kx++)
            for (int ky = 0; ky < s.kw; ky++)
                P.taps[kx * s.kw + ky] = ((kx * s.vdil) << 16) | (ky * s.hdil);
        const long long end = t0 + (long long) ((g.P + 127) / 128) * P.ntiles_n;
        if (end > (1LL << 31) - 1) return cg_set_error(CONVGEMM_ERROR_NOT_SUPPORTED, "%s: more than 2^31 tiles", fn);
        t0 = (int) end;
        P.tile_end = t0;
    }
    *total_tiles = t0;
    return cg_cuda_check(cudaMemcpy(table, host.data(), sizeof(GroupProblem) * n, cudaMemcpyHostToDevice),
                         "copy group table");
}

extern "C" convgemm_status_t convgemm_group_launch(const void *table, int n, int total_tiles, void *stream) {
    if (!table || n < 1 || total_tiles < 1 || ((uintptr_t) table & 63))
        return cg_set_error(CONVGEMM_ERROR_INVALID_VALUE, "convgemm_group_launch: bad arguments");
    int *err = cg_device_error_word();
    if (!err) return cg_set_error(CONVGEMM_ERROR_CUDA, "device error word unavailable");
    static bool attr = false;
    if (!attr) {
        if (convgemm_status_t e = cg_cuda_check(
                cudaFuncSetAttribute(tc_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) GSMEM),
                "grouped kernel attributes"))
            return e;
        attr = true;
    }
    const int sms = tc_num_sms();
    const int grid = total_tiles < sms ? total_tiles : sms;
    return cg_cuda_check(cg_launch_pdl(tc_group_kernel, dim3(grid), dim3(GTHREADS), GSMEM, (cudaStream_t) stream,
                                       (const GroupProblem *) table, n, total_tiles, err),
                         "grouped kernel launch");
}
