// das_iq.cu -- host side of the complex (IQ) kernels (das_iq.cuh).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <cmath>
#include <cstring>

#include "das_iq.cuh"
#include "das_staged_host.cuh"
#include "das_tile_plan.cuh"

namespace ffdas {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();   // das_staged.cu

static iq_params make_iq_params(ffdas_context &h, const das_problem &pb, const gather_params &gp, const iq_rows &rows) {
    iq_params q;
    q.s = base_params(h, pb, gp);
    q.rows = rows;
    const double turn = (double)gp.wavenum / 6.283185307179586476925;
    q.turn_hi = (float)turn;
    q.turn_lo = (float)(turn - (double)q.turn_hi);
    return q;
}

// Windows per stage.  Forward: 64 KB of ring at most, three CTAs per SM.
// Adjoint: two CTAs per SM beside the gradient bins of the windows and the
// position gradients of the stage's channels.
constexpr int iq_windows(int WB, int BT, int SC, bool adjoint) {
    const int most = BT == 3 ? 24 : 32;
    if (!adjoint) return most;
    const int cap = SC == 1 ? (8 * BT < most / 2 ? 8 * BT : most / 2) : 4 * SC * BT;
    return most * 32 / WB < cap ? most * 32 / WB : cap;
}

template <int K, int SC, int WB, int BT>
static ffdas_error_t launch_t(ffdas_context &h, const iq_params &q, const CUtensorMap &map, dim3 grid) {
    constexpr int NW = iq_windows(WB, BT, SC, false);
    constexpr size_t smem = iq_geom<WB, K, BT, NW>::smem_bytes;
    FFDAS_TRY((prepare_once<das_iq_kernel<K, SC, WB, BT, NW>>(smem)));
    das_iq_kernel<K, SC, WB, BT, NW><<<grid, kStThreads, smem, h.stream>>>(q, map);
    return ffdas_launch_check(h.stream);
}

template <int K, int SC, int WB, int BT>
static ffdas_error_t launch_bwd_t(ffdas_context &h, const iq_params &q, const CUtensorMap &map, dim3 grid) {
    constexpr int NW = iq_windows(WB, BT, SC, true);
    constexpr size_t smem = iq_bwd_layout<WB, K, SC, BT, NW>::smem_bytes;
    FFDAS_TRY((prepare_once<das_iq_bwd_kernel<K, SC, WB, BT, NW>>(smem)));
    das_iq_bwd_kernel<K, SC, WB, BT, NW><<<grid, kStThreads, smem, h.stream>>>(q, map);
    return ffdas_launch_check(h.stream);
}

template <int K, int WB, int BT, bool ADJOINT>
static ffdas_error_t launch_sc(ffdas_context &h, const iq_params &q, const CUtensorMap &map, int SC, dim3 grid) {
    if constexpr (ADJOINT)
        return SC == 1 ? launch_bwd_t<K, 1, WB, BT>(h, q, map, grid) : launch_bwd_t<K, 4, WB, BT>(h, q, map, grid);
    else
        return SC == 1 ? launch_t<K, 1, WB, BT>(h, q, map, grid) : launch_t<K, 4, WB, BT>(h, q, map, grid);
}

static int sample_bytes(int kind) { return kind == ST_C32 ? 8 : 4; }

// Box {WB samples, 1 event, 1 channel, BT items} over the sample rows (a stride
// of a single-element dimension is never used).
static ffdas_error_t sample_map(CUtensorMap &map, const das_problem &pb, const iq_rows &r, int kind, int WB, int BT) {
    const int sb = sample_bytes(kind), units = sb / 4;
    auto bytes = [&](int64_t stride, int n) { return (cuuint64_t)(n > 1 ? stride * sb : 16); };
    const cuuint64_t dims[4] = {(cuuint64_t)pb.N * units, (cuuint64_t)pb.S, (cuuint64_t)pb.C, (cuuint64_t)pb.B};
    const cuuint64_t strides[3] = {bytes(r.ss, pb.S), bytes(r.cs, pb.C), bytes(r.bs, pb.B)};
    const cuuint32_t box[4] = {(cuuint32_t)(WB * units), 1u, 1u, (cuuint32_t)BT};
    const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
    const CUresult res = tensor_map_encoder()(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, const_cast<void *>(r.x), dims, strides,
                                              box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return res == CUDA_SUCCESS ? FFDAS_SUCCESS : FFDAS_ERROR_CUDA_DRIVER;
}

template <int K, bool ADJOINT>
static ffdas_error_t launch_width(ffdas_context &h, const das_problem &pb, const iq_params &q, int SC, int WB, int BT,
                                  dim3 grid) {
    CUtensorMap map;
    std::memset(&map, 0, sizeof(map));
    FFDAS_TRY(sample_map(map, pb, q.rows, K, WB, BT));
    if (WB == 32) {
        if (BT == 1) return launch_sc<K, 32, 1, ADJOINT>(h, q, map, SC, grid);
        if (BT == 2) return launch_sc<K, 32, 2, ADJOINT>(h, q, map, SC, grid);
        if (BT == 3) return launch_sc<K, 32, 3, ADJOINT>(h, q, map, SC, grid);
        return launch_sc<K, 32, 4, ADJOINT>(h, q, map, SC, grid);
    }
    if (BT == 1) return launch_sc<K, 64, 1, ADJOINT>(h, q, map, SC, grid);
    if (BT == 2) return launch_sc<K, 64, 2, ADJOINT>(h, q, map, SC, grid);
    if (BT == 3) return launch_sc<K, 64, 3, ADJOINT>(h, q, map, SC, grid);
    return launch_sc<K, 64, 4, ADJOINT>(h, q, map, SC, grid);
}
// Both widths: the one not planned returns at once.
template <bool ADJOINT>
static ffdas_error_t launch_planned(ffdas_context &h, const das_problem &pb, int kind, const iq_params &q, int SC, int BT,
                                    dim3 grid) {
    for (int WB = 32; WB <= 64; WB += 32) {
        if (kind == ST_C32) FFDAS_TRY((launch_width<ST_C32, ADJOINT>(h, pb, q, SC, WB, BT, grid)));
        else FFDAS_TRY((launch_width<ST_C16, ADJOINT>(h, pb, q, SC, WB, BT, grid)));
    }
    return FFDAS_SUCCESS;
}

bool iq_supported(const das_problem &pb, int kind) {
    if (pb.sparse || (kind != ST_C32 && kind != ST_C16) || !staged_batch_supported()) return false;
    const int64_t rows = (int64_t)pb.B * pb.C * pb.S;
    return pb.C > 0 && pb.S > 0 && pb.N > 0 && rows < INT32_MAX && pb.B <= 65535 &&
           plan_max_tiles(pb, kStConsumers) > 0 && plan_max_tiles(pb, kStConsumers) <= INT32_MAX;
}

// Reads of x in place: samples of the type computed on, 16-byte rows.
static bool in_place(const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x, const float *gain) {
    const int a = 16 / sample_bytes(kind);
    auto ok = [a](int64_t stride, int n) { return n <= 1 || (stride > 0 && stride % a == 0); };
    return xt == (kind == ST_C32 ? FFDAS_C_32F : FFDAS_C_16F) && !gain && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
           ok(pb.x_bstride, pb.B) && ok(pb.x_cstride, pb.C) && ok(pb.x_sstride, pb.S);
}
static int64_t row_length(const das_problem &pb) { return ((int64_t)pb.N + 3) & ~int64_t(3); }

size_t iq_workspace(const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x, const float *gain) {
    const size_t rows = in_place(pb, xt, kind, x, gain) ? 0 : (size_t)pb.B * pb.C * pb.S * row_length(pb) * sample_bytes(kind);
    return rows + 256;   // the tile plan, the rows
}

template <typename Tin, int K>
static ffdas_error_t copy_rows(ffdas_context &h, const das_problem &pb, const void *x, const float *gain, int gain_bstride,
                               void *out) {
    const int npad = (int)row_length(pb);
    const dim3 grid((unsigned)((npad / 4 + 255) / 256), (unsigned)std::min(pb.S, 65535),
                    (unsigned)std::min<int64_t>((int64_t)pb.B * pb.C, 65535));
    iq_rows_kernel<Tin, K><<<grid, 256, 0, h.stream>>>(static_cast<const Tin *>(x), pb.x_bstride, pb.x_cstride, pb.x_sstride,
                                                      pb.C, pb.S, pb.N, pb.B * pb.C, npad, gain, gain_bstride,
                                                      static_cast<typename iq_sample<K>::type *>(out));
    return ffdas_launch_check(h.stream);
}

// The sample rows of a call, x itself or its copy, and its tile plan.
static ffdas_error_t prepare(ffdas_context &h, const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x,
                             const float *gain, int gain_bstride, int mode, gather_params &gp, void *ws, iq_rows &r,
                             int *launches) {
    *launches = 1;
    r = iq_rows{x, pb.x_bstride, pb.x_cstride, pb.x_sstride};
    if (!in_place(pb, xt, kind, x, gain)) {
        const int64_t np = row_length(pb);
        void *out = static_cast<char *>(ws) + 256;
        r = iq_rows{out, np * pb.S * pb.C, np * pb.S, np};
        if (xt == FFDAS_C_32F && kind == ST_C32) FFDAS_TRY((copy_rows<float2, ST_C32>(h, pb, x, gain, gain_bstride, out)));
        else if (xt == FFDAS_C_32F) FFDAS_TRY((copy_rows<float2, ST_C16>(h, pb, x, gain, gain_bstride, out)));
        else if (xt == FFDAS_C_16F && kind == ST_C16)
            FFDAS_TRY((copy_rows<__half2, ST_C16>(h, pb, x, gain, gain_bstride, out)));
        else return FFDAS_ERROR_INTERNAL;
        *launches = 2;
    }
    gp.plan = ws;
    return launch_tile_plan(h, make_plan(pb, kind, gp.srcpos, gp.dstpos, gp.offsets, pb.N, kStConsumers, mode, ws));
}

// Channel slices of at least 8 channels, whole stages; sets gp.cchunk.
static int iq_slices(ffdas_context &h, const das_problem &pb, int64_t ctas, int resident, gather_params &gp) {
    int n = balanced_slices(ctas, h.sm_count, resident, std::min(32, pb.C / 8));
    gp.cchunk = 0;
    if (n > 1) {
        const int chunk = ((pb.C + n - 1) / n + 3) / 4 * 4;
        n = (pb.C + chunk - 1) / chunk;
        if (n > 1) gp.cchunk = chunk;
    }
    return n;
}

// Items per CTA: four, or three where that leaves fewer items past the batch.
static int iq_batch_tile(int B) {
    if (B <= 3) return B;
    return (B + 2) / 3 * 3 < (B + 3) / 4 * 4 ? 3 : 4;
}

ffdas_error_t launch_iq(ffdas_context &h, const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x,
                        const float *gain, int gain_bstride, gather_params gp, void *ws) {
    const int BT = iq_batch_tile(pb.B), bch = (pb.B + BT - 1) / BT, SC = pb.n_events == 1 ? 1 : 4;
    iq_rows rows;
    int launches = 0;
    FFDAS_TRY(prepare(h, pb, xt, kind, x, gain, gain_bstride, kPlanForward, gp, ws, rows, &launches));
    const int64_t tiles = plan_max_tiles(pb, kStConsumers);
    const int slices = iq_slices(h, pb, plan_min_tiles(pb, kStConsumers) * bch, 3, gp);
    h.last.variant = 2;
    h.last.batch_tile = BT;
    h.last.event_chunk = SC;
    h.last.storage = kind;
    h.last.copy_engine = 1;
    h.last.grid = tiles * bch * slices;
    h.last.kernels = launches + (slices > 1 ? 3 : 2);   // (rows,) plan, (image preparation,) delay-and-sum, the width not taken
    h.mark_start();
    if (gp.cchunk) {
        const dim3 sg((unsigned)((pb.V + 255) / 256), (unsigned)std::min(pb.B, 65535));
        iq_scale_image_kernel<<<sg, 256, 0, h.stream>>>(static_cast<float2 *>(gp.out), pb.out_bstride, pb.V, pb.B,
                                                        (float)gp.beta_re, (float)gp.beta_im, gp.beta_zero);
        FFDAS_TRY(ffdas_launch_check(h.stream));
    }
    const iq_params q = make_iq_params(h, pb, gp, rows);
    const ffdas_error_t err =
        launch_planned<false>(h, pb, kind, q, SC, BT, dim3((unsigned)tiles, (unsigned)bch, (unsigned)slices));
    h.mark_stop();
    return err;
}

ffdas_error_t launch_iq_bwd(ffdas_context &h, const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x,
                            gather_params gp, const staged_grads &gr, void *ws) {
    const int BT = iq_batch_tile(pb.B), bch = (pb.B + BT - 1) / BT, SC = pb.n_events == 1 ? 1 : 4;
    iq_rows rows;
    int launches = 0;
    FFDAS_TRY(prepare(h, pb, xt, kind, x, nullptr, 0, kPlanAdjoint, gp, ws, rows, &launches));
    const int64_t tiles = plan_max_tiles(pb, kStConsumers);
    const int slices = iq_slices(h, pb, plan_min_tiles(pb, kStConsumers) * bch, 2, gp);
    const bool shared_v = bch > 1 || slices > 1;   // several CTAs add into the voxel-side gradients
    FFDAS_TRY(clear_gradients(h, shared_v ? gr.gw : nullptr, shared_v ? gr.goff : nullptr, (int64_t)pb.n_events * pb.V,
                              shared_v ? gr.gdst : nullptr, pb.V * 3, gr.gsrc, (int64_t)pb.C * 3));
    h.last.variant = 8;
    h.last.batch_tile = BT;
    h.last.event_chunk = SC;
    h.last.storage = kind;
    h.last.copy_engine = 1;
    h.last.grid = tiles * bch * slices;
    h.last.kernels = launches + 2;   // (rows,) plan, adjoint, the width not taken
    iq_params q = make_iq_params(h, pb, gp, rows);
    q.s.gout = gr.gout;
    q.s.gout_bstride = gr.gout_bstride;
    q.s.gx = gr.gx; q.s.goff = gr.goff; q.s.gw = gr.gw; q.s.gdst = gr.gdst; q.s.gsrc = gr.gsrc;
    h.mark_start();
    const ffdas_error_t err =
        launch_planned<true>(h, pb, kind, q, SC, BT, dim3((unsigned)tiles, (unsigned)bch, (unsigned)slices));
    h.mark_stop();
    return err;
}

}  // namespace ffdas
