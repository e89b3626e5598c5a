// das_entries.cu -- host side of the sorted-entry das_sparse kernels (das_entries.cuh).
#include <cuda.h>
#include <algorithm>
#include <climits>
#include <cstring>

#include <cudaTypedefs.h>
#include "das_entries.cuh"
#include "das_staged_host.cuh"

namespace ffdas {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();   // das_staged.cu

bool entries_supported(const das_problem &pb, int kind) {
    if (!pb.sparse || (kind != ST_F32 && kind != ST_F16 && kind != ST_BF16) || !staged_batch_supported()) return false;
    const int64_t rows = (int64_t)pb.B * pb.C * pb.S;
    // At least 2^27 list places x channels x items -- 2^24 from 256 channels on,
    // where the kernel otherwise taken is the staged one over all of x's events
    // (256 channels, 16 of 32 events, 200 x 200 pixels: 1102 us, here 201) -- and
    // 256 list places per event and tile: with fewer, a window serves too few
    // entries.  Four tiles at least (1024 channels, 64 x 50 pixels: 169 us there, 197).
    const int64_t least = int64_t(1) << (pb.C >= 256 ? 24 : 27);
    if (pb.V < 4 * kEnTile || (int64_t)pb.V * pb.n_events * pb.C * pb.B < least || (int64_t)kEnTile * pb.n_events < (int64_t)256 * pb.S)
        return false;
    return pb.C > 0 && pb.S > 0 && pb.S <= kEnMaxEvents && pb.n_events >= 1 && pb.n_events <= kEnMaxList &&
           rows < INT32_MAX && pb.B <= 65535 && pb.N >= kEnWB && pb.V <= INT_MAX;
}

// 32 x 32 voxels where the grid is that wide, narrower or longer tiles for
// thin grids, 1024 in a row for a list of points.
static void entries_tile(const das_problem &pb, int &T0, int &T1, int &T2) {
    auto fit = [](int want, int dim) {   // power of two up to want, not past the first one >= dim
        int t = 1;
        while (t * 2 <= want && t < dim) t *= 2;
        return t;
    };
    T0 = fit(pb.D1 <= 1 && pb.D2 <= 1 ? kEnTile : 32, pb.D0);
    T1 = fit(kEnTile / T0, pb.D1);
    T2 = fit(kEnTile / (T0 * T1), pb.D2);
    T0 = kEnTile / (T1 * T2);
}

// Reads of x in place: FP32 samples as they are, 16-byte rows.
static bool in_place(const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x, const float *gain) {
    auto ok = [](int64_t stride, int n) { return n <= 1 || (stride > 0 && stride % 4 == 0); };
    return xt == FFDAS_R_32F && kind == ST_F32 && !gain && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
           ok(pb.x_bstride, pb.B) && ok(pb.x_cstride, pb.C) && ok(pb.x_sstride, pb.S);
}
static int64_t row_length(const das_problem &pb) { return ((int64_t)pb.N + 3) & ~int64_t(3); }
static size_t rows_bytes(const das_problem &pb) {
    return ((size_t)pb.B * pb.C * pb.S * row_length(pb) * sizeof(float) + 255) & ~size_t(255);
}

template <typename Tin, int K>
static ffdas_error_t copy_rows_t(ffdas_context &h, const das_problem &pb, const void *x, const float *gain, int gain_bstride,
                                 float *out) {
    const int npad = (int)row_length(pb);
    const dim3 grid((unsigned)((npad / 4 + 255) / 256), (unsigned)std::min(pb.S, 65535),
                    (unsigned)std::min<int64_t>((int64_t)pb.B * pb.C, 65535));
    entry_rows_kernel<Tin, K><<<grid, 256, 0, h.stream>>>(static_cast<const Tin *>(x), pb.x_bstride, pb.x_cstride,
                                                         pb.x_sstride, pb.C, pb.S, pb.N, pb.B * pb.C, npad, gain,
                                                         gain_bstride, out);
    return ffdas_launch_check(h.stream);
}
template <typename Tin>
static ffdas_error_t copy_rows(ffdas_context &h, const das_problem &pb, int kind, const void *x, const float *gain,
                               int gain_bstride, float *out) {
    if (kind == ST_F16) return copy_rows_t<Tin, ST_F16>(h, pb, x, gain, gain_bstride, out);
    if (kind == ST_BF16) return copy_rows_t<Tin, ST_BF16>(h, pb, x, gain, gain_bstride, out);
    return copy_rows_t<Tin, ST_F32>(h, pb, x, gain, gain_bstride, out);
}

// The sample rows of a call: x itself, or its copy at `buf` (rows_bytes).
static ffdas_error_t make_rows(ffdas_context &h, const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x,
                               const float *gain, int gain_bstride, void *buf, en_rows &r, bool *copied) {
    *copied = !in_place(pb, xt, kind, x, gain);
    if (!*copied) {
        r = en_rows{static_cast<const float *>(x), pb.x_bstride, pb.x_cstride, pb.x_sstride};
        return FFDAS_SUCCESS;
    }
    const int64_t np = row_length(pb);
    float *out = static_cast<float *>(buf);
    r = en_rows{out, np * pb.S * pb.C, np * pb.S, np};
    switch (xt) {
        case FFDAS_R_32F: return copy_rows<float>(h, pb, kind, x, gain, gain_bstride, out);
        case FFDAS_R_16F: return copy_rows<__half>(h, pb, kind, x, gain, gain_bstride, out);
        case FFDAS_R_16BF: return copy_rows<__nv_bfloat16>(h, pb, kind, x, gain, gain_bstride, out);
        case FFDAS_R_16I: return copy_rows<int16_t>(h, pb, kind, x, gain, gain_bstride, out);
        default: return FFDAS_ERROR_INTERNAL;
    }
}

static en_params make_params(const das_problem &pb, const gather_params &gp) {
    en_params e;
    std::memset(&e, 0, sizeof(e));
    e.n = pb.n_events; e.S = pb.S; e.C = pb.C; e.V = pb.V;
    e.D0 = pb.D0; e.D1 = pb.D1; e.D2 = pb.D2;
    entries_tile(pb, e.T0, e.T1, e.T2);
    e.n0 = (pb.D0 + e.T0 - 1) / e.T0;
    e.n1 = (pb.D1 + e.T1 - 1) / e.T1;
    e.srcpos = gp.srcpos; e.dstpos = gp.dstpos; e.offsets = gp.offsets; e.weights = gp.weights;
    e.idx = gp.sparse_idx;
    e.slots_cap = (int)std::min<int64_t>((int64_t)kEnBlocks * pb.S, (int64_t)kEnTile * pb.n_events) + 1;
    return e;
}

static int64_t entries_tiles(const das_problem &pb, const en_params &e) {
    return (int64_t)e.n0 * e.n1 * ((pb.D2 + e.T2 - 1) / e.T2);
}

size_t entries_workspace(const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x, const float *gain) {
    gather_params gp;
    std::memset(&gp, 0, sizeof(gp));
    const en_params e = make_params(pb, gp);
    const int64_t tiles = entries_tiles(pb, e);
    return (in_place(pb, xt, kind, x, gain) ? 0 : rows_bytes(pb)) + (size_t)tiles * (sizeof(en_tile) + sizeof(en_slot) * e.slots_cap + sizeof(en_entry) * kEnTile * e.n);
}

// Sorts the lists of every tile into `ws`.
static ffdas_error_t launch_sort(ffdas_context &h, const das_problem &pb, en_params &e, char *ws, int64_t *tiles) {
    *tiles = entries_tiles(pb, e);
    if (*tiles > INT32_MAX) return FFDAS_ERROR_DIMS_TOO_LARGE;
    static_assert(sizeof(en_tile) == 256 && sizeof(en_slot) == 16 && sizeof(en_entry) == 16, "workspace layout");
    char *w = ws;
    e.entries = reinterpret_cast<en_entry *>(w);
    w += (size_t)*tiles * sizeof(en_entry) * kEnTile * e.n;
    e.tiles = reinterpret_cast<en_tile *>(w);
    w += (size_t)*tiles * sizeof(en_tile);
    e.slots = reinterpret_cast<en_slot *>(w);
    // counts and indices of the buckets, an entry's rank per list position and voxel
    const size_t smem = (size_t)kEnBlocks * pb.S * 2 * sizeof(int) + (size_t)e.n * kEnTile * sizeof(uint16_t);
    if (ffdas_raise_smem_limit(reinterpret_cast<const void *>(entries_sort_kernel), h.device_id,
                               (size_t)kEnBlocks * kEnMaxEvents * 2 * sizeof(int) +
                                   (size_t)kEnMaxList * kEnTile * sizeof(uint16_t)) != cudaSuccess)
        return FFDAS_ERROR_CUDA_RUNTIME;
    entries_sort_kernel<<<(unsigned)*tiles, kEnTile, smem, h.stream>>>(e);
    return ffdas_launch_check(h.stream);
}

// Boxes {128 samples, 1 event, 8 / 4 / 2 / 1 channels, 1 item} over the sample
// rows (a stride of a single-element dimension is never used).
static ffdas_error_t entry_maps(en_maps &maps, const das_problem &pb, const en_rows &r) {
    auto bytes = [](int64_t stride, int n) { return (cuuint64_t)(n > 1 ? stride * 4 : 16); };
    for (int i = 0; i < 4; i++) {
        const cuuint64_t dims[4] = {(cuuint64_t)pb.N, (cuuint64_t)pb.S, (cuuint64_t)pb.C, (cuuint64_t)pb.B};
        const cuuint64_t strides[3] = {bytes(r.ss, pb.S), bytes(r.cs, pb.C), bytes(r.bs, pb.B)};
        const cuuint32_t box[4] = {(cuuint32_t)kEnWB, 1u, (cuuint32_t)(8 >> i), 1u};
        const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
        const CUresult res = tensor_map_encoder()(&maps.m[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(r.x),
                                                  dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (res != CUDA_SUCCESS) return FFDAS_ERROR_CUDA_DRIVER;
    }
    return FFDAS_SUCCESS;
}

// Channel slices of at least min_channels channels, whole stages of 8.
static int entries_slices(ffdas_context &h, const das_problem &pb, int64_t ctas, int resident, int min_channels,
                          int *cchunk) {
    int n = balanced_slices(ctas, h.sm_count, resident, std::min(32, pb.C / min_channels));
    const int chunk = ((pb.C + n - 1) / n + kEnChannels - 1) / kEnChannels * kEnChannels;
    n = (pb.C + chunk - 1) / chunk;
    *cchunk = n > 1 ? chunk : 0;
    return n;
}

ffdas_error_t launch_entries(ffdas_context &h, const das_problem &pb, ffdas_datatype_t xt, int kind, const void *x,
                             const float *gain, int gain_bstride, gather_params gp, void *ws) {
    en_params e = make_params(pb, gp);
    bool copied = false;
    FFDAS_TRY(make_rows(h, pb, xt, kind, x, gain, gain_bstride, ws, e.rows, &copied));
    int64_t tiles = 0;
    FFDAS_TRY(launch_sort(h, pb, e, static_cast<char *>(ws) + (copied ? rows_bytes(pb) : 0), &tiles));
    gp.T0 = e.T0; gp.T1 = e.T1; gp.T2 = e.T2; gp.n0 = e.n0; gp.n1 = e.n1;
    const int slices = entries_slices(h, pb, tiles * pb.B, 3, 16, &gp.cchunk);
    if (gp.cchunk)
        FFDAS_TRY(launch_scale_image(h, pb, static_cast<float *>(gp.out), (float)gp.beta_re, gp.beta_zero));
    en_maps maps;
    std::memset(&maps, 0, sizeof(maps));
    FFDAS_TRY(entry_maps(maps, pb, e.rows));
    const staged_params sp = base_params(h, pb, gp);
    h.last.variant = 9;
    h.last.tile_x = e.T0; h.last.tile_y = e.T1; h.last.tile_z = e.T2;
    h.last.batch_tile = 1;
    h.last.event_chunk = 0;
    h.last.copy_engine = 1;
    h.last.grid = tiles * pb.B * slices;
    h.last.kernels = 2 + (copied ? 1 : 0) + (gp.cchunk ? 1 : 0);   // (rows,) sort, (image preparation,) delay-and-sum
    const dim3 grid((unsigned)tiles, (unsigned)pb.B, (unsigned)slices);
    constexpr size_t smem = en_smem<kEnStages>::bytes;
    FFDAS_TRY((prepare_once<das_entries_kernel>(smem)));
    das_entries_kernel<<<grid, kStThreads, smem, h.stream>>>(sp, e, maps);
    return ffdas_launch_check(h.stream);
}

}  // namespace ffdas
