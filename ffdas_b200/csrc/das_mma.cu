// das_mma.cu -- host side of the tensor-core delay-and-sum (das_mma.cuh).
#include <cuda.h>
#include <algorithm>
#include <climits>
#include <cstring>

#include "das_mma.cuh"
#include "das_staged_host.cuh"
#include "das_tile_plan.cuh"

namespace ffdas {

// Fewest items: a window's weights cost the same for any number of items.
constexpr int kMmaMinItems = 32;

bool mma_supported(const das_problem &pb, ffdas_datatype_t xt, ffdas_datatype_t ot, int kind) {
    return xt == FFDAS_R_16F && ot == FFDAS_R_32F && kind == ST_F16 && !pb.sparse && pb.B >= kMmaMinItems && pb.C > 0 &&
           pb.S > 0 && pb.S <= kMmaMaxEvents && pb.N >= kMmaW && pb.B <= 65535 && tensor_map_encoder() != nullptr &&
           plan_max_tiles(pb, kMmaTile) > 0 && plan_max_tiles(pb, kMmaTile) <= INT32_MAX;
}

// A (channel, event) of a tile takes the products 1.3 us on an SM whatever the items;
// the batch tiles take 0.45 ps a voxel and item of every event place, in passes of
// four.  Where the windows fit they meet at 85 to 125 items of whole passes (times of
// both, us: 160 channels, 3 events, 400 x 256 pixels, 32 items 1670 and 756; 92, 6,
// 150 x 200, 64: 685 and 672; 192, 9, 299 x 102, 81: 2726 and 2572; 64, 3, 400 x 256,
// 81: 661 and 809; 128, 8, 200 x 100, 128: 993 and 1265), and windows that overflow cost
// the batch tiles up to 5.4 times that (192, 8, 100 x 64, 56: 953 and 2780).  Both are
// launched below 100 (what the loser costs, 12 us on a call of 300 and 20 on one of 100,
// buys the choice), and the products run from a padding and overflow on that bring the
// items to 112 (48 items, 192, 2, 299 x 102: 625 and 537).
float mma_products_above(const das_problem &pb) {
    const float places = (float)((pb.S + 3) / 4 * 4) / (float)pb.S;
    const float items = (float)pb.B * places;
    return items < 100.f ? 112.f / items : 0.f;
}

// 4-D map over x: samples, events, channels, items; box {64, 1, 1, items},
// 128-byte swizzle; samples and items past the end read as zeros.
static ffdas_error_t sample_map(CUtensorMap &map, const void *x, const das_problem &pb, int64_t bs, int64_t cs, int64_t ss,
                                int items) {
    const cuuint64_t dims[4] = {(cuuint64_t)pb.N, (cuuint64_t)pb.S, (cuuint64_t)pb.C, (cuuint64_t)pb.B};
    const cuuint64_t strides[3] = {(cuuint64_t)ss * 2, (cuuint64_t)cs * 2, (cuuint64_t)bs * 2};
    const cuuint32_t box[4] = {(cuuint32_t)kMmaW, 1u, 1u, (cuuint32_t)items};
    const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
    const CUresult r = tensor_map_encoder()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(x), dims, strides,
                                            box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? FFDAS_SUCCESS : FFDAS_ERROR_CUDA_DRIVER;
}

ffdas_error_t launch_mma(ffdas_context &h, const das_problem &pb, const das_call &a, float *out, void *made,
                         const int *run_if) {
    // items per CTA: at most 256 columns of tensor memory per product, evenly
    const int groups = (pb.B + 255) / 256;
    const int items = ((pb.B + groups - 1) / groups + 15) / 16 * 16;
    const int chunks = (pb.B + items - 1) / items;

    // rows TMA can read: 16-byte aligned base and strides (a stride of a
    // single-element dimension is never used)
    int64_t bs = pb.B > 1 ? pb.x_bstride : 8, cs = pb.C > 1 ? pb.x_cstride : 8, ss = pb.S > 1 ? pb.x_sstride : 8;
    const __half *x = static_cast<const __half *>(a.x);
    const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && bs > 0 && cs > 0 && ss > 0 && bs % 8 == 0 &&
                         cs % 8 == 0 && ss % 8 == 0;
    const int64_t npad = ((int64_t)pb.N + 7) & ~int64_t(7);
    const size_t packed = aligned ? 0 : (size_t)pb.B * pb.C * pb.S * npad * sizeof(__half);
    workspace W(h);
    FFDAS_TRY(W.alloc(packed + 512));
    void *plan = W.get<char>() + ((packed + 255) & ~size_t(255));
    if (!aligned) {
        __half *xp = W.get<__half>();
        dim3 grid((unsigned)((npad / 8 + 255) / 256), (unsigned)std::min(pb.S, 65535),
                  (unsigned)std::min<int64_t>((int64_t)pb.B * pb.C, 65535));
        // blocks that may have nothing to do are few, and walk the rows
        if (run_if) grid.z = std::min(grid.z, std::max(1u, 4096u / (grid.x * grid.y)));
        mma_repack_kernel<<<grid, 256, 0, h.stream>>>(x, pb.x_bstride, pb.x_cstride, pb.x_sstride, pb.C, pb.S, pb.N,
                                                      pb.B * pb.C, (int)npad, xp, run_if);
        FFDAS_TRY(ffdas_launch_check(h.stream));
        x = xp;
        ss = npad;
        cs = npad * pb.S;
        bs = npad * pb.S * pb.C;
    }

    if (!made)
        FFDAS_TRY(launch_tile_plan(h, make_plan(pb, ST_F16, a.srcpos, a.dstpos, a.offsets, pb.N, kMmaTile, kPlanMma, plan)));

    mma_params p;
    std::memset(&p, 0, sizeof(p));
    p.plan = static_cast<const tile_plan *>(made ? made : plan);
    p.nonfinite = &static_cast<tile_plan *>(made ? made : plan)->nonfinite;
    p.run_if = run_if;
    p.srcpos = a.srcpos; p.dstpos = a.dstpos; p.offsets = a.offsets; p.weights = a.weights;
    p.srcdir = reinterpret_cast<const float4 *>(a.srcdir);
    p.C = pb.C; p.S = pb.S; p.N = pb.N; p.B = pb.B; p.items = items; p.V = pb.V;
    p.D0 = pb.D0; p.D1 = pb.D1; p.D2 = pb.D2;
    p.out = out;
    p.out_bstride = pb.out_bstride;
    p.status = h.status;

    // One CTA per SM: channel slices (16 channels or more, adding into a zeroed
    // image) where the tiles leave SMs without work or a last wave nearly empty.
    const int64_t tiles = plan_max_tiles(pb, kMmaTile), ctas = tiles * chunks;
    int z = balanced_slices(plan_min_tiles(pb, kMmaTile) * chunks, h.sm_count, 1, std::min(16, pb.C / 16));
    if (z > 1) {
        p.cchunk = (pb.C + z - 1) / z;
        z = (pb.C + p.cchunk - 1) / p.cchunk;
    }
    if (z <= 1) p.cchunk = 0;
    else if (pb.out_bstride == pb.V) FFDAS_CUDA(cudaMemsetAsync(out, 0, (size_t)pb.B * pb.V * sizeof(float), h.stream));
    else FFDAS_TRY(launch_scale_image(h, pb, out, 0.f, 1));

    CUtensorMap map;
    std::memset(&map, 0, sizeof(map));
    FFDAS_TRY(sample_map(map, x, pb, bs, cs, ss, items));
    const size_t smem = mma_smem_bytes(items);
    if (ffdas_raise_smem_limit(reinterpret_cast<const void *>(das_mma_kernel), h.device_id, mma_smem_bytes(256)) !=
        cudaSuccess)
        return FFDAS_ERROR_CUDA_RUNTIME;
    h.last = ffdas_kernel_info_t{};
    h.last.variant = 10;
    h.last.tile_x = kMmaTile; h.last.tile_y = 1; h.last.tile_z = 1;
    h.last.batch_tile = items;
    h.last.storage = ST_F16;
    h.last.copy_engine = 1;
    h.last.kernels = 3 + (aligned ? 0 : 1) + (z > 1 ? 1 : 0);   // plan, products, fix-up
    h.last.grid = ctas * z;
    h.mark_start();
    das_mma_kernel<<<dim3((unsigned)tiles, (unsigned)chunks, (unsigned)z), kMmaThreads, smem, h.stream>>>(map, p);
    h.mark_stop();
    FFDAS_TRY(ffdas_launch_check(h.stream));
    mma_fixup_kernel<<<(unsigned)std::max(1, h.sm_count * 8), 256, 0, h.stream>>>(p, x, bs, cs, ss);
    return ffdas_launch_check(h.stream);
}

}  // namespace ffdas
