// das_mma.cuh -- delay-and-sum of large half-precision batches on the tensor
// cores (tcgen05).
//
// The delays do not depend on the batch item, so for one (channel, event) the
// interpolation of a tile is a product: image (voxels x items) += W (voxels x
// window) X (window x items), where row v of W holds w (1 - t) and w t in the
// two columns its tap falls on and zeros elsewhere, and X is the raw channel
// data of the window.  A tap costs a thread a delay, a split and a few
// half-word stores once for ALL items, and the arithmetic runs on the tensor
// cores, mostly on zeros: 48 columns for two useful ones, at 4096
// multiply-adds per clock per SM against 128 for FMAs.  (On the pair kernels a
// 200-frame ensemble, 128 channels, 11 plane waves, 400 x 256 pixels takes
// 10.3 ms and its pair ingest 0.65 ms; here 5.0 ms in all: the raw samples need no
// ingest.)
//
// Precision: the samples are the data's own half-precision values, exact.  A
// weight a (FP32) enters as hi + lo, both half precision, with the voxel's
// weights scaled by a power of two to a magnitude below 2^14: hi carries 11
// bits and lo the next 11, down to 2^-38 of the largest weight.  Products are
// exact and the sums are FP32 in tensor memory; the tensor core truncates each
// sum, which drifts with the number of addends, so the accumulators are added
// to the image (FP32, rounded) every kMmaDrain (channel, event) pairs.  What
// the drift costs, the fraction of the delay gains back: the rounding of
// tau = offset + r (2^-15 of a sample at 1000) is most of the error of an FP32
// image, and its remainder is added to the fraction here.
// Error against 64 bits of the pair kernels with FP32 weights and sums, of the
// products without the remainder, and with it: 192 channels, 9 events, 512
// samples 1.52e-5, 1.62e-5, 1.14e-5; 128, 11, 1536: 4.13e-5, 4.18e-5, 2.41e-5;
// 48, 1, 512: 1.35e-5, 1.35e-5, 0.79e-5.  (A drain every 32 pairs in its place:
// 1.52e-5, 4.14e-5, 1.35e-5, and 6.1 against 5.0 ms.)
//
// A sample that is not finite meets the zeros of W and spoils the whole tile's
// sum of its item.  mma_fixup_kernel, launched afterwards, recomputes every
// value that is not finite directly from the samples, as the other kernels
// would have.
//
// One CTA: 256 voxels (two M = 128 products) x up to 256 items.
//   warp 0     copies windows {64 samples, items} with TMA from x itself
//              (128-byte rows, 128-byte swizzle: the K-major operand layout);
//   warp 1     issues the products, one lane;
//   warps 2-17 build W, a voxel per thread, eight warps for each of the two
//              buffers (one set building both was slower than the products:
//              5.0 ms); a thread clears the two columns it wrote last time.
// Every role walks the same list of windows, computed by each warp for itself
// from the tile's box and delay ranges (a lane per channel), so nothing but
// the buffers' barriers passes between them.  A tile whose windows are wider
// than 57 samples takes several windows per (channel, event), each with the
// taps that fall into it.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "das_common.cuh"
#include "das_problem.h"
#include "das_staged.cuh"
#include "gram_tc.cuh"

namespace ffdas {

constexpr int kMmaTile = kMmaTileVoxels;   // voxels per CTA
constexpr int kMmaW = 64;          // samples per window: one 128-byte row
constexpr int kMmaStep = 56;       // taps of a window: first samples k0 .. k0 + 55
constexpr int kMmaBuilders = 256;  // threads that build one buffer
constexpr int kMmaBStages = 3, kMmaAStages = 2;
constexpr int kMmaThreads = 64 + kMmaAStages * kMmaBuilders;
constexpr int kMmaMaxEvents = 128;
constexpr int kMmaDrain = 192;     // (channel, event) pairs between drains of the accumulators
constexpr uint32_t kMmaPart = 2u * 128 * 128;        // bytes of one part (hi or lo) of W: 256 rows of 128 bytes
constexpr uint32_t kMmaAStage = 2 * kMmaPart;

struct mma_params {
    const tile_plan *plan;
    const float *srcpos, *dstpos, *offsets, *weights;
    const float4 *srcdir;
    int C, S, N, B, items;          // items: product width (a multiple of 16, at most 256)
    int64_t V;
    int D0, D1, D2, T0, T1, n0, n1;
    int cchunk;                     // channels per blockIdx.z slice (0: all)
    float *out;
    int64_t out_bstride;
    int *status;
    int *nonfinite;                 // set when a value added to the image is not finite
    const int *run_if;              // device word without which nothing is done, or null
};

constexpr size_t mma_smem_bytes(int items) {
    return 1024 + kMmaAStages * (size_t)kMmaAStage + kMmaBStages * (size_t)items * 128 + 2 * kMmaMaxEvents * 4 +
           (2 * kMmaAStages + 2 * kMmaBStages + 2) * 8 + 6 * 4 + 32;
}

// kind::f16 descriptor: FP32 accumulator, half-precision A and B, both K-major.
__host__ __device__ constexpr uint32_t mma_f16_idesc(int M, int N) {
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void st_half(uint32_t a, uint32_t bits) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((unsigned short)bits) : "memory");
}

// Windows of channels cb .. cb + 31 for one event, a lane per channel: the
// first window's first sample (a multiple of 8) and the number of samples from
// there to the last a tap can read, or 0 when no tap lies in the record.
struct mma_block {
    int k0, len;
    float px, py, pz;
};
__device__ __forceinline__ mma_block mma_windows(const mma_params &p, const float *box, float olo, float ohi, int c,
                                                 int cend) {
    mma_block w = {0, 0, 0.f, 0.f, 0.f};
    if (c >= cend) return w;
    w.px = __ldg(p.srcpos + 3 * c);
    w.py = __ldg(p.srcpos + 3 * c + 1);
    w.pz = __ldg(p.srcpos + 3 * c + 2);
    const float dx = fmaxf(fmaxf(box[0] - w.px, w.px - box[3]), 0.f);
    const float dy = fmaxf(fmaxf(box[1] - w.py, w.py - box[4]), 0.f);
    const float dz = fmaxf(fmaxf(box[2] - w.pz, w.pz - box[5]), 0.f);
    const float ex = fmaxf(fabsf(w.px - box[0]), fabsf(w.px - box[3]));
    const float ey = fmaxf(fabsf(w.py - box[1]), fabsf(w.py - box[4]));
    const float ez = fmaxf(fabsf(w.pz - box[2]), fabsf(w.pz - box[5]));
    // (a channel position that is not finite has no window: NaN, or nothing in
    // range; the builders spoil their voxels and the fix-up decides)
    float lo, hi;
    tap_range(olo, ohi, sqrtf(dx * dx + dy * dy + dz * dz), sqrtf(ex * ex + ey * ey + ez * ez), lo, hi);
    if (!isfinite(w.px + w.py + w.pz) || !(hi >= 0.f) || !(lo < (float)(p.N - 1))) return w;
    w.k0 = (int)fmaxf(lo, 0.f) & ~7;
    w.len = (int)fminf(hi, (float)(p.N - 1)) - w.k0 + 1;
    return w;
}
// 16-sample steps of window i of `len` samples.
__device__ __forceinline__ int mma_ksteps(int len, int i) { return (min(len - i * kMmaStep, kMmaStep + 1) + 15) >> 4; }
__device__ __forceinline__ int mma_count(int len) { return len > 1 ? (len - 1 + kMmaStep - 1) / kMmaStep : (len > 0 ? 1 : 0); }

__global__ void __launch_bounds__(kMmaThreads, 1) das_mma_kernel(const __grid_constant__ CUtensorMap map,
                                                                 const mma_params params) {
    mma_params p = params;
    if (p.run_if && *p.run_if == 0) return;   // uniform over the grid
    if (p.plan) {
        p.T0 = p.plan->T0; p.T1 = p.plan->T1; p.n0 = p.plan->n0; p.n1 = p.plan->n1;
        if ((int64_t)blockIdx.x >= (int64_t)p.n0 * p.n1 * p.D2) return;
    }
    extern __shared__ unsigned char smem_raw[];
    const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
    unsigned char *abuf = smem_raw + pad;
    const uint32_t a_u32 = smem_u32(abuf), b_u32 = a_u32 + kMmaAStages * kMmaAStage, b_bytes = (uint32_t)p.items * 128;
    float *olo = reinterpret_cast<float *>(abuf + kMmaAStages * kMmaAStage + kMmaBStages * b_bytes), *ohi = olo + kMmaMaxEvents;
    uint64_t *bars = reinterpret_cast<uint64_t *>(ohi + kMmaMaxEvents);
    // barriers: W built / free, window loaded / free, products done, accumulators read
    const uint32_t a_full = smem_u32(bars), a_free = a_full + 8 * kMmaAStages, b_full = a_free + 8 * kMmaAStages,
                   b_free = b_full + 8 * kMmaBStages, done = b_free + 8 * kMmaBStages, drained = done + 8;
    float *box = reinterpret_cast<float *>(bars + 2 * kMmaAStages + 2 * kMmaBStages + 2);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(box + 6);
    int *abort_word = reinterpret_cast<int *>(tmem_slot + 1);
    volatile int *abort = abort_word;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kMmaAStages; i++) {
            mbar_init(a_full + 8 * i, kMmaBuilders / 32);
            mbar_init(a_free + 8 * i, 1);
        }
        for (int i = 0; i < kMmaBStages; i++) {
            mbar_init(b_full + 8 * i, 1);
            mbar_init(b_free + 8 * i, 1);
        }
        mbar_init(done, 1);
        mbar_init(drained, kMmaAStages * kMmaBuilders / 32);
        *abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // voxel of a builder thread: row (warp % 4) * 32 + lane of product ((warp - 2) / 4) % 2;
    // its buffer (and half of the accumulators' columns): (warp - 2) / 8
    const int row = (warp & 3) * 32 + lane, m = warp >= 2 ? ((warp - 2) >> 2) & 1 : 0, set = warp >= 2 ? (warp - 2) >> 3 : 0;
    int64_t v = -1;
    float vx = 0.f, vy = 0.f, vz = 0.f, poison = 0.f, scale = 1.f, inv_scale = 1.f;
    int *ibox = reinterpret_cast<int *>(box), *ilo = reinterpret_cast<int *>(olo), *ihi = reinterpret_cast<int *>(ohi);
    if (threadIdx.x < 6) ibox[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
    for (int e = threadIdx.x; e < p.S; e += kMmaThreads) {
        ilo[e] = INT_MAX;
        ihi[e] = INT_MIN;
    }
    for (uint32_t i = threadIdx.x; i < kMmaAStages * kMmaAStage / 16; i += kMmaThreads)
        reinterpret_cast<uint4 *>(abuf)[i] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    auto ordered = [](float f) {   // monotone float -> int
        const int i = __float_as_int(f);
        return i >= 0 ? i : i ^ 0x7fffffff;
    };
    if (warp >= 2) {
        const int l = m * 128 + row, tile = blockIdx.x;
        const int t0 = tile % p.n0, t1 = (tile / p.n0) % p.n1, t2 = tile / (p.n0 * p.n1);
        const int g0 = t0 * p.T0 + l % p.T0, g1 = t1 * p.T1 + l / p.T0;
        if (g0 < p.D0 && g1 < p.D1) {
            v = ((int64_t)t2 * p.D1 + g1) * p.D0 + g0;
            vx = __ldg(p.dstpos + 3 * v); vy = __ldg(p.dstpos + 3 * v + 1); vz = __ldg(p.dstpos + 3 * v + 2);
            // NaN where a distance overflows or is NaN: the fix-up recomputes the voxel
            poison = fmaxf(fmaxf(fabsf(vx), fabsf(vy)), fabsf(vz)) <= 1e18f && vx == vx && vy == vy && vz == vz ? 0.f : NAN;
        }
        const float q[3] = {vx, vy, vz};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            int lo = (v >= 0 && q[a] == q[a]) ? ordered(q[a]) : INT_MAX, hi = lo == INT_MAX ? INT_MIN : lo;
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == 0) {
                atomicMin(&ibox[a], lo);
                atomicMax(&ibox[3 + a], hi);
            }
        }
        float wmax = 0.f;
        for (int e = 0; e < p.S; e++) {
            const float o = v >= 0 ? __ldg(p.offsets + (int64_t)e * p.V + v) : INFINITY;
            if (v >= 0) {
                const float w = __ldg(p.weights + (int64_t)e * p.V + v);
                wmax = fmaxf(wmax, fabsf(w));
                // NaN for a delay or a weight that is not finite, whether or not a tap meets a window
                poison = __fmaf_rn(o, 0.f, __fmaf_rn(w, 0.f, poison));
            }
            int lo = isfinite(o) ? ordered(o) : INT_MAX, hi = isfinite(o) ? ordered(o) : INT_MIN;
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == 0) {
                atomicMin(&ilo[e], lo);
                atomicMax(&ihi[e], hi);
            }
        }
        // scaled weights below 2^14 in magnitude (a weight that is not finite
        // leaves the scale at 1 and the sum not finite)
        if (wmax > 0.f && wmax <= 3.0e38f) {
            const int ex = min(max((int)(__float_as_uint(wmax) >> 23) - 127, -100), 100);   // 2^ex <= wmax < 2^(ex + 1)
            scale = __uint_as_float((uint32_t)(127 + 13 - ex) << 23);
            inv_scale = __uint_as_float((uint32_t)(127 - 13 + ex) << 23);
        }
    }
    __syncthreads();
    auto unordered = [](int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); };
    if (threadIdx.x < 6) {
        const int i = ibox[threadIdx.x];
        box[threadIdx.x] = (i == INT_MAX || i == INT_MIN) ? NAN : unordered(i);
    }
    for (int e = threadIdx.x; e < p.S; e += kMmaThreads) {
        const int lo = ilo[e], hi = ihi[e];
        float flo = lo == INT_MAX ? INFINITY : unordered(lo);     // no finite delay: no window
        float fhi = hi == INT_MIN ? -INFINITY : unordered(hi);
        widen_delays(flo, fhi);
        olo[e] = flo;
        ohi[e] = fhi;
    }
    gram_tc::fence_before_sync();
    __syncthreads();
    gram_tc::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const int cbeg = p.cchunk ? (int)blockIdx.z * p.cchunk : 0, cend = p.cchunk ? min(p.C, cbeg + p.cchunk) : p.C;
    const int b0 = blockIdx.y * p.items;

    uint32_t n = 0;         // windows so far, the same in every role
    int since = 0;          // (channel, event) pairs since the accumulators were drained
    uint32_t drains = 0;
    bool fresh = true;      // nothing accumulated since the last drain
    bool spoiled = false;   // poison (of every voxel) since the last drain
    bool dead = false, first_out = true;
    int prev = -1;          // column this thread wrote into its buffer last time
    bool odd = false;       // a value that is not finite went into the image
    uint32_t b_issued = 0;

    // Adds the accumulators to the image (builders); hands them back (issuer).
    auto drain = [&]() {
        if (warp == 1) {
            if (lane == 0 && !dead) {
                gram_tc::mma_commit(done);
                if (!gram_tc::wait(drained, drains & 1, abort, p.status)) dead = true;
                gram_tc::fence_after_sync();
            }
            dead = __shfl_sync(0xffffffffu, (int)dead, 0);
        } else if (warp >= 2) {
            if (!dead && !gram_tc::wait(done, drains & 1, abort, p.status)) dead = true;
            dead = __any_sync(0xffffffffu, dead);
            if (!dead) {
                gram_tc::fence_after_sync();
                for (int c0 = 16 * set; c0 < p.items; c0 += 16 * kMmaAStages) {
                    uint32_t r[16];
                    __syncwarp();
                    if (!fresh) gram_tc::tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(m * 256 + c0), r);
                    if (v >= 0) {
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            if (b0 + c0 + i < p.B) {
                                float *o = p.out + (int64_t)(b0 + c0 + i) * p.out_bstride + v;
                                const float val = __fmaf_rn(fresh ? 0.f : __uint_as_float(r[i]), inv_scale, poison);
                                odd |= !isfinite(val);
                                if (first_out && gridDim.z == 1) *o = val;
                                else atomicAdd(o, val);
                            }
                        }
                    }
                }
                gram_tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(drained);
            }
            first_out = false;
        }
        drains++;
        fresh = true;
        spoiled = false;
        since = 0;
    };

    for (int e = 0; e < p.S; e++) {
        const float elo = olo[e], ehi = ohi[e];
        float ofs = 1e30f, w = 0.f;
        if (v >= 0) {
            ofs = __ldg(p.offsets + (int64_t)e * p.V + v);
            w = __ldg(p.weights + (int64_t)e * p.V + v) * scale;
        }
        for (int cb = cbeg; cb < cend; cb += 32) {
            const mma_block blk = mma_windows(p, box, elo, ehi, cb + lane, cend);
            const int nc = min(32, cend - cb);
            if (__any_sync(0xffffffffu, !isfinite(blk.px + blk.py + blk.pz))) {
                poison = NAN;
                spoiled = true;
            }
            for (int j = 0; j < nc; j++) {
                const int len = __shfl_sync(0xffffffffu, blk.len, j), k00 = __shfl_sync(0xffffffffu, blk.k0, j);
                const int count = mma_count(len);
                uint32_t rel = 0xffffffffu;   // first sample of this thread's tap from k00, huge outside the record
                float t = 0.f;
                // (a window of this (channel, event) goes into this set's buffer)
                if (warp >= 2 && (count > 1 || (count == 1 && (int)(n % kMmaAStages) == set))) {
                    const float cx = __shfl_sync(0xffffffffu, blk.px, j), cy = __shfl_sync(0xffffffffu, blk.py, j),
                                cz = __shfl_sync(0xffffffffu, blk.pz, j);
                    recv_geom g = receive_geometry(vx, vy, vz, cx, cy, cz);
                    if (p.srcdir) apply_directivity(g, vx, vy, vz, cx, cy, cz, __ldg(p.srcdir + cb + j));
                    const float tau = __fmaf_rn(g.rsq, g.rinv, ofs), part = tau - ofs;
                    const tau_split ts = split_tau(tau);
                    // the remainder of the sum offset + r (Knuth's two-sum, the product
                    // unrounded); more than a unit of tau is none: far distances that far
                    // delays cancel leave `part` inexact
                    const float rest = (ofs - (tau - part)) + __fmaf_rn(g.rsq, g.rinv, -part);
                    t = ts.t + (fabsf(rest) <= tau * 0x1p-23f ? rest : 0.f);
                    if (v >= 0 && ts.k < (uint32_t)(p.N - 1)) rel = ts.k - (uint32_t)k00;
                }
                for (int i = 0; i < count; i++, n++) {
                    const int as = n % kMmaAStages, bs = n % kMmaBStages;
                    const uint32_t au = n / kMmaAStages, bu = n / kMmaBStages;
                    if (warp == 0) {
                        if (lane == 0 && !dead) {
                            if (bu > 0 && !gram_tc::wait(b_free + 8 * bs, (bu - 1) & 1, abort, p.status)) {
                                dead = true;
                            } else {
                                mbar_arrive_expect_tx(b_full + 8 * bs, b_bytes);
                                tma_load_box4(b_u32 + bs * b_bytes, &map, k00 + i * kMmaStep, e, cb + j, b0, b_full + 8 * bs);
                                b_issued = n + 1;
                            }
                        }
                    } else if (warp == 1) {
                        if (lane == 0 && !dead) {
                            if (!gram_tc::wait(a_full + 8 * as, au & 1, abort, p.status) ||
                                !gram_tc::wait(b_full + 8 * bs, bu & 1, abort, p.status)) {
                                dead = true;
                            } else {
                                gram_tc::fence_after_sync();
                                const uint32_t id = mma_f16_idesc(128, p.items);
                                const int ks = mma_ksteps(len, i);
                                const uint32_t a0 = a_u32 + as * kMmaAStage, bb = b_u32 + bs * b_bytes;
                                for (int mm = 0; mm < 2; mm++)
                                    for (int part = 0; part < 2; part++)
                                        for (int k = 0; k < ks; k++)
                                            mma_f16(tmem + mm * 256,
                                                    gram_tc::sw128_desc(a0 + part * kMmaPart + mm * (kMmaPart / 2) + k * 32),
                                                    gram_tc::sw128_desc(bb + k * 32), id,
                                                    (fresh && part == 0 && k == 0) ? 0u : 1u);
                                gram_tc::mma_commit(a_free + 8 * as);
                                gram_tc::mma_commit(b_free + 8 * bs);
                            }
                        }
                    } else if (!dead && as == set) {
                        if (au > 0 && !gram_tc::wait(a_free + 8 * as, (au - 1) & 1, abort, p.status)) dead = true;
                        dead = __any_sync(0xffffffffu, dead);
                        if (!dead) {
                            const uint32_t rb = a_u32 + as * kMmaAStage + m * (kMmaPart / 2) + row * 128;
                            const uint32_t x = (uint32_t)(row & 7) << 4;
                            if (prev >= 0) {
                                const uint32_t c0 = rb + (((uint32_t)prev * 2) ^ x), c1 = rb + (((uint32_t)prev * 2 + 2) ^ x);
                                st_half(c0, 0u);
                                st_half(c1, 0u);
                                st_half(c0 + kMmaPart, 0u);
                                st_half(c1 + kMmaPart, 0u);
                            }
                            const uint32_t col = rel - (uint32_t)(i * kMmaStep);
                            prev = -1;
                            if (rel != 0xffffffffu && col < (uint32_t)kMmaStep) {
                                const float a1 = w * t, a0 = __fmaf_rn(-w, t, w);
                                const __half h0 = __float2half_rn(a0), h1 = __float2half_rn(a1);
                                const __half l0 = __float2half_rn(a0 - __half2float(h0)), l1 = __float2half_rn(a1 - __half2float(h1));
                                const uint32_t c0 = rb + ((col * 2) ^ x), c1 = rb + ((col * 2 + 2) ^ x);
                                st_half(c0, __half_as_ushort(h0));
                                st_half(c1, __half_as_ushort(h1));
                                st_half(c0 + kMmaPart, __half_as_ushort(l0));
                                st_half(c1 + kMmaPart, __half_as_ushort(l1));
                                prev = (int)col;
                            }
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) mbar_arrive(a_full + 8 * as);
                        }
                    }
                    fresh = false;
                }
            }
            since += nc;
            if (since >= kMmaDrain) drain();
        }
    }
    // (a channel that spoils its voxels may have no window after the last drain)
    if (!fresh || drains == 0 || spoiled) drain();

    if (warp >= 2 && __any_sync(0xffffffffu, odd) && lane == 0) *p.nonfinite = 1;
    // copies still in flight land before the CTA leaves
    if (warp == 0 && lane == 0)
        for (uint32_t i = b_issued > kMmaBStages ? b_issued - kMmaBStages : 0; i < b_issued; i++)
            gram_tc::settle(b_full + 8 * (i % kMmaBStages), (i / kMmaBStages) & 1);
    gram_tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        gram_tc::fence_after_sync();
        if (*abort) {
            // products may be in flight: wait (bounded) for them before the columns are released
            if (lane == 0) {
                gram_tc::mma_commit(done);
                gram_tc::settle(done, drains & 1);
            }
            __syncwarp();
        }
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// When the products left a value that is not finite: recomputes every such value
// of the image straight from x, tap by tap, as the direct kernel does.
__global__ void __launch_bounds__(256) mma_fixup_kernel(const mma_params p, const __half *x, int64_t bstride,
                                                        int64_t cstride, int64_t sstride) {
    if (*p.nonfinite == 0) return;   // uniform
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < p.V * p.B; i += (int64_t)gridDim.x * 256) {
        const int b = (int)(i / p.V);
        const int64_t v = i - b * p.V;
        float *o = p.out + (int64_t)b * p.out_bstride + v;
        if (isfinite(*o)) continue;
        const float vx = __ldg(p.dstpos + 3 * v), vy = __ldg(p.dstpos + 3 * v + 1), vz = __ldg(p.dstpos + 3 * v + 2);
        float acc = 0.f;
        for (int c = 0; c < p.C; c++) {
            const float cx = __ldg(p.srcpos + 3 * c), cy = __ldg(p.srcpos + 3 * c + 1), cz = __ldg(p.srcpos + 3 * c + 2);
            recv_geom g = receive_geometry(vx, vy, vz, cx, cy, cz);
            if (p.srcdir) apply_directivity(g, vx, vy, vz, cx, cy, cz, __ldg(p.srcdir + c));
            for (int e = 0; e < p.S; e++) {
                const tau_split ts = split_tau(__fmaf_rn(g.rsq, g.rinv, __ldg(p.offsets + (int64_t)e * p.V + v)));
                float x0 = 0.f, x1 = 0.f;
                if (ts.k < (uint32_t)(p.N - 1)) {
                    const __half *q = x + (int64_t)b * bstride + (int64_t)c * cstride + (int64_t)e * sstride + ts.k;
                    x0 = __half2float(q[0]);
                    x1 = __half2float(q[1]);
                }
                acc = __fmaf_rn(__ldg(p.weights + (int64_t)e * p.V + v), __fmaf_rn(ts.t, x1 - x0, x0), acc);
            }
        }
        *o = acc;
    }
}

// Rows of x copied to rows of Npad samples (a multiple of 8), for data whose
// rows TMA cannot read in place.
__global__ void __launch_bounds__(256) mma_repack_kernel(const __half *__restrict__ x, int64_t bstride, int64_t cstride,
                                                         int64_t sstride, int C, int S, int N, int BC, int Npad,
                                                         __half *__restrict__ out, const int *run_if) {
    const int k0 = (blockIdx.x * 256 + threadIdx.x) * 8;
    if (k0 >= Npad || (run_if && *run_if == 0)) return;
    for (int s = blockIdx.y; s < S; s += gridDim.y)
        for (int bc = blockIdx.z; bc < BC; bc += gridDim.z) {
            const __half *r = x + (int64_t)(bc / C) * bstride + (int64_t)(bc % C) * cstride + (int64_t)s * sstride;
            uint16_t h[8];
#pragma unroll
            for (int i = 0; i < 8; i++) h[i] = k0 + i < N ? __half_as_ushort(r[k0 + i]) : (uint16_t)0;
            *reinterpret_cast<uint4 *>(out + ((int64_t)bc * S + s) * Npad + k0) = *reinterpret_cast<const uint4 *>(h);
        }
}

}  // namespace ffdas
