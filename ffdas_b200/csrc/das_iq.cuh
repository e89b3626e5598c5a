// das_iq.cuh -- delay-and-sum of complex (IQ) data on staged windows: forward
// and adjoint, batch tiles of BT items.
//
// The forward adds, per tap, w exp(i wavenum tau) v with v the interpolated
// sample and tau = offset + r (src/das/das_alg1_kernels.cuh:79-99).  The phase
// of a tap splits into one factor per (voxel, event) and one per (voxel,
// channel):
//     exp(i wavenum tau) = E_e R_c,  E_e = exp(i wavenum offset_e),  R_c = exp(i wavenum r_c)
// so a tap's factor is the product of two, one kept in registers for a pass and
// one for a channel: no sine, cosine or range reduction per tap.  Each factor's angle is reduced in turns with the
// wavenumber as a two-part constant, so a phase of thousands of radians keeps
// an absolute error near 2^-21; a single FP32 product wavenum * tau loses
// 2^-24 of its magnitude (1e-4 at 2000 rad).
//
// A complex product is two packed FMAs on (re, im) pairs when the factor's real
// and imaginary part accumulate apart: s1 += (ar, ar) v, s2 += (ai, ai) v, and
// the sum is (s1.re - s2.im, s1.im + s2.re), formed once per voxel.
//
// Ring and producer are those of the real batch tiles (das_staged.cuh): one CTA
// = a 256-voxel tile x BT items, one 4-D TMA box per (channel, event) for the BT
// items' windows.  The windows are plain samples, read from x in place where its
// rows are 16-byte aligned: interpolation pairs are twice the bytes through the
// L2 and shared memory, and an ingest of x (40 us of 343 for 4 frames of 128
// channels, 8 plane waves, 2048 samples), for one subtraction a tap less.
//
// Measured on those frames, 256 x 256 pixels: 207 us, where the gather kernel
// with a sine and cosine per tap took 538 us and its ingest 40; the adjoint of
// two frames, 192 x 256 pixels, 358 us against 1886 for the gather form with
// global atomics.
#pragma once

#include "das_pairs.cuh"
#include "das_staged.cuh"

namespace ffdas {

// The sample rows: x itself or its copy (iq_rows_kernel), strides in samples.
struct iq_rows {
    const void *x;
    int64_t bs, cs, ss;
};

struct iq_params {
    staged_params s;
    iq_rows rows;
    float turn_hi, turn_lo;   // wavenum / (2 pi) as an unevaluated sum
};

template <int K> struct iq_sample {};
template <> struct iq_sample<ST_C32> {
    using type = float2;
    static __device__ __forceinline__ float2 value(float2 a) { return a; }
    static __device__ __forceinline__ float2 store(float2 a) { return a; }
};
template <> struct iq_sample<ST_C16> {
    using type = __half2;
    static __device__ __forceinline__ float2 value(__half2 a) { return __half22float2(a); }
    static __device__ __forceinline__ __half2 store(float2 a) { return __float22half2_rn(a); }
};

// exp(2 pi i (x * turn)) with the turns reduced to [-1/2, 1/2] before the
// sine and cosine are taken.
__device__ __forceinline__ float2 iq_phase(float x, float turn_hi, float turn_lo) {
    const float n = rintf(x * turn_hi);
    float f = __fmaf_rn(x, turn_hi, -n);   // exact up to one rounding
    f = __fmaf_rn(x, turn_lo, f);
    float2 r;
    __sincosf(6.28318530717958647692f * f, &r.y, &r.x);
    return r;
}

template <int WB, int K, int BT, int NW> struct iq_geom {
    static constexpr int sample_bytes = (int)sizeof(typename iq_sample<K>::type);
    static constexpr int units = sample_bytes / 4;          // 4-byte elements of the tensor map
    static constexpr int align = 16 / sample_bytes;         // samples per 16 bytes: a box starts on one
    static constexpr int item_bytes = WB * sample_bytes;
    static constexpr int group_bytes = BT * item_bytes;
    static constexpr int groups = NW / BT;
    static constexpr int stage_bytes = NW * item_bytes;
    static constexpr int ring_bytes = stage_bytes * kStages;
    static_assert(group_bytes % 128 == 0 && groups * BT == NW && NW <= kStWin, "group layout");
    static constexpr size_t smem_bytes = ring_bytes + slot_geom<WB, K>::bytes + kStMiscBytes + 128 + group_bytes;
};

// Sample and slope of a tap at shared-memory address `at` + OFF (x1 - x0 in one
// rounding, as the interpolation pairs hold it).
template <int K, int OFF>
__device__ __forceinline__ void iq_tap(uint32_t at, float2 &x0, float2 &d) {
    float2 x1;
    if constexpr (K == ST_C32) {
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2 + %3];" : "=f"(x0.x), "=f"(x0.y) : "r"(at), "n"(OFF));
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2 + %3];" : "=f"(x1.x), "=f"(x1.y) : "r"(at), "n"(OFF + 8));
    } else {
        uint32_t a, b;
        asm volatile("ld.shared.b32 %0, [%1 + %2];" : "=r"(a) : "r"(at), "n"(OFF));
        asm volatile("ld.shared.b32 %0, [%1 + %2];" : "=r"(b) : "r"(at), "n"(OFF + 4));
        x0 = __half22float2(*reinterpret_cast<__half2 *>(&a));
        x1 = __half22float2(*reinterpret_cast<__half2 *>(&b));
    }
    d = __ffma2_rn(x0, make_float2(-1.f, -1.f), x1);
}
// The same from the rows (a window wider than its slot); k past the record: zeros.
template <int K>
__device__ __forceinline__ void iq_tap_row(const iq_rows &rows, int b, int c, int s, uint32_t k, uint32_t nlast, float2 &x0,
                                           float2 &d) {
    using st = typename iq_sample<K>::type;
    x0 = d = make_float2(0.f, 0.f);
    if (k >= nlast) return;
    const st *r = static_cast<const st *>(rows.x) + b * rows.bs + c * rows.cs + s * rows.ss + k;
    x0 = iq_sample<K>::value(__ldg(r));
    d = __ffma2_rn(x0, make_float2(-1.f, -1.f), iq_sample<K>::value(__ldg(r + 1)));
}

// Producer warp: the windows of one stage (channels c0 .., SC events), one box
// of BT items per (channel, event), as staged_produce_batch.
template <int K, int WB, int SC, int BT, int NW>
__device__ __forceinline__ void iq_produce(const staged_params &p, const CUtensorMap *tmap, staged_smem<K, WB> &sm,
                                           const staged_ctx &cx, int stage, uint32_t phase, int e0, int sc, int c0,
                                           bool &dead, uint32_t &issued_mask) {
    using IG = iq_geom<WB, K, BT, NW>;
    const int cend = chan_end(p);
    const uint32_t full_bar = smem_u32(&sm.full[stage]);
    const uint32_t empty_bar = smem_u32(&sm.empty[stage]);
    const uint32_t stage_u32 = smem_u32(sm.ring + stage * IG::stage_bytes);
    const int lane = cx.lane;
    bool issued = false, overflow = false;
    uint32_t m = kZeroWindow;
    int k0 = 0, c = c0, j = 0;
    float px = 0.f, py = 0.f, pz = 0.f;
    if (lane < IG::groups) {   // everything that needs no ring slot, before waiting for it
        c = c0 + lane / SC;
        j = lane % SC;
        if (c < cend) {
            px = __ldg(p.srcpos + 3 * c);
            py = __ldg(p.srcpos + 3 * c + 1);
            pz = __ldg(p.srcpos + 3 * c + 2);
        }
        if (c < cend && j < sc) {
            const float *ab = sm.aabb;
            const float dx = fmaxf(fmaxf(ab[0] - px, px - ab[3]), 0.f);
            const float dy = fmaxf(fmaxf(ab[1] - py, py - ab[4]), 0.f);
            const float dz = fmaxf(fmaxf(ab[2] - pz, pz - ab[5]), 0.f);
            const float ex = fmaxf(fabsf(px - ab[0]), fabsf(px - ab[3]));
            const float ey = fmaxf(fabsf(py - ab[1]), fabsf(py - ab[4]));
            const float ez = fmaxf(fabsf(pz - ab[2]), fabsf(pz - ab[5]));
            const float rmin = sqrtf(dx * dx + dy * dy + dz * dz);
            const float rmax = sqrtf(ex * ex + ey * ey + ez * ez);
            float lo, hi;
            tap_range(sm.ofs_lo[j], sm.ofs_hi[j], rmin, rmax, lo, hi);
            // taps k of the record: 0 <= k < N - 1, each with its next sample
            if (lo == lo && hi == hi && hi >= 0.f && lo < (float)(p.N - 1)) {
                k0 = (int)fmaxf(lo, 0.f) & ~(IG::align - 1);
                const int k1 = (int)fminf(hi, (float)(p.N - 2));
                if (k1 - k0 + 2 <= WB) {
                    m = kFloorMagicBits + (uint32_t)k0;
                    issued = true;
                } else {
                    m = kOvf;
                    overflow = true;
                }
            }
        }
    }
    if (!dead && !bounded_wait(empty_bar, phase ^ 1u, sm.abort_flag, p.status)) dead = true;
    const bool drop = p.debug_drop_stage && e0 == 0 && c0 == 0;   // test hook, as in staged_produce
    if (drop) dead = true;
    if (dead) issued = overflow = false;
    if (!dead && lane < IG::groups) {
        if (j == 0) {
            const int cl = lane / SC;
            sm.chan_pos[stage * kStWin + cl] = make_float4(px, py, pz, 0.f);
            if (p.srcdir)
                sm.chan_dir[stage * kStWin + cl] = (c < cend) ? __ldg(p.srcdir + c) : make_float4(0, 0, 0, 2.f);
        }
        if (issued)
            tma_load_box4(stage_u32 + lane * IG::group_bytes, tmap, k0 * IG::units, e0 + j, c, cx.b * BT, full_bar);
        sm.meta[stage * kStWin + lane] = m;
    }
    const unsigned issued_ballot = __ballot_sync(0xffffffffu, issued);
    const unsigned ovf_ballot = __ballot_sync(0xffffffffu, overflow);
    __syncwarp();
    if (lane == 0 && !drop) {
        sm.ovf[stage] = ovf_ballot != 0u;
        mbar_arrive_expect_tx(full_bar, (uint32_t)__popc(issued_ballot) * (uint32_t)IG::group_bytes);
    }
    if (!dead) issued_mask |= (1u << stage);
}

// The event factors w E of a pass.  Events past the chunk and voxels past the
// grid have none (their taps read the zero group).
template <int SC>
__device__ __forceinline__ void iq_event_phases(const iq_params &q, bool active, int sc, const float (&ofs)[SC],
                                                float2 (&E)[SC]) {
#pragma unroll
    for (int j = 0; j < SC; j++)
        E[j] = (active && j < sc) ? iq_phase(ofs[j], q.turn_hi, q.turn_lo) : make_float2(0.f, 0.f);
}

// Distance whose phase is a channel's factor.  With directivity a channel
// infinitely far away (its distance is NaN) lies outside every cone and adds
// nothing: it keeps a finite factor.
__device__ __forceinline__ float iq_distance(const recv_geom &g, const float4 *srcdir) {
    const float r = g.rsq * g.rinv;
    return srcdir ? fminf(r, 1e30f) : r;
}

// Floor split of the delays of two events of a channel (SC >= 2), or one.
template <int SC>
__device__ __forceinline__ void iq_split(const recv_geom &g, const float (&ofs)[SC], float (&t)[SC],
                                         uint32_t (&mb)[SC]) {
    if constexpr (SC >= 2) {
        const float2 rsq2 = make_float2(g.rsq, g.rsq), rinv2 = make_float2(g.rinv, g.rinv);
        const float2 magic2 = make_float2(kFloorMagic, kFloorMagic), neg1 = make_float2(-1.f, -1.f);
#pragma unroll
        for (int j = 0; j < SC; j += 2) {
            const float2 tau2 = __ffma2_rn(rsq2, rinv2, make_float2(ofs[j], ofs[j + 1]));
            const float2 mm2 = __fadd2_rd(tau2, magic2);
            const float2 nfl2 = __ffma2_rn(mm2, neg1, magic2);   // -(floor), exact
            const float2 t2 = __fadd2_rn(tau2, nfl2);
            t[j] = t2.x;
            t[j + 1] = t2.y;
            mb[j] = __float_as_uint(mm2.x);
            mb[j + 1] = __float_as_uint(mm2.y);
        }
    } else {
        const float tau = __fmaf_rn(g.rsq, g.rinv, ofs[0]);
        const float mm = __fadd_rd(tau, kFloorMagic);
        t[0] = tau - (mm - kFloorMagic);
        mb[0] = __float_as_uint(mm);
    }
}

// ------------------------------------------------------------------ forward ---
// Bound by issue and the shared-memory path together: a tap reads two samples
// (four wavefronts a warp for FP32) and takes four packed FMAs, and few warps
// hide their latency, so registers are kept to three CTAs per SM: a tap's
// factor w E_e R_c is formed per (channel, event) instead of per-channel sums
// beside the accumulators.
template <int K, int SC, int WB, int BT, int NW>
__global__ void __launch_bounds__(kStThreads, 3) das_iq_kernel(const iq_params q,
                                                               const __grid_constant__ CUtensorMap tmap) {
    const staged_params &p = q.s;
    tile_shape shape;
    if (!take_plan<WB>(p, shape)) return;
    using IG = iq_geom<WB, K, BT, NW>;
    constexpr int CC = IG::groups / SC;   // channels per stage
    static_assert(IG::groups % SC == 0, "SC * BT must divide the stage");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    staged_smem<K, WB> sm(smem_raw, IG::ring_bytes);
    unsigned char *zero_group = sm.extra;
    for (int i = threadIdx.x; i < IG::group_bytes / 4; i += kStThreads) reinterpret_cast<uint32_t *>(zero_group)[i] = 0u;
    const staged_ctx cx = staged_setup<K, WB, false>(p, shape, sm);   // ends with __syncthreads

    const uint32_t ring_u32 = smem_u32(sm.ring), zero_u32 = smem_u32(zero_group);
    const uint32_t nlast = (uint32_t)(p.N - 1);
    const int cbeg = chan_begin(p), cend = chan_end(p);
    float2 acc1[BT], acc2[BT];
#pragma unroll
    for (int b = 0; b < BT; b++) acc1[b] = acc2[b] = make_float2(0.f, 0.f);
    int stage = 0;
    uint32_t phase = 0;
    bool dead = false;
    uint32_t issued_mask = 0;

    for (int e0 = 0; e0 < p.n_events; e0 += SC) {
        const int sc = min(SC, p.n_events - e0);
        float ofs[SC], w[SC];
        staged_pass_begin<K, WB, SC>(p, sm, cx, e0, sc, ofs, w);
        float2 A[SC];
        iq_event_phases<SC>(q, cx.active, sc, ofs, A);
#pragma unroll
        for (int j = 0; j < SC; j++) A[j] = make_float2(A[j].x * w[j], A[j].y * w[j]);

        for (int c0 = cbeg; c0 < cend; c0 += CC) {
            if (cx.producer) {
                iq_produce<K, WB, SC, BT, NW>(p, &tmap, sm, cx, stage, phase, e0, sc, c0, dead, issued_mask);
            } else {
                const uint32_t full_bar = smem_u32(&sm.full[stage]);
                if (!dead && !bounded_wait(full_bar, phase, sm.abort_flag, p.status)) dead = true;
                if (!dead) {
                    // FAST: every window of the stage is staged; decided once per stage,
                    // so that the taps are plain shared-memory loads
                    auto channel = [&](const int cl, auto fast_c) {
                        constexpr bool FAST = decltype(fast_c)::value;
                        const int c = c0 + cl;
                        const float4 cp = sm.chan_pos[stage * kStWin + cl];
                        recv_geom g = receive_geometry(cx.vx, cx.vy, cx.vz, cp.x, cp.y, cp.z);
                        const float2 R = iq_phase(iq_distance(g, p.srcdir), q.turn_hi, q.turn_lo);
                        if (p.srcdir)
                            apply_directivity(g, cx.vx, cx.vy, cx.vz, cp.x, cp.y, cp.z,
                                              sm.chan_dir[stage * kStWin + cl]);
                        uint32_t k0p[SC], mb[SC];
                        float t[SC];
                        load_meta<SC>(sm.meta, stage, cl, k0p);
                        iq_split<SC>(g, ofs, t, mb);
                        const uint32_t groups = ring_u32 + stage * IG::stage_bytes + (cl * SC) * IG::group_bytes;
#pragma unroll
                        for (int j = 0; j < SC; j++) {
                            const float2 W = make_float2(A[j].x * R.x - A[j].y * R.y, __fmaf_rn(A[j].x, R.y, A[j].y * R.x));
                            const float2 wr = make_float2(W.x, W.x), wi = make_float2(W.y, W.y);
                            const float2 t2 = make_float2(t[j], t[j]);
                            const uint32_t rr = mb[j] - k0p[j], k = mb[j] - kFloorMagicBits;
                            if (FAST || k0p[j] != kOvf) {
                                const uint32_t at = rr < (uint32_t)(WB - 1) && k < nlast
                                                        ? groups + j * IG::group_bytes + rr * (uint32_t)IG::sample_bytes
                                                        : zero_u32;
                                static_for<0, BT>([&](auto bic) {
                                    constexpr int b = decltype(bic)::value;
                                    float2 x0, d;
                                    iq_tap<K, b * IG::item_bytes>(at, x0, d);
                                    const float2 v = __ffma2_rn(t2, d, x0);
                                    acc1[b] = __ffma2_rn(wr, v, acc1[b]);
                                    acc2[b] = __ffma2_rn(wi, v, acc2[b]);
                                });
                            } else {
#pragma unroll
                                for (int b = 0; b < BT; b++) {
                                    float2 x0, d;
                                    iq_tap_row<K>(q.rows, min(cx.b * BT + b, p.B - 1), c, e0 + min(j, sc - 1), k, nlast, x0, d);
                                    const float2 v = __ffma2_rn(t2, d, x0);
                                    acc1[b] = __ffma2_rn(wr, v, acc1[b]);
                                    acc2[b] = __ffma2_rn(wi, v, acc2[b]);
                                }
                            }
                        }
                    };
                    const int nch = min(CC, cend - c0);
                    if (*(volatile int *)&sm.ovf[stage] == 0) {
#pragma unroll 1
                        for (int cl = 0; cl < nch; cl++) channel(cl, std::true_type{});
                    } else {
#pragma unroll 1
                        for (int cl = 0; cl < nch; cl++) channel(cl, std::false_type{});
                    }
                }
                __syncwarp();
                if (cx.lane == 0) mbar_arrive(smem_u32(&sm.empty[stage]));
            }
            if (++stage == kStages) {
                stage = 0;
                phase ^= 1u;
            }
        }
        __syncthreads();
    }

    if (cx.producer) {
        staged_drain<K, WB>(sm, cx, stage, phase, issued_mask);
        return;
    }
    if (!cx.active || dead) return;
#pragma unroll
    for (int b = 0; b < BT; b++) {
        const int bb = cx.b * BT + b;
        if (bb >= p.B) break;
        float2 *o = static_cast<float2 *>(p.out) + (int64_t)bb * p.out_bstride + cx.v;
        const float2 acc = make_float2(acc1[b].x - acc2[b].y, acc1[b].y + acc2[b].x);
        if (p.cchunk) atomicAdd(o, acc);   // channel slices add into the prepared image
        else *o = p.beta_zero ? acc : cfma(make_float2((float)p.beta_re, (float)p.beta_im), *o, acc);
    }
}

// out = beta * out (or 0), complex.
__global__ void __launch_bounds__(256) iq_scale_image_kernel(float2 *out, int64_t bstride, int64_t V, int B, float re,
                                                             float im, int zero) {
    const int64_t v = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (v >= V) return;
    for (int b = blockIdx.y; b < B; b += gridDim.y) {
        float2 *o = out + (int64_t)b * bstride + v;
        *o = zero ? make_float2(0.f, 0.f) : cfma(make_float2(re, im), *o, make_float2(0.f, 0.f));
    }
}

// ------------------------------------------------------------------ adjoint ---
// With g the output gradient and h = conj(R_c) g (one product per channel and
// item), u = conj(E_e) h, a tap v = x0 + t d gives
//   weight   Re(conj(g) E R v)           = u . v
//   delay    w Re(conj(g) E R (i k v + d)) = w (u . d + k (u.im v.re - u.re v.im)),  k = wavenum
//   x_k += (1 - t) w u,  x_{k+1} += t w u
// (a . b the dot product of (re, im)), and the delay term times (v - c) / r for
// the two position sets.  The scatter is the real adjoint's: fixed point of
// 2^22 / amax in shared-memory bins (here a real and an imaginary plane per
// window), two copies by the voxel's checkerboard parity, two sets by stage
// parity, one vector atomic per touched sample at the flush; overflowing
// windows and passes without a positive finite amax add to global memory.
template <int WB, int K, int SC, int BT, int NW>
struct iq_bwd_layout {
    using IG = iq_geom<WB, K, BT, NW>;
    static constexpr int CC = IG::groups / SC;
    static constexpr int GS = bin_stride(WB);
    static constexpr int region = bin_region_words(2 * NW * GS);   // words of one copy
    static constexpr int set = kBinCopies * region;
    static constexpr int cg = CC * 3 * kStConsumers;               // floats of one channel-gradient set
    static constexpr size_t zero_off = ((size_t)(2 * set + 2 * cg + kStWarps) * 4 + 15) & ~size_t(15);
    static constexpr size_t smem_bytes =
        IG::ring_bytes + slot_geom<WB, K>::bytes + kStMiscBytes + 128 + zero_off + IG::group_bytes;
};

// Adds the bins of one stage into gx and clears them: WB / 4 lanes take a
// window, four samples each with 128-bit shared accesses.  row(win, kw) gives
// the window's gx row (null: nothing to add) and first sample.
template <int WB, int REGION, int NW, class RowFn>
__device__ __forceinline__ void iq_flush_bins(int *bins0, int lane, int warp, float finv, int n, RowFn &&row) {
    constexpr int GS = bin_stride(WB);
    constexpr int LPW = WB / 4, WPI = 32 / LPW;
    static_assert(WB % 4 == 0 && 32 % LPW == 0 && REGION % 4 == 0, "flush layout");
    const int sub = lane / LPW, l = lane % LPW;
    for (int w0 = warp * WPI; w0 < NW; w0 += kStWarps * WPI) {
        const int win = w0 + sub;
        int s[2][4], last[2] = {0, 0};
#pragma unroll
        for (int a = 0; a < 2; a++) {
            int *b = bins0 + (2 * win + a) * GS + 4 * l;
            const int4 u = *reinterpret_cast<const int4 *>(b);
            const int4 v = *reinterpret_cast<const int4 *>(b + REGION);
            *reinterpret_cast<int4 *>(b) = make_int4(0, 0, 0, 0);
            *reinterpret_cast<int4 *>(b + REGION) = make_int4(0, 0, 0, 0);
            s[a][0] = u.x + v.x; s[a][1] = u.y + v.y; s[a][2] = u.z + v.z; s[a][3] = u.w + v.w;
            if (l == 0) {
                int *e = bins0 + (2 * win + a) * GS + WB;
                last[a] = e[0] + e[REGION];
                e[0] = 0;
                e[REGION] = 0;
            }
        }
        int kw;
        float2 *g = row(win, kw);
        if (g) {
            g += kw + 4 * l;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (s[0][i] | s[1][i]) atomicAdd(g + i, make_float2((float)s[0][i] * finv, (float)s[1][i] * finv));
            // (not past the row: see flush_bins)
            if ((last[0] | last[1]) && kw + WB < n)
                atomicAdd(g + WB, make_float2((float)last[0] * finv, (float)last[1] * finv));
        }
    }
}

template <int K, int SC, int WB, int BT, int NW>
__global__ void __launch_bounds__(kStThreads, 2) das_iq_bwd_kernel(const iq_params qp,
                                                                   const __grid_constant__ CUtensorMap tmap) {
    const staged_params &p = qp.s;
    tile_shape shape;
    if (!take_plan<WB>(p, shape)) return;
    using IG = iq_geom<WB, K, BT, NW>;
    using L = iq_bwd_layout<WB, K, SC, BT, NW>;
    constexpr int CC = L::CC, GS = L::GS;
    static_assert(IG::groups % SC == 0 && kStages % 2 == 0, "stage layout");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    staged_smem<K, WB> sm(smem_raw, IG::ring_bytes);
    int *gslot = reinterpret_cast<int *>(sm.extra);                    // [2][kBinCopies][window][re, im][GS]
    float *cgrad0 = reinterpret_cast<float *>(gslot + 2 * L::set);     // [2][CC * 3][256]
    float *wmax = cgrad0 + 2 * L::cg;                                  // [kStWarps]
    unsigned char *zero_group = sm.extra + L::zero_off;
    for (int i = threadIdx.x; i < 2 * L::set; i += kStThreads) gslot[i] = 0;
    for (int i = threadIdx.x; i < IG::group_bytes / 4; i += kStThreads) reinterpret_cast<uint32_t *>(zero_group)[i] = 0u;
    const staged_ctx cx = staged_setup<K, WB, false>(p, shape, sm, true);     // ends with __syncthreads
    const uint32_t ring_u32 = smem_u32(sm.ring), zero_u32 = smem_u32(zero_group);
    const uint32_t gslot_u32 = smem_u32(gslot) + cx.par * (L::region * 4);

    const float2 *gout = reinterpret_cast<const float2 *>(p.gout);
    float2 *gx = reinterpret_cast<float2 *>(p.gx);
    const int b0 = cx.b * BT;
    const bool multi = gridDim.y > 1 || gridDim.z > 1;   // several CTAs add into the voxel-side gradients
    const int cbeg = chan_begin(p), cend = chan_end(p);
    const uint32_t nlast = (uint32_t)(p.N - 1);
    float2 g[BT];
    float gmax = 0.f;
    bool gbad = false;
#pragma unroll
    for (int b = 0; b < BT; b++) {
        g[b] = (cx.active && b0 + b < p.B) ? __ldg(gout + (int64_t)(b0 + b) * p.gout_bstride + cx.v)
                                           : make_float2(0.f, 0.f);
        const float a = sqrtf(__fmaf_rn(g[b].x, g[b].x, g[b].y * g[b].y)) * 1.00001f;   // bounds |Re u|, |Im u|
        gbad |= !(a <= 3.0e38f);
        gmax = fmaxf(gmax, a);
    }
    const bool want_pos = p.gdst != nullptr || p.gsrc != nullptr;
    float gpx = 0.f, gpy = 0.f, gpz = 0.f;
    int stage = 0;
    uint32_t phase = 0;
    bool dead = false;
    uint32_t issued_mask = 0;

    for (int e0 = 0; e0 < p.n_events; e0 += SC) {
        const int sc = min(SC, p.n_events - e0);
        float ofs[SC], w[SC];
        staged_pass_begin<K, WB, SC>(p, sm, cx, e0, sc, ofs, w);
        float2 E[SC];
        iq_event_phases<SC>(qp, cx.active, sc, ofs, E);
        float sw[SC], so[SC];   // per event: sums of u . v and of the delay term over channels and items
#pragma unroll
        for (int j = 0; j < SC; j++) sw[j] = so[j] = 0.f;
        float fscale = 0.f, finv = 0.f;
        bool fixed = false;
        if (!cx.producer) {   // amax = max |g| max |w| over the tile, as in the real adjoint
            float wm = 0.f;
            bool bad = gbad;
#pragma unroll
            for (int j = 0; j < SC; j++) {
                wm = fmaxf(wm, fabsf(w[j]));
                bad |= !(fabsf(w[j]) <= 3.0e38f);
            }
            float m = gmax * wm;
            bad |= !(m <= 3.0e38f);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            bad = __any_sync(0xffffffffu, bad);
            if (cx.lane == 0) wmax[cx.warp] = bad ? -1.f : m;
            consumer_sync();
            float amax = 0.f;
            bool any_bad = false;
#pragma unroll
            for (int i = 0; i < kStWarps; i++) {
                const float v = wmax[i];
                any_bad |= v < 0.f;
                amax = fmaxf(amax, v);
            }
            fixed = !any_bad && amax > 0.f && amax <= 3.0e38f;
            if (fixed) {
                fscale = kFixRange / amax;
                finv = amax / kFixRange;
                fixed = fscale <= 3.0e38f;   // a subnormal amax has no scale
            }
            consumer_sync();   // wmax is rewritten by the next pass
        }

        for (int c0 = cbeg; c0 < cend; c0 += CC) {
            if (cx.producer) {
                iq_produce<K, WB, SC, BT, NW>(p, &tmap, sm, cx, stage, phase, e0, sc, c0, dead, issued_mask);
            } else {
                const uint32_t full_bar = smem_u32(&sm.full[stage]);
                int *gstage = gslot + (stage & 1) * L::set;
                const uint32_t gstage_u32 = gslot_u32 + (stage & 1) * (L::set * 4);
                float *cgrad = cgrad0 + (stage & 1) * L::cg;
                if (!dead && !bounded_wait(full_bar, phase, sm.abort_flag, p.status)) dead = true;
                const bool any_ovf = !dead && *(volatile int *)&sm.ovf[stage] != 0;
                if (!dead) {
                    // FAST: every window of the stage is staged and the scatter, if
                    // wanted (SCATTER), is fixed point; decided once per stage
                    auto channel = [&](const int cl, auto fast_c, auto scatter_c) {
                        constexpr bool FAST = decltype(fast_c)::value;
                        constexpr bool SCATTER = decltype(scatter_c)::value;
                        const int c = c0 + cl;
                        const float4 cp = sm.chan_pos[stage * kStWin + cl];
                        recv_geom gm = receive_geometry(cx.vx, cx.vy, cx.vz, cp.x, cp.y, cp.z);
                        const float2 R = iq_phase(iq_distance(gm, p.srcdir), qp.turn_hi, qp.turn_lo);
                        if (p.srcdir)
                            apply_directivity(gm, cx.vx, cx.vy, cx.vz, cp.x, cp.y, cp.z,
                                              sm.chan_dir[stage * kStWin + cl]);
                        float2 h[BT];
#pragma unroll
                        for (int b = 0; b < BT; b++)
                            h[b] = make_float2(__fmaf_rn(R.x, g[b].x, R.y * g[b].y), __fmaf_rn(R.x, g[b].y, -R.y * g[b].x));
                        uint32_t k0p[SC], mb[SC];
                        float t[SC];
                        load_meta<SC>(sm.meta, stage, cl, k0p);
                        iq_split<SC>(gm, ofs, t, mb);
                        const uint32_t groups = ring_u32 + stage * IG::stage_bytes + (cl * SC) * IG::group_bytes;
                        const uint32_t gwin_u32 = gstage_u32 + (cl * SC * BT) * 2 * GS * 4;
                        float q = 0.f;
#pragma unroll
                        for (int j = 0; j < SC; j++) {
                            const uint32_t rr = mb[j] - k0p[j];
                            const bool in_rec = mb[j] - kFloorMagicBits < nlast;
                            const uint32_t at = rr < (uint32_t)(WB - 1) && in_rec
                                                    ? groups + j * IG::group_bytes + rr * (uint32_t)IG::sample_bytes
                                                    : zero_u32;
                            const bool ovfw = !FAST && k0p[j] == kOvf;
                            // a tap outside the record scatters zeros (into its window's
                            // bins, or the zero-only bin past the window)
                            const float ws = in_rec ? w[j] * fscale : 0.f;
                            const float wst = ws * t[j];
                            const uint32_t gb = gwin_u32 + (j * BT * 2 * GS + min(rr, (uint32_t)WB)) * 4;
                            float qj = 0.f, qx = 0.f;
                            static_for<0, BT>([&](auto bic) {
                                constexpr int b = decltype(bic)::value;
                                float2 x0, d;
                                if (FAST || !ovfw)
                                    iq_tap<K, b * IG::item_bytes>(at, x0, d);
                                else
                                    iq_tap_row<K>(qp.rows, min(b0 + b, p.B - 1), c, e0 + min(j, sc - 1),
                                                  mb[j] - kFloorMagicBits, nlast, x0, d);
                                const float2 v = __ffma2_rn(make_float2(t[j], t[j]), d, x0);
                                const float2 u = make_float2(__fmaf_rn(E[j].x, h[b].x, E[j].y * h[b].y),
                                                             __fmaf_rn(E[j].x, h[b].y, -E[j].y * h[b].x));
                                sw[j] = __fmaf_rn(u.x, v.x, __fmaf_rn(u.y, v.y, sw[j]));
                                qj = __fmaf_rn(u.x, d.x, __fmaf_rn(u.y, d.y, qj));
                                qx = __fmaf_rn(u.y, v.x, __fmaf_rn(-u.x, v.y, qx));
                                if constexpr (FAST && SCATTER) {
                                    const int ax = fix_bits_fma(u.x, ws), bx = fix_bits_fma(u.x, wst);
                                    const int ay = fix_bits_fma(u.y, ws), by = fix_bits_fma(u.y, wst);
                                    red_shared_add_at<b * 2 * GS * 4>(gb, ax - bx);
                                    red_shared_add_at<b * 2 * GS * 4 + 4>(gb, bx - (int)kFloorMagicBits);
                                    red_shared_add_at<(b * 2 + 1) * GS * 4>(gb, ay - by);
                                    red_shared_add_at<(b * 2 + 1) * GS * 4 + 4>(gb, by - (int)kFloorMagicBits);
                                } else if constexpr (!FAST) {
                                    if (gx && in_rec && w[j] != 0.f && b0 + b < p.B) {
                                        if (fixed && !ovfw && rr < (uint32_t)(WB - 1)) {
                                            const int ax = fix_bits_fma(u.x, ws), bx = fix_bits_fma(u.x, wst);
                                            const int ay = fix_bits_fma(u.y, ws), by = fix_bits_fma(u.y, wst);
                                            red_shared_add_at<b * 2 * GS * 4>(gb, ax - bx);
                                            red_shared_add_at<b * 2 * GS * 4 + 4>(gb, bx - (int)kFloorMagicBits);
                                            red_shared_add_at<(b * 2 + 1) * GS * 4>(gb, ay - by);
                                            red_shared_add_at<(b * 2 + 1) * GS * 4 + 4>(gb, by - (int)kFloorMagicBits);
                                        } else {
                                            const float cx_ = w[j] * u.x, cy_ = w[j] * u.y;
                                            float2 *gr = gx + (((int64_t)(b0 + b) * p.C + c) * p.S + (e0 + j)) * p.N +
                                                         (mb[j] - kFloorMagicBits);
                                            atomicAdd(gr, make_float2(cx_ - cx_ * t[j], cy_ - cy_ * t[j]));
                                            atomicAdd(gr + 1, make_float2(cx_ * t[j], cy_ * t[j]));
                                        }
                                    }
                                }
                            });
                            qj = __fmaf_rn(p.wavenum, qx, qj);
                            so[j] += qj;
                            q = __fmaf_rn(w[j], qj, q);
                        }
                        if (want_pos) {
                            const float qr = q * gm.rinv;
                            const float ex = (cx.vx - cp.x) * qr, ey = (cx.vy - cp.y) * qr, ez = (cx.vz - cp.z) * qr;
                            gpx += ex; gpy += ey; gpz += ez;
                            if (p.gsrc) {
                                cgrad[(cl * 3 + 0) * kStConsumers + cx.tid] = -ex;
                                cgrad[(cl * 3 + 1) * kStConsumers + cx.tid] = -ey;
                                cgrad[(cl * 3 + 2) * kStConsumers + cx.tid] = -ez;
                            }
                        }
                    };
                    auto run = [&](auto fast_c, auto scatter_c) {
#pragma unroll 1
                        for (int cl = 0; cl < CC; cl++) {
                            if (c0 + cl >= cend) break;
                            channel(cl, fast_c, scatter_c);
                        }
                    };
                    if (any_ovf || (gx && !fixed)) run(std::false_type{}, std::false_type{});
                    else if (gx) run(std::true_type{}, std::true_type{});
                    else run(std::true_type{}, std::false_type{});
                }
                consumer_sync();   // every consumer warp finished this stage's scatter
                if (!dead) {
                    if (gx && fixed) {
                        iq_flush_bins<WB, L::region, NW>(gstage, cx.lane, cx.warp, finv, p.N, [&](int win, int &kw) -> float2 * {
                            const int grp = win / BT, b = win % BT;
                            const int cl = grp / SC, j = grp % SC;
                            kw = (int)(sm.meta[stage * kStWin + grp] - kFloorMagicBits);
                            if (b0 + b >= p.B || c0 + cl >= cend) return nullptr;
                            return gx + (((int64_t)(b0 + b) * p.C + (c0 + cl)) * p.S + (e0 + j)) * p.N;
                        });
                    }
                    if (p.gsrc) {
                        for (int o = cx.warp; o < CC * 3; o += kStWarps) {
                            const int cl = o / 3;
                            if (c0 + cl >= cend) continue;
                            float s = 0.f;
#pragma unroll
                            for (int i = 0; i < kStConsumers / 32; i++) s += cgrad[o * kStConsumers + cx.lane + 32 * i];
#pragma unroll
                            for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
                            if (cx.lane == 0 && s != 0.f) atomicAdd(p.gsrc + 3 * (c0 + cl) + (o % 3), s);
                        }
                    }
                }
                // no barrier: the next stage uses the other set of scratch
                __syncwarp();
                if (cx.lane == 0) mbar_arrive(smem_u32(&sm.empty[stage]));
            }
            if (++stage == kStages) {
                stage = 0;
                phase ^= 1u;
            }
        }
        if (!cx.producer && cx.active && !dead) {
#pragma unroll
            for (int j = 0; j < SC; j++) {
                if (j < sc) {
                    const int64_t idx = (int64_t)(e0 + j) * p.V + cx.v;
                    const float gov = w[j] * so[j];
                    if (multi) {
                        if (p.gw) atomicAdd(p.gw + idx, sw[j]);
                        if (p.goff) atomicAdd(p.goff + idx, gov);
                    } else {
                        if (p.gw) p.gw[idx] = sw[j];
                        if (p.goff) p.goff[idx] = gov;
                    }
                }
            }
        }
        __syncthreads();
    }

    if (cx.producer) {
        staged_drain<K, WB>(sm, cx, stage, phase, issued_mask);
        return;
    }
    if (cx.active && !dead && p.gdst) {
        if (multi) {
            atomicAdd(p.gdst + 3 * cx.v, gpx);
            atomicAdd(p.gdst + 3 * cx.v + 1, gpy);
            atomicAdd(p.gdst + 3 * cx.v + 2, gpz);
        } else {
            p.gdst[3 * cx.v] = gpx;
            p.gdst[3 * cx.v + 1] = gpy;
            p.gdst[3 * cx.v + 2] = gpz;
        }
    }
}

// x (any strides, with an optional per-channel gain, rounded to the sample type)
// as rows of Npad samples, zeros past the record.
template <typename Tin, int K>
__global__ void __launch_bounds__(256) iq_rows_kernel(const Tin *__restrict__ x, int64_t bstride, int64_t cstride,
                                                      int64_t sstride, int C, int S, int N, int BC, int Npad,
                                                      const float *__restrict__ gain, int gain_bstride,
                                                      typename iq_sample<K>::type *__restrict__ out) {
    const int k0 = (blockIdx.x * 256 + threadIdx.x) * 4;
    if (k0 >= Npad) return;
    struct alignas(16) quad { typename iq_sample<K>::type v[4]; };
    for (int s = blockIdx.y; s < S; s += gridDim.y)
        for (int bc = blockIdx.z; bc < BC; bc += gridDim.z) {
            const int c = bc % C, b = bc / C;
            const Tin *r = x + (int64_t)b * bstride + (int64_t)c * cstride + (int64_t)s * sstride;
            const float g = gain ? __ldg(gain + (int64_t)b * gain_bstride + c) : 1.f;
            quad f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float2 v = k0 + i < N ? to_c32(sample_io<Tin>::load(r + k0 + i)) : make_float2(0.f, 0.f);
                if (gain) v = scaled(v, g);
                f.v[i] = iq_sample<K>::store(v);
            }
            *reinterpret_cast<quad *>(out + ((int64_t)bc * S + s) * Npad + k0) = f;
        }
}

}  // namespace ffdas
