// das_tile_plan.cuh -- tile shape and window width chosen from the geometry.
//
// A staged kernel copies, per (tile, channel, event), one window of WB
// samples; a window that would have to be wider is read tap by tap from global
// memory, several times slower.  How wide the windows get depends on the pixel
// pitch, which only the device knows: a 32 x 16 tile of a frame with 1.6
// samples between rows spans 52 two-way samples, the same tile of a
// micrometre-sampled region fits 32.  So one block samples the grid before the
// staged kernels run: for every candidate shape it bounds the windows of nine
// tiles (three along each in-plane axis) x five channels x three events the
// way the producers do, and picks the shape and width with the least
//     padded voxels x cost(WB) x (1 + kPlanSlow * share of stages with a window too wide).
// The staged kernels, launched for both widths, read the choice; the instance
// of the other width returns at once.
// Measured on 401 x 255 pixels, 127 channels, 11 plane waves (B200): 398 us on
// the fixed 32 x 16 tile, whose windows all overflow 32 samples; 134 us on the
// plan's 32 x 16 tile with windows of 64.
#pragma once

#include "das_staged.cuh"

namespace ffdas {

constexpr int kPlanShapes = 8;
constexpr int kPlanAnchors = 9, kPlanEvents = 3, kPlanChannels = 5;
constexpr int kPlanThreads = kPlanShapes * kPlanAnchors * kPlanEvents;   // 216
// A too-wide window slows its whole stage (8 channels x 4 events), so what counts
// is the share of (tile, channel) pairs with one at any event: 1.7 times the
// rest's cost (173 channels, 9 plane waves, rows 2.9 samples apart: 42 % of the
// stages slow 233 us, all of them 290; 196 us since two events' pairs are loaded at a
// time, and 1.2 or 2.5 in place of 1.7 change the mean of 190 frames and volumes by
// less than 0.2 %), more in the adjoints, whose bins it bypasses.
constexpr float kPlanSlow = 1.7f, kPlanSlowAdjoint = 4.f;
// 64-sample windows against 32: twice the bytes and two instead of three CTAs
// per SM (784 channels, 3 waves, 96 x 86 x 86 voxels: 1.21 to 1.34 ms); in the
// adjoints the gradient bins double as well
constexpr float kPlanWide = 1.15f, kPlanWideAdjoint = 1.3f;
// Batch tiles whose windows all overflow against ones whose windows fit: 5.4 times
// the time (56 items, 192 channels, 8 events, 100 x 64 pixels: 2.78 ms).
constexpr float kPlanSlowBatch = 4.4f;

struct plan_params {
    const float *srcpos, *dstpos, *offsets;
    int C, n_events, align;    // align: pairs per 16 bytes
    int64_t V, npad;
    int D0, D1, D2;
    int shapes;
    int T0[kPlanShapes], T1[kPlanShapes];
    int mode;   // kPlanForward, kPlanBatch, kPlanAdjoint or kPlanMma
    float products_above;   // kPlanBatch: padding x overflow above which the products run (0: never)
    tile_plan *plan;
};

// By one block of at least kPlanThreads threads.
__device__ __forceinline__ void tile_plan_block(const plan_params &q) {
    // per (shape, anchor tile): the channels with a window too wide at any event
    __shared__ int over[2][kPlanShapes][kPlanAnchors], wide[kPlanShapes];
    const int tid = threadIdx.x;
    if (tid < kPlanShapes * kPlanAnchors) over[0][tid / kPlanAnchors][tid % kPlanAnchors] = over[1][tid / kPlanAnchors][tid % kPlanAnchors] = 0;
    if (tid < kPlanShapes) wide[tid] = 0;
    __syncthreads();
    const int sh = tid / (kPlanAnchors * kPlanEvents), an = (tid / kPlanEvents) % kPlanAnchors, ei = tid % kPlanEvents;
    if (sh < q.shapes) {
        const int T0 = q.T0[sh], T1 = q.T1[sh];
        const int n0 = (q.D0 + T0 - 1) / T0, n1 = (q.D1 + T1 - 1) / T1;
        const int a0 = an % 3, a1 = an / 3;
        const int g0 = (n0 - 1) * a0 / 2 * T0, g1 = (n1 - 1) * a1 / 2 * T1, g2 = (q.D2 - 1) * ((a0 + a1) % 3) / 2;
        const int x1 = min(g0 + T0, q.D0) - 1, y1 = min(g1 + T1, q.D1) - 1;
        const int64_t e = (int64_t)(q.n_events - 1) * ei / 2;
        float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
        float olo = INFINITY, ohi = -INFINITY;
#pragma unroll
        for (int i = 0; i < 9; i++) {   // the tile's corners, edge midpoints and centre
            const int x = g0 + (x1 - g0) * (i % 3) / 2, y = g1 + (y1 - g1) * (i / 3) / 2;
            const int64_t v = ((int64_t)g2 * q.D1 + y) * q.D0 + x;
            const float o = __ldg(q.offsets + e * q.V + v);
            olo = fminf(olo, o);
            ohi = fmaxf(ohi, o);
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const float c = __ldg(q.dstpos + 3 * v + a);
                mn[a] = fminf(mn[a], c);
                mx[a] = fmaxf(mx[a], c);
            }
        }
        float pos[kPlanChannels][3];
#pragma unroll
        for (int ci = 0; ci < kPlanChannels; ci++) {
            const int64_t c = (int64_t)(q.C - 1) * ci / (kPlanChannels - 1);
#pragma unroll
            for (int a = 0; a < 3; a++) pos[ci][a] = __ldg(q.srcpos + 3 * c + a);
        }
        int m32 = 0, m64 = 0, wsum = 0;
#pragma unroll
        for (int ci = 0; ci < kPlanChannels; ci++) {
            float n2 = 0.f, x2 = 0.f;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const float p = pos[ci][a];
                const float gap = fmaxf(fmaxf(mn[a] - p, p - mx[a]), 0.f);
                const float ext = fmaxf(fabsf(p - mn[a]), fabsf(p - mx[a]));
                n2 += gap * gap;
                x2 += ext * ext;
            }
            const float lo = floorf(olo + sqrtf(n2)) - 2.f, hi = floorf(ohi + sqrtf(x2)) + 2.f;
            if (hi < 0.f || lo >= (float)q.npad) continue;   // outside the record: no copy
            // a non-finite bound counts as too wide, for every shape alike
            const float w = hi - lo + (float)q.align;
            m32 |= !(w <= 32.f) << ci;
            m64 |= !(w <= 64.f) << ci;
            wsum += (int)fminf(fmaxf(w, 0.f), 4096.f);
        }
        if (m32) atomicOr(&over[0][sh][an], m32);
        if (m64) atomicOr(&over[1][sh][an], m64);
        atomicAdd(&wide[sh], wsum);
    }
    __syncthreads();
    if (tid >= 32) return;   // (no barrier below)
    // a lane per (shape, width); the least cost wins, ties to the lower lane
    constexpr float kSamples = (float)(kPlanAnchors * kPlanEvents * kPlanChannels);
    const int i = tid >> 1, wb = (tid & 1) ? 64 : 32;
    float cost = INFINITY, batch = 0.f;
    if (i < q.shapes) {
        const int n0 = (q.D0 + q.T0[i] - 1) / q.T0[i], n1 = (q.D1 + q.T1[i] - 1) / q.T1[i];
        const float waste = (float)(n0 * q.T0[i]) * (float)(n1 * q.T1[i]) / ((float)q.D0 * (float)q.D1);
        int n = 0;
        for (int a = 0; a < kPlanAnchors; a++) n += __popc(over[tid & 1][i][a]);
        const float slow = (float)n / (float)(kPlanAnchors * kPlanChannels);
        batch = waste * (1.f + kPlanSlowBatch * slow);
        if (q.mode == kPlanMma) {
            // the products grow with the windows, whatever their width; the
            // image is read and written in rows of T0 voxels
            cost = wb == 32 ? waste * ((float)wide[i] / kSamples + 16.f) * (q.T0[i] < 16 ? 1.2f : 1.f) : INFINITY;
        } else {
            // (the batch tiles run 64-sample windows only: 32-sample ones are
            // no faster there, 144 against 139 us on the autofocus frames)
            const bool adjoint = q.mode == kPlanAdjoint;
            const float width = wb == 32 ? 1.f : (adjoint ? kPlanWideAdjoint : kPlanWide);
            cost = (q.mode == kPlanBatch && wb == 32)
                       ? INFINITY
                       : waste * width * (1.f + (adjoint ? kPlanSlowAdjoint : kPlanSlow) * slow);
            // near ties: the forward takes the squarer tile (ties to the wider; a
            // 32 x 8 tile of 3 % less padding ran 10 % slower than 16 x 16),
            // the adjoint the shape nearest 8 x 32, whose scatter meets the
            // fewest equal samples where the second axis is depth
            const int l0 = __ffs(q.T0[i]), l1 = __ffs(q.T1[i]);
            cost += adjoint ? 0.02f * fabsf((float)(l0 - 4)) : 0.04f * fabsf((float)(l0 - l1) - 0.5f);
        }
    }
    int best = tid;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float c = __shfl_xor_sync(0xffffffffu, cost, o);
        const int l = __shfl_xor_sync(0xffffffffu, best, o);
        if (c < cost || (c == cost && l < best)) {
            cost = c;
            best = l;
        }
    }
    batch = __shfl_sync(0xffffffffu, batch, best);
    if (tid != 0) return;
    const int k = best >> 1;
    tile_plan pl;
    pl.T0 = q.T0[k];
    pl.T1 = q.T1[k];
    pl.n0 = (q.D0 + pl.T0 - 1) / pl.T0;
    pl.n1 = (q.D1 + pl.T1 - 1) / pl.T1;
    pl.products = q.products_above > 0.f && batch > q.products_above;
    pl.wb = pl.products ? 0 : ((best & 1) ? 64 : 32);
    pl.nonfinite = 0;
    *q.plan = pl;
}

// One block per plan: a call's own, and where the pair rows are kept for a
// backward, that of the adjoint.  The ingest launched next overlaps it
// (programmatic launch): it needs nothing of the plan, and a plan takes as long
// as the ingest of a frame (4 us).  Made by the ingest's first block instead it
// took 10 us, and its registers cost the ingest occupancy (volume: 121 -> 150 us).
static __global__ void __launch_bounds__(256) tile_plan_kernel(const plan_params own, const plan_params adjoint) {
    asm volatile("griddepcontrol.launch_dependents;");
    tile_plan_block(blockIdx.x == 0 ? own : adjoint);
}

}  // namespace ffdas
