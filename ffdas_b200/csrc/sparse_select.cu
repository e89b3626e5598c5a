// sparse_select.cu -- ffdas_sparse_select: the per-voxel event lists that a
// das_sparse call sums.
//
// The reference builds das_sparse inputs with its host array library
// (bindings/python/examples/sparse_compounding.py:141-144): per voxel the k
// events with the largest weight (argpartition over the event axis), then the
// weights and delays gathered at them (take_along_axis).  This kernel does the
// same on the device in one pass, one thread per voxel: consecutive threads
// read consecutive voxels, so every row of weights, delays and results is
// read and written in whole cache lines.  The thread keeps the best KC >= k
// entries sorted in registers and takes the events KC at a time: it sorts the
// KC new entries with a merge-exchange network (Batcher, Knuth vol. 3
// algorithm 5.2.2M), keeps the better of each pair best[i], new[KC-1-i] -- the
// KC best of both, a bitonic sequence -- and sorts that with log2(KC) levels
// of half-cleaners.  No lane talks to another and every index is a compile-time
// constant, so the 2 KC entries stay in registers.
//
// Bound by compare-exchange issue (a 64-bit compare and four selects each):
// for 64 events and k = 32, 494 per voxel (16 of 32 merged pairs keep one side
// only), against 672 on 64-bit shuffled keys for a warp-wide bitonic sort of
// 64 entries.  The delays of the tile are copied to shared memory
// asynchronously while the entries are sorted (column tid of row e lies in
// bank tid % 32 whatever the lanes' e, so the gather at the end meets no bank
// conflict).
//
// Order: larger weight first, NaN above every number (the host library sorts
// NaN last in ascending order, so NaN weights are among its k largest), ties
// to the lower event index.  argpartition leaves the order inside the k
// unspecified and may resolve ties differently; das_sparse sums the list, so
// only the rounding of the sum depends on the order.
#include "core.h"

namespace ffdas {

constexpr int kSelectThreads = 128;
constexpr int kSelectMaxK = 32;
// Events whose delays are staged in shared memory (4 bytes x threads each);
// longer lists gather them from global memory.
constexpr int kSelectStaged = 96;

// Entry: key orders the weights (larger ranks first), ns is the complement of
// the event, so that the pair compares as one 64-bit number.
struct select_entry {
    uint32_t key, ns;
};

// The weight's bits mapped to an order-preserving unsigned integer: -0 taken as
// +0, every NaN above +inf.
__device__ __forceinline__ uint32_t select_key(float x) {
    uint32_t u = __float_as_uint(x);
    if (u == 0x80000000u) u = 0u;
    return x != x ? 0xffffffffu : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
}

// a ranks before b: larger key, ties to the lower event.
__device__ __forceinline__ bool select_before(const select_entry &a, const select_entry &b) {
    const unsigned long long ka = ((unsigned long long)a.key << 32) | a.ns;
    const unsigned long long kb = ((unsigned long long)b.key << 32) | b.ns;
    return ka > kb;
}

// Compare-exchange: afterwards a ranks before b.
__device__ __forceinline__ void select_order(select_entry &a, select_entry &b) {
    const bool ok = select_before(a, b);
    const select_entry x = a, y = b;
    a.key = ok ? x.key : y.key;
    a.ns = ok ? x.ns : y.ns;
    b.key = ok ? y.key : x.key;
    b.ns = ok ? y.ns : x.ns;
}

// Sorts n = 2^m entries, best first: for every p = 1, 2, 4, ... n/2 and
// k = p, p/2, ... 1 the pairs (j + i, j + i + k) of Batcher's merge exchange.
template <int KC>
__device__ __forceinline__ void select_sort(select_entry (&e)[KC]) {
#pragma unroll
    for (int p = 1; p < KC; p *= 2) {
#pragma unroll
        for (int k = p; k >= 1; k /= 2) {
#pragma unroll
            for (int i = 0; i < KC; i++) {
                // i is the lower index of a pair of this step
                const int off = i - k % p;
                if (off >= 0 && (off % (2 * k)) < k && i + k < KC && i / (2 * p) == (i + k) / (2 * p))
                    select_order(e[i], e[i + k]);
            }
        }
    }
}

// The KC weights of events s0 .. s0 + KC - 1, and as entries; events past the
// last rank below every real one (key 0 and a higher event than any).
template <int KC>
__device__ __forceinline__ void select_load(const float *__restrict__ w, int s0, int S, int64_t V, float (&x)[KC]) {
#pragma unroll
    for (int i = 0; i < KC; i++) x[i] = s0 + i < S ? __ldg(w + (int64_t)(s0 + i) * V) : 0.f;
}
template <int KC>
__device__ __forceinline__ void select_entries(const float (&x)[KC], int s0, int S, select_entry (&e)[KC]) {
#pragma unroll
    for (int i = 0; i < KC; i++) {
        e[i].key = s0 + i < S ? select_key(x[i]) : 0u;
        e[i].ns = ~(uint32_t)(s0 + i);
    }
}

template <int KC>
__global__ void __launch_bounds__(kSelectThreads) sparse_select_kernel(
    const float *__restrict__ w, const float *__restrict__ offs, int S, int64_t V, int k, bool staged,
    int *__restrict__ idx, float *__restrict__ sw, float *__restrict__ so) {
    extern __shared__ float delays[];   // [S][kSelectThreads] when staged; a thread reads its own column only
    const int tid = threadIdx.x;
    const int64_t v = (int64_t)blockIdx.x * kSelectThreads + tid;
    if (v >= V) return;
    if (staged) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(delays + tid);
        for (int s = 0; s < S; s++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(base + (uint32_t)s * (kSelectThreads * 4)),
                         "l"(offs + (int64_t)s * V + v)
                         : "memory");
    }
    // each group's weights are loaded before the group ahead of it is sorted
    float x[KC], nx[KC];
    select_load<KC>(w + v, 0, S, V, x);
    select_load<KC>(w + v, KC, S, V, nx);
    select_entry best[KC];
    select_entries<KC>(x, 0, S, best);
    select_sort<KC>(best);
    for (int s0 = KC; s0 < S; s0 += KC) {
        select_entry e[KC];
        select_entries<KC>(nx, s0, S, e);
        if (s0 + KC < S) select_load<KC>(w + v, s0 + KC, S, V, nx);
        select_sort<KC>(e);
#pragma unroll
        for (int i = 0; i < KC; i++)
            if (!select_before(best[i], e[KC - 1 - i])) best[i] = e[KC - 1 - i];
#pragma unroll
        for (int d = KC / 2; d >= 1; d /= 2) {
#pragma unroll
            for (int i = 0; i < KC; i++)
                if ((i & d) == 0) select_order(best[i], best[i + d]);
        }
    }
    if (staged) asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int p = 0; p < KC; p++) {
        if (p < k) {
            const int64_t o = (int64_t)p * V + v;
            const uint32_t key = best[p].key, s = ~best[p].ns;
            idx[o] = (int)s;
            if (sw) {
                // the key gives the weight's bits back, except for zeros (either
                // sign) and NaN payloads, which are read again
                float x = __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
                if (key == 0x80000000u || key == 0xffffffffu) x = __ldg(w + (int64_t)s * V + v);
                sw[o] = x;
            }
            if (so) so[o] = staged ? delays[s * kSelectThreads + tid] : __ldg(offs + (int64_t)s * V + v);
        }
    }
}

template <int KC>
static ffdas_error_t launch_select(ffdas_context &h, const float *w, const float *offs, int S, int64_t V, int k,
                                   int *idx, float *sw, float *so) {
    const int64_t blocks = (V + kSelectThreads - 1) / kSelectThreads;
    if (blocks > INT32_MAX) return FFDAS_ERROR_DIMS_TOO_LARGE;
    const bool staged = so && S <= kSelectStaged;
    const size_t smem = staged ? (size_t)S * kSelectThreads * sizeof(float) : 0;   // at most 48 KB
    sparse_select_kernel<KC><<<(unsigned)blocks, kSelectThreads, smem, h.stream>>>(w, offs, S, V, k, staged, idx, sw,
                                                                                   so);
    return ffdas_launch_check(h.stream);
}

}  // namespace ffdas

using namespace ffdas;

extern "C" ffdas_error_t ffdas_sparse_select(ffdas_handle_t handle, const float *weights, const float *offsets,
                                             int n_events, int64_t n_voxels, int k, int *sparse_indices,
                                             float *sparse_weights, float *sparse_offsets) {
    if (!handle) return FFDAS_ERROR_INVALID_HANDLE;
    FFDAS_TRY(handle->check_device());
    if (n_events <= 0 || n_voxels < 0 || k <= 0 || k > n_events || k > kSelectMaxK)
        return FFDAS_ERROR_INVALID_ARGUMENT;
    if (n_voxels == 0) return FFDAS_SUCCESS;
    if (!weights || !sparse_indices || (sparse_offsets && !offsets)) return FFDAS_ERROR_NULL_POINTER;
    ffdas_context &h = *handle;
    const float *offs = sparse_offsets ? offsets : nullptr;
    // KC = the smallest power of two from 4 that holds k: the network and the
    // registers grow with KC, and k entries of KC are written
    if (k <= 4) return launch_select<4>(h, weights, offs, n_events, n_voxels, k, sparse_indices, sparse_weights, sparse_offsets);
    if (k <= 8) return launch_select<8>(h, weights, offs, n_events, n_voxels, k, sparse_indices, sparse_weights, sparse_offsets);
    if (k <= 16) return launch_select<16>(h, weights, offs, n_events, n_voxels, k, sparse_indices, sparse_weights, sparse_offsets);
    return launch_select<32>(h, weights, offs, n_events, n_voxels, k, sparse_indices, sparse_weights, sparse_offsets);
}
