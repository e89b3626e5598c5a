// das_entries.cuh -- das_sparse with a lane per list entry on staged windows.
//
// A voxel's list names its own events, so a thread that owns a voxel reads a
// different row at every list place than its neighbours: 32 sectors per warp
// load, bound by the L2 (0.67 ms for 2.2e8 units of the focused 64-transmit
// frame).  Here the entries of a 1024-voxel tile are sorted by event first
// (entries_sort_kernel, once per call), and the beamforming kernel takes them
// 512 at a time in sorted order, two per lane in the packed FP32 halves.  Such a
// run meets few events, so one window per (channel, event), staged by TMA
// through an mbarrier ring, serves hundreds of taps from shared memory; no lane
// works on a padding entry, an entry's sum over the channels stays in registers,
// and it is added to its voxel once.  Lists may name an event twice.
//
// The windows are plain samples, 128 of 4 bytes: a tap reads its two samples and
// subtracts, one more load and add than an interpolation pair, but the copies
// out of the L2 set the pace (1.9 GB a call with 64-pair windows: 0.45 ms at
// 4.2 TB/s), and a sample row is half a pair row; FP32 data with 16-byte rows
// is read in place, with no ingest.  A stage holds D x G windows: the D buckets
// of the run and G = 8, 4, 2 or 1 consecutive channels, whose windows of one
// bucket start at the same sample so that one box {128 samples, G channels}
// copies them.  Where every tap of a stage lies inside its window and, with its
// next sample, inside the record or outside it altogether, its address is one
// multiply-add of the floor bits and the bucket's bias; other stages test each
// tap, and a window that would have to be wider than 128 samples is read from
// the rows.
//
// The tile is cut into NB blocks of consecutive voxels and a bucket holds the
// entries of one (block, event), so that the block's extent, not the tile's,
// sets the window: the sort takes the smallest NB whose blocks' windows fit
// (delays change by at most one sample per wavelength of distance, which bounds
// the transmit part).
//
// Measured on that frame: sort 38 us, this kernel 351 us, against 656 us for the
// gather kernel and 32 for its ingest.  Below 2^27 list places x channels x items
// (2^24 from 256 channels on) the gather kernel's shorter chain wins (138 channels,
// 12 of 24 events, 166 x 170 pixels: 109 against 149 us), and with under a quarter of the events listed a window serves too few
// entries (20 of 100: 402 against 412).
#pragma once

#include "das_staged.cuh"

namespace ffdas {

constexpr int kEnTile = 1024;       // voxels per tile
constexpr int kEnBlocks = 8;        // most blocks of a tile
constexpr int kEnMaxList = 64;      // list length
constexpr int kEnMaxEvents = 480;   // events of x (the sort's tables: 64 bytes each)
constexpr int kEnRun = 512;         // entries per run: two per consumer lane
constexpr int kEnSlots = 32;        // most buckets of a run (one producer lane each)
constexpr int kEnWB = 128;          // samples per window
constexpr int kEnStages = 3;
constexpr int kEnChannels = 8;      // most channels of a stage

// One nonempty bucket of a tile: its first entry, event and block, and the
// range of its finite delays.
struct __align__(16) en_slot {
    int start, event_block;   // event | block << 16
    float lo, hi;
};
struct __align__(16) en_tile {
    int slots, entries;
    int pad[2];
    float box[kEnBlocks][6];  // voxel positions of each block (min xyz, max xyz); blocks past NB unused
    int pad2[12];             // 256 bytes
};
struct __align__(16) en_entry {
    float ofs, w;
    uint32_t key;             // voxel of the tile | bucket << 16
    uint32_t pad;
};

// The sample rows: x itself or its copy (entry_rows_kernel), strides in samples.
struct en_rows {
    const float *x;
    int64_t bs, cs, ss;
    __device__ __forceinline__ const float *row(int b, int c, int s) const { return x + b * bs + c * cs + s * ss; }
};

struct en_params {
    en_rows rows;
    int n, S, C;              // list length, events, channels
    int64_t V;
    int D0, D1, D2, T0, T1, T2, n0, n1;
    const float *srcpos, *dstpos, *offsets, *weights;
    const int *idx;
    en_tile *tiles;
    en_slot *slots;           // [tile][slots_cap]
    en_entry *entries;        // [tile][kEnTile * n]
    int slots_cap;
};

__device__ __forceinline__ int en_ordered(float f) {   // monotone float -> int
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float en_unordered(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// Voxel of local index l in tile (t0, t1, t2), or -1 past the grid.
template <typename P> __device__ __forceinline__ int64_t en_voxel(const P &p, int tile, int l) {
    const int t0 = tile % p.n0, t1 = (tile / p.n0) % p.n1, t2 = tile / (p.n0 * p.n1);
    const int g0 = t0 * p.T0 + l % p.T0, g1 = t1 * p.T1 + (l / p.T0) % p.T1, g2 = t2 * p.T2 + l / (p.T0 * p.T1);
    if (g0 >= p.D0 || g1 >= p.D1 || g2 >= p.D2) return -1;
    return ((int64_t)g2 * p.D1 + g1) * p.D0 + g0;
}

// Sorts the list entries of one tile into (block, event) buckets.  A thread
// owns a voxel and walks its list twice: the first walk takes an entry's rank
// in its bucket with one shared-memory atomic (about 30 clocks of the SM for a
// warp's 32 scattered adds: they set the kernel's time, so the delay ranges
// are reduced from the sorted entries instead) and keeps it, the second writes
// the entry at its place.  Consecutive threads read consecutive voxels.
__global__ void __launch_bounds__(kEnTile) entries_sort_kernel(const en_params p) {
    extern __shared__ int en_sort_smem[];
    __shared__ int box[kEnBlocks][6], wide[4], scan[kEnTile / 32][2], total[2], nb_s;
    const int buckets = kEnBlocks * p.S;
    int *cnt = en_sort_smem, *where = cnt + buckets;
    uint16_t *rank = reinterpret_cast<uint16_t *>(where + buckets);   // [n][kEnTile]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x;
    for (int i = tid; i < buckets; i += kEnTile) cnt[i] = 0;
    if (tid < kEnBlocks * 6) box[tid / 6][tid % 6] = (tid % 6) < 3 ? INT_MAX : INT_MIN;
    if (tid < 4) wide[tid] = 0;
    __syncthreads();
    const int64_t v = en_voxel(p, tile, tid);
    {
        const int fb = tid / (kEnTile / kEnBlocks);   // uniform over a warp
#pragma unroll
        for (int a = 0; a < 3; a++) {
            int lo = INT_MAX, hi = INT_MIN;
            if (v >= 0) {
                // a position that is not finite opens the block's box: its
                // windows are then read tap by tap
                const float q = __ldg(p.dstpos + 3 * v + a);
                lo = en_ordered(isfinite(q) ? q : -INFINITY);
                hi = en_ordered(isfinite(q) ? q : INFINITY);
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == 0) {
                atomicMin(&box[fb][a], lo);
                atomicMax(&box[fb][3 + a], hi);
            }
        }
    }
    __syncthreads();
    // windows of every (block count, block) for five channels
    if (tid < 15 * 5) {
        const int combo = tid / 5, ci = tid % 5;
        const int lv = combo >= 7 ? 3 : (combo >= 3 ? 2 : (combo >= 1 ? 1 : 0));   // NB = 1 << lv
        const int blk = combo - ((1 << lv) - 1), per = kEnBlocks >> lv;
        int b[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};
        for (int i = blk * per; i < (blk + 1) * per; i++)
            for (int a = 0; a < 6; a++) b[a] = a < 3 ? min(b[a], box[i][a]) : max(b[a], box[i][a]);
        if (b[0] <= b[3] && p.C > 0) {
            const int64_t c = (int64_t)(p.C - 1) * ci / 4;
            float n2 = 0.f, x2 = 0.f, d2 = 0.f;
            for (int a = 0; a < 3; a++) {
                const float q = __ldg(p.srcpos + 3 * c + a), mn = en_unordered(b[a]), mx = en_unordered(b[3 + a]);
                const float gap = fmaxf(fmaxf(mn - q, q - mx), 0.f), ext = fmaxf(fabsf(q - mn), fabsf(q - mx));
                n2 += gap * gap;
                x2 += ext * ext;
                d2 += (mx - mn) * (mx - mn);
            }
            // 7 for the rounding margins, 4 for the channels that share a window's start
            if (!(sqrtf(x2) - sqrtf(n2) + sqrtf(d2) + 11.f <= (float)kEnWB)) atomicExch(&wide[lv], 1);
        }
    }
    __syncthreads();
    if (tid == 0) nb_s = !wide[0] ? 0 : (!wide[1] ? 1 : (!wide[2] ? 2 : 3));
    __syncthreads();
    const int lv = nb_s, NB = 1 << lv;
    const int base = (tid >> (10 - lv)) * p.S;   // this voxel's block
    auto listed = [&](int64_t i, int &e, float &w) {   // does list place i hold an entry
        e = __ldg(p.idx + i);
        w = __ldg(p.weights + i);
        return (unsigned)e < (unsigned)p.S && w != 0.f;
    };
    if (v >= 0) {
#pragma unroll 4
        for (int j = 0; j < p.n; j++) {
            int e;
            float w;
            if (listed((int64_t)j * p.V + v, e, w)) rank[j * kEnTile + tid] = (uint16_t)atomicAdd(&cnt[base + e], 1);
        }
    }
    __syncthreads();
    // exclusive scan of (entries, nonempty buckets): a thread takes a run of buckets
    const int nbk = NB * p.S, per = (nbk + kEnTile - 1) / kEnTile;
    const int i0 = min(tid * per, nbk), i1 = min(i0 + per, nbk);
    int se = 0, sb = 0;
    for (int i = i0; i < i1; i++) {
        se += cnt[i];
        sb += cnt[i] != 0;
    }
    int ie = se, ib = sb;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, ie, d), b = __shfl_up_sync(0xffffffffu, ib, d);
        if (lane >= d) {
            ie += a;
            ib += b;
        }
    }
    if (lane == 31) {
        scan[warp][0] = ie;
        scan[warp][1] = ib;
    }
    __syncthreads();
    int pe = 0, pbk = 0;
    for (int i = 0; i < warp; i++) {
        pe += scan[i][0];
        pbk += scan[i][1];
    }
    int re = pe + ie - se, rb = pbk + ib - sb;
    if (tid == kEnTile - 1) {
        total[0] = pe + ie;
        total[1] = pbk + ib;
    }
    en_slot *slots = p.slots + (int64_t)tile * p.slots_cap;
    for (int i = i0; i < i1; i++) {
        const int c = cnt[i];
        if (c) {
            slots[rb].start = re;
            slots[rb].event_block = (i % p.S) | ((i / p.S) << 16);
        }
        cnt[i] = re;       // from here on the bucket's first entry
        where[i] = rb;     // and its index among the nonempty ones
        re += c;
        rb += c != 0;
    }
    __syncthreads();
    const int nslots = total[1], nentries = total[0];
    if (tid == 0) {
        p.tiles[tile].slots = nslots;
        p.tiles[tile].entries = nentries;
        slots[nslots].start = nentries;
        slots[nslots].event_block = 0;
    }
    if (tid < NB * 6) {   // boxes of the chosen blocks
        const int blk = tid / 6, a = tid % 6, pb = kEnBlocks >> lv;
        int b = a < 3 ? INT_MAX : INT_MIN;
        for (int i = blk * pb; i < (blk + 1) * pb; i++) b = a < 3 ? min(b, box[i][a]) : max(b, box[i][a]);
        p.tiles[tile].box[blk][a] = en_unordered(b);
    }
    en_entry *entries = p.entries + (int64_t)tile * kEnTile * p.n;
    if (v >= 0) {
#pragma unroll 4
        for (int j = 0; j < p.n; j++) {
            const int64_t i = (int64_t)j * p.V + v;
            int ev;
            en_entry e;
            if (!listed(i, ev, e.w)) continue;
            const int bk = base + ev;
            e.ofs = __ldg(p.offsets + i);
            e.key = (uint32_t)tid | ((uint32_t)where[bk] << 16);
            e.pad = 0u;
            entries[cnt[bk] + rank[j * kEnTile + tid]] = e;
        }
    }
    __syncthreads();
    // delay range of every bucket, a warp each; a delay that is not finite
    // opens the range, and the bucket's windows are read tap by tap
    for (int s = warp; s < nslots; s += kEnTile / 32) {
        const int b0 = slots[s].start, b1 = slots[s + 1].start;
        float lo = INFINITY, hi = -INFINITY;
        for (int i = b0 + lane; i < b1; i += 32) {
            const float o = entries[i].ofs;
            lo = fminf(lo, isfinite(o) ? o : -INFINITY);
            hi = fmaxf(hi, isfinite(o) ? o : INFINITY);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            slots[s].lo = lo;
            slots[s].hi = hi;
        }
    }
}

// Four tensor maps over the sample rows, boxes {128 samples, 1 event, 8 / 4 / 2 / 1 channels, 1 item}.
struct en_maps {
    CUtensorMap m[4];
};

template <int ST>   // ring stages
struct en_smem {
    static constexpr int row_bytes = kEnWB * 4;                  // one window; a bucket's G windows lie back to back
    static constexpr int stage_bytes = row_bytes * kEnSlots;
    static constexpr size_t ring_bytes = (size_t)stage_bytes * ST;
    static constexpr size_t misc_bytes = ST * kEnChannels * (32 + 16)           // channel pairs, normals
                                         + ST * kEnSlots * 4                    // window starts
                                         + kEnTile * 4                          // sums
                                         + kEnBlocks * 6 * 4 + ST * 16 + ST * 4 + 16;   // boxes, barriers, modes, abort
    static constexpr size_t bytes = (ring_bytes + misc_bytes + 15) & ~size_t(15);
    unsigned char *ring;
    float4 *chan_pair, *chan_dir;
    uint32_t *meta;      // [ST][kEnSlots]: bits(1.5 * 2^23) + first sample, or kOvf
    float *sum, *box;
    uint64_t *full, *empty;
    int *mode;           // [ST]: kStageEmpty, kStageFast
    volatile int *abort_flag;

    __device__ explicit en_smem(unsigned char *raw) {
        ring = raw;
        chan_pair = reinterpret_cast<float4 *>(raw + ring_bytes);
        chan_dir = chan_pair + ST * kEnChannels * 2;
        full = reinterpret_cast<uint64_t *>(chan_dir + ST * kEnChannels);
        empty = full + ST;
        meta = reinterpret_cast<uint32_t *>(empty + ST);
        sum = reinterpret_cast<float *>(meta + ST * kEnSlots);
        box = sum + kEnTile;
        mode = reinterpret_cast<int *>(box + kEnBlocks * 6);
        abort_flag = mode + ST;
    }
};

// The two samples of a tap at a shared address.
__device__ __forceinline__ void en_samples(uint32_t a, float &x0, float &x1) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x0) : "r"(a));
    asm volatile("ld.shared.f32 %0, [%1+4];" : "=f"(x1) : "r"(a));
}

// Channels of a stage for D buckets, and the map whose box holds them.
__device__ __forceinline__ int en_group_log2(int D) { return D <= 4 ? 3 : (D <= 8 ? 2 : (D <= 16 ? 1 : 0)); }

// The run of entries that starts at entry p0 (inside bucket s0): its buckets
// [s0, s0 + D) and end p1.  Every warp computes the same.
struct en_run {
    int D, p1;
    en_slot mine;    // bucket s0 + lane
};
__device__ __forceinline__ en_run en_next_run(const en_slot *slots, int nslots, int s0, int p0, int lane) {
    en_run r;
    const int s = min(s0 + lane, nslots);
    r.mine = slots[s];
    int next = __shfl_down_sync(0xffffffffu, r.mine.start, 1);   // the start of the following bucket
    if (lane == 31) next = slots[min(s0 + 32, nslots)].start;
    if (s0 + lane >= nslots) next = INT_MAX;
    const unsigned full = __ballot_sync(0xffffffffu, next >= p0 + kEnRun);
    const int avail = min(nslots - s0, kEnSlots);
    const int f = full ? __ffs(full) - 1 : 32;
    if (f < avail) {
        r.D = f + 1;
        r.p1 = p0 + kEnRun;
    } else {
        r.D = avail;
        r.p1 = __shfl_sync(0xffffffffu, next, avail - 1);
    }
    return r;
}
// First bucket of the run after [s0, s0 + D) ending at p1.
__device__ __forceinline__ int en_after(const en_run &r, int s0, int end_next) {
    return end_next == r.p1 ? s0 + r.D : s0 + r.D - 1;
}

// Producer warp: all stages of one run for the channels [cbeg, cend).  Lane
// d * G + g bounds the window of bucket d and channel c0 + g; the G lanes of a
// bucket agree on the union, and the first of them copies all G windows.  The
// channel positions are loaded a stage ahead.
template <int ST>
__device__ __forceinline__ void en_produce_run(const staged_params &p, const en_maps &maps, const en_smem<ST> &sm,
                                               const en_run &r, int lane, int b, int cbeg, int cend, int &stage,
                                               uint32_t &phase, bool &dead, uint32_t &issued_mask) {
    using SM = en_smem<ST>;
    const int gl = en_group_log2(r.D), G = 1 << gl, d = lane >> gl, g = lane & (G - 1);
    const CUtensorMap *map = &maps.m[3 - gl];
    const bool own = d < r.D;
    const int event = __shfl_sync(0xffffffffu, r.mine.event_block & 0xffff, d);
    const int block = __shfl_sync(0xffffffffu, r.mine.event_block >> 16, d);
    const float olo = __shfl_sync(0xffffffffu, r.mine.lo, d), ohi = __shfl_sync(0xffffffffu, r.mine.hi, d);
    const float *ab = sm.box + (own ? block : 0) * 6;
    const float ax0 = ab[0], ay0 = ab[1], az0 = ab[2], ax1 = ab[3], ay1 = ab[4], az1 = ab[5];
    int c = cbeg + g;
    float px = 0.f, py = 0.f, pz = 0.f;
    if (c < cend) {
        px = __ldg(p.srcpos + 3 * c);
        py = __ldg(p.srcpos + 3 * c + 1);
        pz = __ldg(p.srcpos + 3 * c + 2);
    }
    for (int c0 = cbeg; c0 < cend; c0 += G) {
        const int cn = c + G;
        float qx = 0.f, qy = 0.f, qz = 0.f;
        if (cn < cend) {
            qx = __ldg(p.srcpos + 3 * cn);
            qy = __ldg(p.srcpos + 3 * cn + 1);
            qz = __ldg(p.srcpos + 3 * cn + 2);
        }
        const bool have = own && c < cend;
        float lo = INFINITY, hi = -INFINITY;
        bool bad = false;
        if (have) {
            const float dx = fmaxf(fmaxf(ax0 - px, px - ax1), 0.f);
            const float dy = fmaxf(fmaxf(ay0 - py, py - ay1), 0.f);
            const float dz = fmaxf(fmaxf(az0 - pz, pz - az1), 0.f);
            const float ex = fmaxf(fabsf(px - ax0), fabsf(px - ax1));
            const float ey = fmaxf(fabsf(py - ay0), fabsf(py - ay1));
            const float ez = fmaxf(fabsf(pz - az0), fabsf(pz - az1));
            const float n2 = dx * dx + dy * dy + dz * dz, x2 = ex * ex + ey * ey + ez * ez;
            lo = floorf(olo + (n2 > 0.f ? n2 * rsqrtf(n2) : 0.f)) - 2.f;
            hi = floorf(ohi + (x2 > 0.f ? x2 * rsqrtf(x2) : 0.f)) + 2.f;
            // with bounds below 2^20 every tap's floor lies in [lo + 1, hi - 1]
            bad = !(fabsf(lo) <= kSaneRange) || !(fabsf(hi) <= kSaneRange) || !(x2 <= kSaneRange * kSaneRange);
        }
#pragma unroll
        for (int o = 1; o < kEnChannels; o <<= 1) {
            if (o < G) {
                lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
                bad |= (bool)__shfl_xor_sync(0xffffffffu, (int)bad, o);
            }
        }
        // Taps' floors lie in [lo + 1, hi - 1].  `out`: none has a tap in the
        // record (0 <= k <= N - 2).  `inner`: every one does, or reads only
        // samples past the row's ends, which arrive as zeros.
        const float k_lo = lo + 1.f, k_hi = hi - 1.f, last = (float)(p.N - 2);
        const bool out = own && !bad && (k_hi < 0.f || k_lo > last);
        const bool inner = (k_lo >= 0.f && k_hi <= last) || k_hi < -1.f || k_lo > last + 1.f;
        const int k0 = bad ? 0 : ((int)lo & ~3);
        const bool wide = own && (bad || !(hi - (float)k0 <= (float)(kEnWB - 1)));
        const bool edge = own && !inner;
        const unsigned own_mask = __ballot_sync(0xffffffffu, own);
        const bool all_out = __ballot_sync(0xffffffffu, out) == own_mask;
        const bool tested = __ballot_sync(0xffffffffu, wide || edge) != 0u || p.srcdir;
        const bool issue = own && g == 0 && !wide && !all_out;

        const uint32_t full_bar = smem_u32(&sm.full[stage]);
        if (!dead && !bounded_wait(smem_u32(&sm.empty[stage]), phase ^ 1u, sm.abort_flag, p.status)) dead = true;
        if (!dead) {
            if (d == 0) {
                sm.chan_pair[(stage * kEnChannels + g) * 2] = make_float4(px, px, py, py);
                sm.chan_pair[(stage * kEnChannels + g) * 2 + 1] = make_float4(pz, pz, 0.f, 0.f);
                if (p.srcdir && have) sm.chan_dir[stage * kEnChannels + g] = __ldg(p.srcdir + c);
            }
            if (issue)
                tma_load_box4(smem_u32(sm.ring + stage * SM::stage_bytes + lane * SM::row_bytes), map, k0, event, c0, b,
                            full_bar);
            sm.meta[stage * kEnSlots + lane] = wide ? kOvf : kFloorMagicBits + (uint32_t)k0;
        }
        const unsigned issued = dead ? 0u : __ballot_sync(0xffffffffu, issue);
        __syncwarp();
        if (lane == 0) {
            sm.mode[stage] = (all_out ? kStageEmpty : 0) | (tested ? 0 : kStageFast);
            mbar_arrive_expect_tx(full_bar, (uint32_t)__popc(issued) * (uint32_t)(G * SM::row_bytes));
        }
        if (!dead) issued_mask |= (1u << stage);
        if (++stage == ST) {
            stage = 0;
            phase ^= 1u;
        }
        c = cn;
        px = qx; py = qy; pz = qz;
    }
}

// After an abort: waits (bounded) until every copy of this CTA has landed.
template <int ST>
__device__ __forceinline__ void en_drain(const en_smem<ST> &sm, int lane, int stage, uint32_t phase,
                                         uint32_t issued_mask) {
    if (*sm.abort_flag && lane == 0) {
        for (int i = 0; i < ST; i++) {
            const int s = (stage + i) % ST;
            if (!(issued_mask & (1u << s))) continue;
            const uint32_t par = (s < stage) ? phase : (phase ^ 1u);
            const long long t0 = clock64();
            while (!mbar_try_wait(smem_u32(&sm.full[s]), par) && clock64() - t0 < kWaitCycles) __nanosleep(64);
        }
    }
}

// CTA set-up: barriers, voxel sums, block boxes.
template <int ST>
__device__ __forceinline__ void en_setup(en_smem<ST> &sm, const en_tile &t) {
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int i = 0; i < ST; i++) {
            mbar_init(smem_u32(&sm.full[i]), 1u);
            mbar_init(smem_u32(&sm.empty[i]), kStWarps);
        }
        *sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int l = tid; l < kEnTile; l += kStThreads) sm.sum[l] = 0.f;
    for (int i = tid; i < kEnBlocks * 6; i += kStThreads) sm.box[i] = (&t.box[0][0])[i];
    __syncthreads();
}

// Geometry of two entries (packed halves) and one channel: d = c - v.
struct en_geom {
    float2 dx, dy, dz, rsq, rinv;
};
__device__ __forceinline__ en_geom en_geometry(uint32_t cp, float2 nvx2, float2 nvy2, float2 nvz2) {
    const float4 qa = lds_f4(cp), qb = lds_f4(cp + 16);
    en_geom g;
    g.dx = __fadd2_rn(make_float2(qa.x, qa.y), nvx2);
    g.dy = __fadd2_rn(make_float2(qa.z, qa.w), nvy2);
    g.dz = __fadd2_rn(make_float2(qb.x, qb.y), nvz2);
    float2 r2 = __fmul2_rn(g.dx, g.dx);
    r2 = __ffma2_rn(g.dy, g.dy, r2);
    r2 = __ffma2_rn(g.dz, g.dz, r2);
    g.rsq = make_float2(fmaxf(r2.x, 1e-7f), fmaxf(r2.y, 1e-7f));
    g.rinv = make_float2(rsqrtf(g.rsq.x), rsqrtf(g.rsq.y));
    return g;
}
// The test of apply_directivity, on the negated difference.
__device__ __forceinline__ void en_directivity(en_geom &g, float4 dir) {
    float2 pr2 = __fmul2_rn(g.dx, make_float2(dir.x, dir.x));
    pr2 = __ffma2_rn(g.dy, make_float2(dir.y, dir.y), pr2);
    pr2 = __ffma2_rn(g.dz, make_float2(dir.z, dir.z), pr2);
    const bool oka = -(pr2.x * g.rinv.x) > dir.w, okb = -(pr2.y * g.rinv.y) > dir.w;
    g.rsq = make_float2(oka ? g.rsq.x : 1e30f, okb ? g.rsq.y : 1e30f);
    g.rinv = make_float2(oka ? g.rinv.x : 1.f, okb ? g.rinv.y : 1.f);
}
// Floor bits and fractions of both entries' delays.
__device__ __forceinline__ float2 en_split(const en_geom &g, float2 ofs2, uint32_t &ba, uint32_t &bb) {
    const float2 magic2 = make_float2(kFloorMagic, kFloorMagic);
    const float2 tau2 = __ffma2_rn(g.rsq, g.rinv, ofs2);
    const float2 mm2 = __fadd2_rd(tau2, magic2);
    const float2 nfl2 = __ffma2_rn(mm2, make_float2(-1.f, -1.f), magic2);   // -(floor), exact
    ba = __float_as_uint(mm2.x);
    bb = __float_as_uint(mm2.y);
    return __fadd2_rn(tau2, nfl2);
}
// Sample and slope of an entry's tap on a stage that is not kStageFast: zeros
// outside the record, else from its window or (wider than 128 samples) the row.
__device__ __forceinline__ void en_tap_tested(const en_rows &rows, int b, int c, int s, uint32_t nlast, uint32_t meta,
                                              uint32_t bits, uint32_t window, float &x0, float &d) {
    x0 = d = 0.f;
    const uint32_t k = bits - kFloorMagicBits;
    if (k >= nlast) return;
    float x1;
    if (meta == kOvf) {
        const float *r = rows.row(b, c, s) + k;
        x0 = __ldg(r);
        x1 = __ldg(r + 1);
    } else {
        en_samples(window + (bits - meta) * 4u, x0, x1);
    }
    d = x1 - x0;
}

// What a consumer lane holds of a run: two entries.
struct en_lane {
    bool ina, inb, any;       // entry a, b present; any entry in the warp
    en_entry a, b;
    int la, lb, da, db;       // voxels of the tile, buckets of the run
    float2 ofs2, nvx2, nvy2, nvz2;
};
__device__ __forceinline__ en_lane en_load(const staged_params &p, const en_entry *entries, const en_run &r, int tile, int p0,
                                           int s0, int warp, int lane) {
    en_lane e;
    const int i = p0 + warp * 64 + 2 * lane;
    e.ina = i < r.p1;
    e.inb = i + 1 < r.p1;
    e.any = p0 + warp * 64 < r.p1;
    // a lane without an entry repeats the run's last one: its taps stay inside
    // the windows, its sums are dropped
    e.a = entries[min(i, r.p1 - 1)];
    e.b = entries[min(i + 1, r.p1 - 1)];
    e.la = e.a.key & 0xffff;
    e.lb = e.b.key & 0xffff;
    e.da = (int)(e.a.key >> 16) - s0;
    e.db = (int)(e.b.key >> 16) - s0;
    e.ofs2 = make_float2(e.a.ofs, e.b.ofs);
    const float *va = p.dstpos + 3 * en_voxel(p, tile, e.la), *vb = p.dstpos + 3 * en_voxel(p, tile, e.lb);
    e.nvx2 = make_float2(-__ldg(va), -__ldg(vb));
    e.nvy2 = make_float2(-__ldg(va + 1), -__ldg(vb + 1));
    e.nvz2 = make_float2(-__ldg(va + 2), -__ldg(vb + 2));
    return e;
}

// Forward: about 14 instructions a unit (packed geometry of two entries 6, delay
// and split 2, address 1, samples 2, interpolation 2, sum 1/2).
static __global__ void __launch_bounds__(kStThreads, 3) das_entries_kernel(const staged_params p, const en_params ep,
                                                                    const __grid_constant__ en_maps maps) {
    constexpr int ST = kEnStages;
    using SM = en_smem<ST>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SM sm(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x, b = blockIdx.y;
    const en_tile &tl = ep.tiles[tile];
    en_setup<ST>(sm, tl);
    const int nslots = tl.slots, nentries = tl.entries;
    const en_slot *slots = ep.slots + (int64_t)tile * ep.slots_cap;
    const en_entry *entries = ep.entries + (int64_t)tile * kEnTile * ep.n;
    const int cbeg = chan_begin(p), cend = chan_end(p);
    const bool producer = warp == kStWarps;
    const uint32_t nlast = (uint32_t)(p.N - 1);
    int stage = 0;
    uint32_t phase = 0, issued_mask = 0;
    bool dead = false;
    const uint32_t ring_u32 = smem_u32(sm.ring), pair_u32 = smem_u32(sm.chan_pair), meta_u32 = smem_u32(sm.meta);

    for (int p0 = 0, s0 = 0; p0 < nentries;) {
        const en_run r = en_next_run(slots, nslots, s0, p0, lane);
        const int end_next = slots[min(s0 + r.D, nslots)].start;
        const int gl = en_group_log2(r.D), G = 1 << gl;
        if (producer) {
            en_produce_run<ST>(p, maps, sm, r, lane, b, cbeg, cend, stage, phase, dead, issued_mask);
        } else {
            const en_lane e = en_load(p, entries, r, tile, p0, s0, warp, lane);
            float2 acc2 = make_float2(0.f, 0.f);
            for (int c0 = cbeg; c0 < cend; c0 += G) {
                if (!dead && !bounded_wait(smem_u32(&sm.full[stage]), phase, sm.abort_flag, p.status)) dead = true;
                const int mode = dead ? kStageEmpty : *(volatile int *)&sm.mode[stage];
                if (e.any && !(mode & kStageEmpty)) {
                    const int n = min(G, cend - c0);
                    const uint32_t ma = lds_u32(meta_u32 + (stage * kEnSlots + (e.da << gl)) * 4);
                    const uint32_t mb = lds_u32(meta_u32 + (stage * kEnSlots + (e.db << gl)) * 4);
                    uint32_t wa = ring_u32 + stage * SM::stage_bytes + (e.da << gl) * SM::row_bytes;
                    uint32_t wb = ring_u32 + stage * SM::stage_bytes + (e.db << gl) * SM::row_bytes;
                    uint32_t cp = pair_u32 + stage * kEnChannels * 32;
                    if (mode & kStageFast) {
                        wa -= ma * 4u;
                        wb -= mb * 4u;
                        auto channel = [&](int cl) {
                            const en_geom g = en_geometry(cp + cl * 32, e.nvx2, e.nvy2, e.nvz2);
                            uint32_t ba, bb;
                            const float2 t2 = en_split(g, e.ofs2, ba, bb);
                            float2 x0, x1;
                            en_samples(ba * 4u + (wa + cl * SM::row_bytes), x0.x, x1.x);
                            en_samples(bb * 4u + (wb + cl * SM::row_bytes), x0.y, x1.y);
                            const float2 d = __ffma2_rn(x0, make_float2(-1.f, -1.f), x1);   // x1 - x0, one rounding
                            acc2 = __fadd2_rn(acc2, __ffma2_rn(t2, d, x0));
                        };
                        if (n == 8) {
#pragma unroll
                            for (int cl = 0; cl < 8; cl++) channel(cl);
                        } else if (n == 4) {
#pragma unroll
                            for (int cl = 0; cl < 4; cl++) channel(cl);
                        } else {
#pragma unroll 1
                            for (int cl = 0; cl < n; cl++) channel(cl);
                        }
                    } else {
                        const int sa = slots[s0 + e.da].event_block & 0xffff, sb = slots[s0 + e.db].event_block & 0xffff;
#pragma unroll 1
                        for (int cl = 0; cl < n; cl++) {
                            en_geom g = en_geometry(cp + cl * 32, e.nvx2, e.nvy2, e.nvz2);
                            if (p.srcdir) en_directivity(g, sm.chan_dir[stage * kEnChannels + cl]);
                            uint32_t ba, bb;
                            const float2 t2 = en_split(g, e.ofs2, ba, bb);
                            float xa, da, xb, db;
                            en_tap_tested(ep.rows, b, c0 + cl, sa, nlast, ma, ba, wa + cl * SM::row_bytes, xa, da);
                            en_tap_tested(ep.rows, b, c0 + cl, sb, nlast, mb, bb, wb + cl * SM::row_bytes, xb, db);
                            acc2 = __fadd2_rn(acc2, __ffma2_rn(t2, make_float2(da, db), make_float2(xa, xb)));
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sm.empty[stage]));
                if (++stage == ST) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            if (e.ina) atomicAdd(sm.sum + e.la, e.a.w * acc2.x);
            if (e.inb) atomicAdd(sm.sum + e.lb, e.b.w * acc2.y);
        }
        s0 = en_after(r, s0, end_next);
        p0 = r.p1;
    }
    const int any_dead = __syncthreads_or(dead);
    if (producer) {
        en_drain<ST>(sm, lane, stage, phase, issued_mask);
        return;
    }
    if (any_dead) return;
    float *out = static_cast<float *>(p.out) + (int64_t)b * p.out_bstride;
    for (int l = tid; l < kEnTile; l += kStConsumers) {
        const int64_t v = en_voxel(p, tile, l);
        if (v < 0) continue;
        if (p.cchunk) atomicAdd(out + v, sm.sum[l]);   // channel slices add into the prepared image
        else out[v] = p.beta_zero ? sm.sum[l] : __fmaf_rn((float)p.beta_re, out[v], sm.sum[l]);
    }
}

// x (any type and strides, with an optional per-channel gain, rounded to the
// pair storage's type) as rows of Npad floats, zeros past the record.
template <typename Tin, int K>
__global__ void __launch_bounds__(256) entry_rows_kernel(const Tin *__restrict__ x, int64_t bstride, int64_t cstride,
                                                         int64_t sstride, int C, int S, int N, int BC, int Npad,
                                                         const float *__restrict__ gain, int gain_bstride,
                                                         float *__restrict__ out) {
    const int k0 = (blockIdx.x * 256 + threadIdx.x) * 4;
    if (k0 >= Npad) return;
    for (int s = blockIdx.y; s < S; s += gridDim.y)
        for (int bc = blockIdx.z; bc < BC; bc += gridDim.z) {
            const int c = bc % C, b = bc / C;
            const Tin *r = x + (int64_t)b * bstride + (int64_t)c * cstride + (int64_t)s * sstride;
            const float g = gain ? __ldg(gain + (int64_t)b * gain_bstride + c) : 1.f;
            float f[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                f[i] = k0 + i < N ? (float)sample_io<Tin>::load(r + k0 + i) : 0.f;
                if (gain) f[i] = scaled(f[i], g);
                if constexpr (K == ST_F16) f[i] = __half2float(__float2half_rn(f[i]));
                if constexpr (K == ST_BF16) f[i] = __bfloat162float(__float2bfloat16_rn(f[i]));
            }
            *reinterpret_cast<float4 *>(out + ((int64_t)bc * S + s) * Npad + k0) = make_float4(f[0], f[1], f[2], f[3]);
        }
}

}  // namespace ffdas
