// k_cluster.cu — the fused path from labels to quads.
//
// The reference groups boundary points with a global 64-bit sort_by_key over
// every point (main.cpp:515), reduces ClusterBounds per key (:571-585),
// filters, maps points back to clusters with a binary search (:621-675) and
// sorts again by (cluster, theta) (:737).  Only the ORDER of the surviving
// clusters and the ORDER of points inside a cluster influence the result,
// and both are fixed by keys, so here:
//   1. k_boundaries_pairs: each CTA finds its boundary points, aggregates
//      them per cluster pair in a shared-memory hash table (warp-level
//      reductions first), merges the per-pair ClusterBounds sums into a
//      per-frame global hash table with one set of atomics per (CTA, pair),
//      and appends its points, tagged with their pair slot, to a list
//      (in batches, points of pairs that earlier tiles already pushed over
//      the cluster size limit are skipped);
//   2. k_pairs_finalize: one CTA per frame sorts the distinct pair keys
//      (hundreds to a few thousand), applies ValidBlobFilter and assigns
//      each surviving pair its cluster index and extent;
//   3. k_scatter_points: points of surviving pairs go straight into their
//      cluster's segment with their theta key; the rest are dropped;
//   4. k_cluster_sort: one CTA per cluster sorts by (theta, point) in
//      shared memory and writes ClusterPoints and the line-fit inputs;
//      k_cluster_lines: line-fit prefix sums and fit_lines (windowed errors,
//      7-tap filter, peaks), a warp per run of points;
//   5. k_peaks_scan / k_index_quads / k_compact_quads: peak extents, the 10
//      best peaks, do_indexing and the corner intersection, quads in reference
//      order.
#include "atag_kernels.cuh"
#include "atag_pairs.cuh"
#include "atag_quads.cuh"

namespace atag {

// ---------------------------------------------------------------------------
// reset
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_reset_frames(const __grid_constant__ FrameSet fs, uint32_t* cursors,
                                                      uint32_t n_cursors) {
    if (fs.overlap) await_previous_kernel();
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < n_cursors) cursors[threadIdx.x] = 0u;
    const FrameDesc& F = fs.get(blockIdx.y);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < F.pair_cap; i += gridDim.x * blockDim.x) {
        F.pair_keys[i] = EMPTY_KEY;
        F.pair_bbox[i] = make_uint4(0xFFFFFFFFu, 0u, 0xFFFFFFFFu, 0u);
        F.pair_gsum[i] = make_int2(0, 0);
        F.pair_pxgx[i] = 0ull;
        F.pair_count[i] = 0u;
        F.pair_cluster[i] = INVALID;
    }
    if (blockIdx.x == 0 && threadIdx.x < CNT_COUNT) F.counters[threadIdx.x] = 0u;
    if (blockIdx.x == 0 && threadIdx.x < DEAD_PAIRS && F.dead_pairs) F.dead_pairs[threadIdx.x] = EMPTY_KEY;
}

// ---------------------------------------------------------------------------
// 1. boundaries + per-pair aggregation
// ---------------------------------------------------------------------------
constexpr int BP_W = 64;                       // tile width; BP_H (8 or 16) rows is a tuning choice
constexpr int BP_SW = BP_W + 8;  // label row: x0 - 4 .. x0 + BP_W + 3 (16-byte aligned body)
constexpr int BP_LC = 64;                      // CTA hash-table entries (a tile has a few dozen pairs; more go straight to the frame's table)
constexpr uint32_t BP_VALUE = 0x3FFFFFFFu;  // label value without the colour bit

// The CTA's pair table.  Fields that start at all ones come first, then the
// zeroed ones: both halves are filled with 16-byte stores.
struct __align__(16) PairTableSmem {
    unsigned long long key[BP_LC];
    uint32_t xmin[BP_LC], ymin[BP_LC], gslot[BP_LC];
    uint32_t cnt[BP_LC], xmax[BP_LC], ymax[BP_LC];
    int gx[BP_LC];
    int pxgx[BP_LC];  // a tile's sum fits 32 bits: at most 4096 points, |x| < 2^13
};
constexpr int BP_TABLE_ONES = BP_LC * (8 + 3 * 4) / 16, BP_TABLE_QUADS = sizeof(PairTableSmem) / 16;

// Insert-or-find in the CTA's pair table; a plain read first avoids the
// atomic for keys that are already present (the common case).  *fresh is
// set when this call inserted the key.
__device__ __forceinline__ int local_insert(PairTableSmem& T, unsigned long long key, bool* fresh) {
    // a 32-bit multiplicative hash of both labels (the table has 64 slots)
    uint32_t h = (((uint32_t)key ^ ((uint32_t)(key >> 32) * 0x85EBCA6Bu)) * 0x9E3779B1u) >> 26;
    for (int p = 0; p < BP_LC; p++) {
        unsigned long long k = *(volatile unsigned long long*)&T.key[h];
        if (k == key) return (int)h;
        if (k == EMPTY_KEY) {
            k = atomicCAS(&T.key[h], EMPTY_KEY, key);
            if (k == EMPTY_KEY) {
                *fresh = true;
                return (int)h;
            }
            if (k == key) return (int)h;
        }
        h = (h + 1) & (BP_LC - 1);
    }
    return -1;
}
// A staged point: CTA table slot (8 bits), tile-relative x (6) and y (4),
// neighbour test (2) and colour direction (1).
constexpr uint32_t STAGE_DIRECT = 1u << 21; // point already accounted for in global memory
__device__ __forceinline__ uint32_t stage_entry(int ls, int xo, int yo, int t, int dir) {
    return ((uint32_t)ls << 13) | (uint32_t)xo | ((uint32_t)yo << 6) | ((uint32_t)t << 10) | ((uint32_t)dir << 12);
}
__device__ __forceinline__ uint32_t stage_packed(uint32_t e, uint32_t x0, uint32_t y0) {
    // x0 + 63 < 2^14 and y0 + 15 < 2^15: the sums leave the flag bits clear
    const uint32_t xy = (x0 | (y0 << 16)) + (e & 63) + (((e >> 6) & 15) << 16);
    return xy | (((e >> 10) & 3) << 14) | (((e >> 12) & 1) << 31);
}
// The two label words of a pair: it joins a white label (colour bit | an even
// root slot) and a black one (an odd root slot, or label 0 of pixels that are
// neither 0 nor 255).  White in the high word.
__device__ __forceinline__ unsigned long long pair_labels(unsigned long long key) {
    const uint32_t kA = (uint32_t)(key >> 32), kB = (uint32_t)key;
    if ((kA ^ kB) & 1u) {
        const uint32_t white = (kA & 1u) ? kB : kA, black = (kA & 1u) ? kA : kB;
        return (unsigned long long)(LABEL_PIXEL_MASK | white) << 32 | black;
    }
    return kA == 0u ? (unsigned long long)(LABEL_PIXEL_MASK | kB) << 32 : EMPTY_KEY;
}

// find_boundaries (find_boundaries.cpp:10-155) fused with the per-pair
// ClusterBounds reduction (main.cpp:571-585) and the compaction of points.
//
// Bound by instruction issue (~0.8 per scheduler and clock at 90% occupancy),
// a third of it the tile load, and before this form half of it the rounds
// over staged points: match_any per round and seven reductions over every
// key's lanes were ~480 instructions per 32 points.  A strip's points belong
// to 1.4 pairs on average, so a warp keeps one pair's sums in registers across
// its rounds and reduces them when the pair changes.  64 frames of 1080p 926
// -> 877 us.  Strips of many pairs pay for the changes: 32 frames of diagonal
// stripes, 6 px wide, take 2,090 us instead of 1,500.  Lanes that add their own
// points there need 650, but choosing between the two costs the others 5-25% of
// the pass: the kernel has 32 registers (eight CTAs per SM) and spills 44 bytes
// already.
template <int BP_H>
__device__ __forceinline__ void boundaries_pairs_impl(const FrameSet& fs, uint32_t min_size) {
    constexpr int BP_SH = BP_H + 1;
    constexpr int NW = BP_H / 2;               // warps: two tile rows each
    constexpr int BP_STAGE = BP_W * BP_H * 4;  // at most 4 points per pixel
    constexpr int BP_WSTAGE = 2 * BP_W * 4;    // the part of one warp (two tile rows)
    constexpr unsigned FULL = 0xFFFFFFFFu;
    static_assert(BP_W == 64, "two 32-pixel words per row");
    // frame from blockIdx.x, tile column and row from blockIdx.y and .z:
    // CTAs are dispatched frame-fastest, so the tiles in flight at once span
    // every frame of the batch and a frame's later tiles start after its
    // first ones published their over-limit pairs
    const FrameDesc& F = fs.of_table(blockIdx.x);
    const int w = F.width, h = F.height;
    const int ntx = (w + BP_W - 1) / BP_W, nty = (h + BP_H - 1) / BP_H;
    if ((int)blockIdx.y >= ntx || (int)blockIdx.z >= nty) return;
    const int x0 = blockIdx.y * BP_W, y0 = blockIdx.z * BP_H;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    // labels of the tile and its halo (column c = pixel x0 + c - 4: 3 = x0 -
    // 1, BP_W + 4 = x0 + BP_W; row BP_H is the row below the tile), and four
    // bit planes of them: per row four words, [0] bit 31 = x0 - 1, [1] and
    // [2] = x0 .. x0 + 63, [3] bit 0 = x0 + 64.  Plane x: the colour bit
    // (255 pixel), y: the component has at least min_size pixels, z and w:
    // the label is one of the two labels of the frame's first / second pair
    // known to be over the cluster size limit.
    __shared__ __align__(16) uint32_t lab[BP_SH][BP_SW];
    __shared__ uint4 planes[BP_SH][4];
    __shared__ PairTableSmem T;
    __shared__ uint32_t stage[BP_STAGE];
    __shared__ uint32_t s_nall;
    const bool track_dead = !F.stage_outputs && F.dead_pairs;

    // label words of the pairs that earlier tiles already pushed over the
    // cluster size limit (snapshots: a pair published later is simply
    // processed in full; points of a published pair can never survive).  Both
    // filter points at emission; all ones, for none, equals no label.
    static_assert(DEAD_PAIRS == 2, "two over-limit pair planes");
    const unsigned long long dead0 = track_dead ? __ldcg(F.dead_pairs) : EMPTY_KEY;
    const unsigned long long dead1 = track_dead ? __ldcg(F.dead_pairs + 1) : EMPTY_KEY;
    const uint32_t dW = (uint32_t)(dead0 >> 32), dK = (uint32_t)dead0, eW = (uint32_t)(dead1 >> 32), eK = (uint32_t)dead1;
    if (threadIdx.x == 0) s_nall = 0;
    for (int i = threadIdx.x; i < BP_TABLE_QUADS; i += blockDim.x) {
        const uint32_t v = i < BP_TABLE_ONES ? FULL : 0u;
        reinterpret_cast<uint4*>(&T)[i] = make_uint4(v, v, v, v);
    }
    // Loads.  Row-word unit u = 2 r + k (row r of the tile and its halo row,
    // 32-pixel word k) belongs to warp u % NW: lane i loads the label of
    // pixel x0 + 32 k + i (one coalesced 128-byte row segment per warp) and
    // gathers its component's size, and four warp ballots of the flags are
    // the unit's four plane words.  The last two warps, which have one unit
    // fewer, also load the left and right halo columns (lane = row).  A
    // lane issues all its label loads before the first size gather.  Labels
    // out of the image are 0, as the reference reads them.
    {
        constexpr int NUNIT = 2 * BP_SH, PER = (NUNIT + NW - 1) / NW;
        static_assert(NUNIT <= NW * (PER - 1) + NW - 2, "the last two warps have a unit fewer");
        // NW is even, so a warp's units share their word k = warp & 1 and
        // their rows are r0 + (NW / 2) j
        static_assert(NW % 2 == 0, "units of a warp share their word");
        const int kk = warp & 1, r0 = warp >> 1;
        const bool xin = x0 + 32 * kk + lane < w;
        const uint32_t* lrow = F.labels + (size_t)(y0 + r0) * w + (x0 + 32 * kk + lane);
        const uint32_t* sizes = F.sizes;
        uint32_t lv[PER], sz[PER];
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const bool in = warp + NW * j < NUNIT && xin && y0 + r0 + (NW / 2) * j < h;
            lv[j] = in ? __ldg(lrow + (size_t)j * (NW / 2) * w) : 0u;
        }
        const bool halo = warp >= NW - 2, right = warp == NW - 1;
        uint32_t hl = 0u, hs = 0u;
        if (halo) {
            const int hx = right ? x0 + BP_W : x0 - 1, hy = y0 + lane;
            if (lane < BP_SH && hx >= 0 && hx < w && hy < h) hl = __ldg(F.labels + (size_t)hy * w + hx);
        }
#pragma unroll
        for (int j = 0; j < PER; j++)
            if (warp + NW * j < NUNIT) sz[j] = __ldg(sizes + (lv[j] & LABEL_VALUE_MASK));
        if (halo) hs = __ldg(sizes + (hl & LABEL_VALUE_MASK));
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int r = r0 + (NW / 2) * j;
            if (warp + NW * j >= NUNIT) break;
            const uint32_t l = lv[j];
            lab[r][4 + 32 * kk + lane] = l;
            uint4 pl;
            pl.x = __ballot_sync(FULL, (int)l < 0);
            pl.y = __ballot_sync(FULL, sz[j] >= min_size);
            pl.z = __ballot_sync(FULL, l == dW || l == dK);
            pl.w = __ballot_sync(FULL, l == eW || l == eK);
            if (lane == 0) planes[r][1 + kk] = pl;
        }
        if (halo && lane < BP_SH) {
            lab[lane][right ? BP_W + 4 : 3] = hl;
            const int sh = right ? 0 : 31;
            planes[lane][right ? 3 : 0] =
                make_uint4((hl >> 31) << sh, (hs >= min_size ? 1u : 0u) << sh, (hl == dW || hl == dK ? 1u : 0u) << sh,
                           (hl == eW || hl == eK ? 1u : 0u) << sh);
        }
    }
    __syncthreads();

    // A: enumerate points in the reference's test order (R, BL unless it
    // would duplicate, B, BR: find_boundaries.cpp:128-150).  Lane (rl, k,
    // t, half) of warp w takes 16 pixels of the 32-pixel word k of tile row
    // 2 w + rl and test t: a pixel emits test t when it is in the image and
    // big and the tested neighbour is big and of the other colour (BL also
    // not when it duplicates the left pixel's BR), computed for the word at
    // once on the bit planes.  Points of the over-limit pairs are counted but
    // not staged.
    uint32_t mt, st;
    const int k = (lane >> 3) & 1, t = (lane >> 1) & 3, r = 2 * warp + (lane >> 4);
    {
        const int xb = x0 + 32 * k;
        // The lane's tested neighbour: the same row for R (t = 0), the row
        // below for BL, B and BR.  Bit i of its plane word is pixel
        // xb + i + dx (dx = +1 for R and BR, -1 for BL, 0 for B): a funnel
        // shift of words lo, lo + 1 of that plane row.
        const int lo = t == 1 ? k : k + 1, amt = t == 1 ? 31 : (t == 2 ? 0 : 1);
        const uint4 own = planes[r][k + 1];
        const uint4* nrow = planes[r + (t != 0 ? 1 : 0)];
        const uint4 a = nrow[lo], b = nrow[lo + 1];
        const uint2 lf = *reinterpret_cast<const uint2*>(&planes[r][k]);  // colour and size of the word to the left
        uint32_t live = (y0 + r < h) ? (xb + 32 <= w ? FULL : (xb < w ? ((1u << (w - xb)) - 1u) : 0u)) : 0u;
        if (xb == 0) live &= ~1u;  // column 0 is never processed
        live &= own.y & ((lane & 1) ? 0xFFFF0000u : 0x0000FFFFu);
        // BL is not emitted where the left pixel's BR covers the same pair
        // (for BL, word b is the one below the lane's own)
        if (t == 1) live &= ~((__funnelshift_l(lf.x, own.x, 1) ^ b.x) & __funnelshift_l(lf.y, own.y, 1) & b.y);
        mt = (__funnelshift_r(a.x, b.x, amt) ^ own.x) & __funnelshift_r(a.y, b.y, amt) & live;
        // points whose two pixels are both labels of one published pair
        st = mt & ~((own.z & __funnelshift_r(a.z, b.z, amt)) | (own.w & __funnelshift_r(a.w, b.w, amt)));
    }
    // Each warp lists its staged points in its own part of the staging
    // array (warp scan) and aggregates them itself, so no CTA barrier
    // separates the masks from the rounds.
    uint32_t* wst = stage + warp * BP_WSTAGE;
    uint32_t nst = 0;
    {
        const uint32_t nall_w = __reduce_add_sync(FULL, (uint32_t)__popc(mt));
        if (lane == 0 && nall_w) atomicAdd(&s_nall, nall_w);
    }
    if (__any_sync(FULL, st != 0u)) {
        const uint32_t ns = (uint32_t)__popc(st);
        uint32_t incl = ns;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += v;
        }
        nst = __shfl_sync(FULL, incl, 31);
        uint32_t pos = incl - ns;
        const uint32_t base = stage_entry(0, 32 * k, r, t, 0) - 1u;  // + ffs: pixel 32 k + ffs - 1 (mod 2^32)
        for (uint32_t mm = st; mm; mm &= mm - 1) wst[pos++] = base + (uint32_t)__ffs(mm);
        __syncwarp();

        // The warp takes its staged points 32 at a time.  The points of one
        // pair at a time add to the warp's sums of its current pair: counts
        // from ballots, extents and the weighted sum per lane.  When the
        // pair changes the sums are reduced into the CTA table's slot.
        unsigned long long cur = EMPTY_KEY;
        int ls = -1, gx = 0, px = 0;
        uint32_t cnt = 0, rows = 0, xmn = FULL, xmx = 0u;  // rows: bit 0 / 1, a point in the warp's first / second row
        auto flush = [&]() {
            if (ls < 0) return;
            const uint32_t a = __reduce_min_sync(FULL, xmn), b = __reduce_max_sync(FULL, xmx);
            const int s = __reduce_add_sync(FULL, px);
            if (lane == 0) {
                const uint32_t yd = 2u * (uint32_t)(y0 + 2 * warp);
                atomicAdd(&T.cnt[ls], cnt);
                atomicMin(&T.xmin[ls], a);
                atomicMax(&T.xmax[ls], b);
                atomicMin(&T.ymin[ls], (rows & 1u) ? yd : yd + 2u);
                atomicMax(&T.ymax[ls], (rows & 2u) ? yd + 2u : yd);
                atomicAdd(&T.gx[ls], gx);
                atomicAdd(&T.pxgx[ls], s);
            }
        };
        for (uint32_t b0 = 0; b0 < nst; b0 += 32) {
            const uint32_t i = b0 + (uint32_t)lane;
            const bool v = i < nst;
            uint32_t e = v ? wst[i] : 0u;
            // the point's pixel and its tested neighbour in the label tile: R is
            // the next word, BL, B and BR the row below (BP_SW - 1, BP_SW, BP_SW + 1)
            static_assert(BP_SW == 72, "neighbour offsets 1, 71, 72, 73");
            const uint32_t* pl = &lab[0][4] + ((e >> 6) & 15u) * BP_SW + (e & 63u);
            const uint32_t p = pl[0], q = pl[(0x49484701u >> (8 * ((e >> 10) & 3u))) & 0xFFu];
            const uint32_t lp = p & BP_VALUE, lq = q & BP_VALUE;
            const uint32_t kA = min(lp, lq), kB = max(lp, lq);
            const bool dir = q > p;  // the colours differ: q is the 255 pixel
            const uint32_t xd = 2u * ((uint32_t)x0 + (e & 63u)) + 1u;
            const unsigned second = __ballot_sync(FULL, (e >> 6) & 1u), up = __ballot_sync(FULL, dir);
            e |= (dir ? 1u : 0u) << 12;
            for (unsigned pend = __ballot_sync(FULL, v); pend;) {
                const int leader = __ffs(pend) - 1;
                const uint32_t gA = __shfl_sync(FULL, kA, leader), gB = __shfl_sync(FULL, kB, leader);
                const bool in = v && kA == gA && kB == gB;
                const unsigned m = __ballot_sync(FULL, in);
                pend &= ~m;
                const unsigned long long key = (unsigned long long)gA << 32 | gB;
                if (key != cur) {
                    flush();
                    cur = key;
                    if (lane == 0) {
                        // a key new to the tile also takes its slot in the frame's
                        // table now, so the merge below needs one round trip less
                        // (0.3% of a batch); by one try only, since a full table
                        // has all its slots tried: the merge does that with a
                        // thread per key, where a warp after the other's first
                        // lane took 99 instead of 54 ms for 32 overflowing frames
                        bool fresh = false;
                        ls = local_insert(T, key, &fresh);
                        if (fresh) T.gslot[ls] = global_insert(F, key, 1);
                    }
                    ls = __shfl_sync(FULL, ls, 0);
                    cnt = rows = xmx = 0u;
                    xmn = FULL;
                    gx = px = 0;
                }
                if (ls >= 0) {
                    cnt += (uint32_t)__popc(m);
                    gx += 2 * __popc(m & up) - __popc(m);
                    rows |= ((m & ~second) ? 1u : 0u) | ((m & second) ? 2u : 0u);
                    if (in) {
                        xmn = min(xmn, xd);
                        xmx = max(xmx, xd);
                        px += dir ? (int)xd : -(int)xd;
                        e |= (uint32_t)ls << 13;
                    }
                } else if (in) {  // CTA table full: account for and list the point directly
                    e |= STAGE_DIRECT;
                    uint32_t* status = F.counters + CNT_STATUS;
                    const uint32_t gs = global_insert(F, key), yd = 2u * (uint32_t)(y0 + (int)((e >> 6) & 15u));
                    if (gs == INVALID) {
                        atomicOr(status, ATAG_DEVFLAG_PAIR_OVERFLOW);
                    } else {
                        const int g = dir ? 1 : -1;
                        global_flush(F, key, gs, 1, xd, xd, yd, yd, g, 0, (unsigned long long)(long long)((int)xd * g));
                        const uint32_t at = atomicAdd(F.counters + CNT_POINTS, 1u);
                        if (at < F.point_cap) F.points[at] = ((unsigned long long)gs << 32) | stage_packed(e, x0, y0);
                        else atomicOr(status, ATAG_DEVFLAG_POINT_OVERFLOW);
                    }
                }
            }
            if (v) wst[i] = e;
        }
        flush();
    }
    __syncthreads();

    // C: merge into the frame's table.  A pair whose running point count
    // already exceeds ValidBlobFilter's maximum 2 (2w + 2h)
    // (cluster_bounds.h:92-93,102) can never survive; its points are counted
    // but not listed.
    const uint32_t max_pixels = 2u * (2u * (uint32_t)w + 2u * (uint32_t)h);
    if (threadIdx.x == 0 && s_nall) atomicAdd(F.counters + CNT_ALLPOINTS, s_nall);
    for (int i = threadIdx.x; i < BP_LC; i += blockDim.x) {
        unsigned long long key = T.key[i];
        if (key == EMPTY_KEY) continue;
        uint32_t gs = T.gslot[i];
        if (gs == INVALID) {  // its first slot held another key
            gs = global_insert(F, key);
            if (gs == INVALID) {  // the frame's table is full
                atomicOr(F.counters + CNT_STATUS, ATAG_DEVFLAG_PAIR_OVERFLOW);
                continue;
            }
        }
        uint32_t old = global_flush(F, key, gs, T.cnt[i], T.xmin[i], T.xmax[i], T.ymin[i], T.ymax[i], T.gx[i], 0,
                                    (unsigned long long)(long long)T.pxgx[i]);
        T.gslot[i] = (old + T.cnt[i] > max_pixels) ? INVALID : gs;
        // the flush that crosses the limit publishes the pair, so that later
        // tiles skip its points (its count only grows: it stays rejected)
        if (track_dead && old <= max_pixels && old + T.cnt[i] > max_pixels) {
            const unsigned long long labels = pair_labels(key);
            for (uint32_t d = 0; d < DEAD_PAIRS; d++)
                if (atomicCAS(F.dead_pairs + d, EMPTY_KEY, labels) == EMPTY_KEY) break;
        }
    }
    __syncthreads();
    if (nst == 0) return;

    // D: each warp lists the points of live pairs from its own staging
    // part: a count pass, one atomic for the warp's place in the list, then
    // the writes in the same order
    auto live_at = [&](uint32_t i) {
        if (i >= nst) return false;
        const uint32_t e = wst[i];
        return !(e & STAGE_DIRECT) && T.gslot[(e >> 13) & 255] != INVALID;
    };
    // the first round's ballot is kept for the writes (most warps have one)
    const unsigned m_first = __ballot_sync(0xFFFFFFFFu, live_at(lane));
    uint32_t nlive = (uint32_t)__popc(m_first);
    for (uint32_t b0 = 32; b0 < nst; b0 += 32) nlive += (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, live_at(b0 + lane)));
    if (nlive == 0) return;
    uint32_t at = 0;
    if (lane == 0) {
        at = atomicAdd(F.counters + CNT_POINTS, nlive);
        if ((unsigned long long)at + nlive > F.point_cap) atomicOr(F.counters + CNT_STATUS, ATAG_DEVFLAG_POINT_OVERFLOW);
    }
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t point_cap = F.point_cap;
    unsigned long long* points = F.points;
    for (uint32_t b0 = 0; b0 < nst; b0 += 32) {
        const uint32_t i = b0 + (uint32_t)lane;
        const unsigned m = b0 == 0 ? m_first : __ballot_sync(0xFFFFFFFFu, live_at(i));
        const bool lv = (m >> lane) & 1u;
        if (lv) {
            const uint32_t e = wst[i], dst = at + (uint32_t)__popc(m & lt);
            if (dst < point_cap) points[dst] = ((unsigned long long)T.gslot[(e >> 13) & 255] << 32) | stage_packed(e, x0, y0);
        }
        at += (uint32_t)__popc(m);
    }
}

// ---------------------------------------------------------------------------
// 2. pair finalisation: sort keys, filter, cluster indices and extents
// ---------------------------------------------------------------------------
constexpr int PF_THREADS = 1024;
constexpr int PF_SMEM_KEYS = 6048;  // with the scan words, under 48 KB of static shared memory

// K block-wide exclusive scans at once (one set of barriers for all):
// v[k] becomes its exclusive prefix, tot[k] the block total.  `red` holds
// K x 33 words.
template <int K>
__device__ __forceinline__ void block_exclusive_scan_multi(uint32_t (&v)[K], uint32_t (*red)[33], uint32_t (&tot)[K]) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    uint32_t x[K];
#pragma unroll
    for (int k = 0; k < K; k++) x[k] = v[k];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int k = 0; k < K; k++) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x[k], o);
            if (lane >= o) x[k] += y;
        }
    __syncthreads();
    if (lane == 31)
#pragma unroll
        for (int k = 0; k < K; k++) red[k][wid] = x[k];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const uint32_t s = lane < nw ? red[k][lane] : 0u;
            uint32_t q = s;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, q, o);
                if (lane >= o) q += y;
            }
            red[k][lane] = q - s;  // exclusive prefix of warp totals
            if (lane == 31) red[k][32] = q;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) {
        tot[k] = red[k][32];
        v[k] = red[k][wid] + x[k] - v[k];
    }
}

// Ascending sort of n <= 1024 E keys at src into dst (shared memory, 1024 E
// words) by a CTA of 1024 threads: the flip form of the bitonic network with E
// keys a thread in registers.  Partners up to 32 E positions apart are in the
// thread or its warp; only the others go through shared memory and barriers
// (10 of 45 steps for 512 keys).
template <int E>
__device__ __forceinline__ void sort_keys(const unsigned long long* src, unsigned long long* dst, uint32_t n) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const uint32_t t = threadIdx.x;
    unsigned long long k[E];
#pragma unroll
    for (int e = 0; e < E; e++) k[e] = t * E + e < n ? src[t * E + e] : ~0ull;
    uint32_t lg = 0;
    while ((1u << lg) < n) lg++;
    const bool act = (t & ~31u) * E < n;  // warps of padding only keep the barriers
    for (uint32_t lk = 1; lk <= lg; lk++) {
        for (int lj = (int)lk - 1; lj >= 0; lj--) {
            // position i meets i ^ m; the one without bit lj keeps the smaller
            const bool flip = lj == (int)lk - 1;
            const uint32_t m = flip ? (1u << lk) - 1u : 1u << lj, mt = m / E;
            auto order = [&](unsigned long long& a, unsigned long long& b) {
                const unsigned long long lo = a < b ? a : b, hi = a < b ? b : a;
                a = lo;
                b = hi;
            };
            if (m < E) {
                if constexpr (E == 2) order(k[0], k[1]);
                if constexpr (E == 4) {
                    if (m == 1) order(k[0], k[1]), order(k[2], k[3]);
                    else if (m == 2) order(k[0], k[2]), order(k[1], k[3]);
                    else order(k[0], k[3]), order(k[1], k[2]);
                }
                continue;
            }
            unsigned long long o[E];
            if (mt < 32) {
                if (!act) continue;
#pragma unroll
                for (int e = 0; e < E; e++) o[e] = __shfl_xor_sync(FULL, k[e], (int)mt);
            } else {
                if (act)
#pragma unroll
                    for (int e = 0; e < E; e++) dst[e * 1024 + t] = k[e];
                __syncthreads();
                if (act)
#pragma unroll
                    for (int e = 0; e < E; e++) o[e] = (t ^ mt) * E < n ? dst[e * 1024 + (t ^ mt)] : ~0ull;
                __syncthreads();
                if (!act) continue;
            }
            const bool upper = ((t * E) >> lj) & 1u;
#pragma unroll
            for (int e = 0; e < E; e++) {
                const unsigned long long v = flip ? o[E - 1 - e] : o[e];
                k[e] = (v < k[e]) != upper ? v : k[e];
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; e++)
        if (t * E + e < n) dst[t * E + e] = k[e];
    __syncthreads();
}

// The end of a kernel of one CTA per frame: the CTA that finishes last makes
// the prefix offsets of the per-frame counters over the batch (the flattened
// work spaces of the per-cluster kernels), a warp per list.
__device__ __forceinline__ void batch_offsets(const FrameSet& fs, const BatchOffsets& a) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const uint32_t n_frames = gridDim.x, lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();  // this thread wrote the frame's counters
        last = n_frames == 1 || atomicAdd(a.ticket, 1u) == n_frames - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last || k >= 3) return;
    uint32_t* offsets = k == 0 ? a.offsets[0] : (k == 1 ? a.offsets[1] : a.offsets[2]);
    const uint32_t which = k == 0 ? a.which[0] : (k == 1 ? a.which[1] : a.which[2]);
    if (!offsets) return;
    uint32_t carry = 0;
    for (uint32_t f0 = 0; f0 < n_frames; f0 += 32) {
        const uint32_t f = f0 + lane, v = f < n_frames ? __ldcg(fs.get(f).counters + which) : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (f < n_frames) offsets[f] = carry + x - v;
        carry += __shfl_sync(FULL, x, 31);
    }
    if (lane == 0) offsets[n_frames] = carry;
}

// One CTA per frame, bound by the latency of its serial steps: reading the key
// list instead of counting and gathering the table's used slots, the sort in
// registers and the batch's work lists made here took a lone 1080p frame's 333
// keys from 28 to 21 us and a 4K frame's 1254 from 56 to 36 (with the list
// kernel that followed).
__global__ void __launch_bounds__(PF_THREADS) k_pairs_finalize(const __grid_constant__ FrameSet fs,
                                                               PipelineParams p, uint32_t small_max,
                                                               BatchOffsets a) {
    if (fs.overlap) await_previous_kernel();
    const FrameDesc& F = fs.get(blockIdx.x);
    uint32_t* status = F.counters + CNT_STATUS;
    __shared__ unsigned long long s_keys[PF_SMEM_KEYS];
    __shared__ uint32_t red4[4][33];
    // the frame's distinct keys, listed in any order: sorted in shared memory
    // when they fit, else in place
    const uint32_t C = F.counters[CNT_PAIRS];
    unsigned long long* list = F.cluster_keys + F.cluster_cap;
    unsigned long long* keys = C <= (uint32_t)PF_SMEM_KEYS ? s_keys : list;
    if (C <= 1024u) sort_keys<1>(list, s_keys, C);
    else if (C <= 2048u) sort_keys<2>(list, s_keys, C);
    else if (C <= 4096u) sort_keys<4>(list, s_keys, C);
    else {
        if (keys == s_keys)
            for (uint32_t i = threadIdx.x; i < C; i += blockDim.x) keys[i] = list[i];
        __syncthreads();
        bitonic_sort_u64(keys, C);
        __syncthreads();
    }
    FilterParams fp;
    fp.min_cluster_pixels = p.min_cluster_pixels;
    fp.max_cluster_pixels = 2u * (2u * F.width + 2u * F.height);
    fp.tag_width = p.tag_width;
    fp.normal_border = p.normal_border;
    fp.reversed_border = p.reversed_border;
    uint32_t carry_start = 0, carry_cluster = 0, carry_fstart = 0, carry_small = 0, carry_large = 0, carry_fit = 0;
    uint32_t carry_runs = 0;
    for (uint32_t c0 = 0; c0 < C; c0 += blockDim.x) {
        uint32_t c = c0 + threadIdx.x;
        uint32_t slot = INVALID, cnt = 0;
        bool keep = false;
        uint4 bb = make_uint4(0, 0, 0, 0);
        int2 gs = make_int2(0, 0);
        long long pxgx = 0;
        if (c < C) {
            slot = global_lookup(F, keys[c]);
            cnt = F.pair_count[slot];
            bb = F.pair_bbox[slot];
            gs = F.pair_gsum[slot];
            pxgx = (long long)F.pair_pxgx[slot];
            keep = valid_blob(fp, cnt, bb.x, bb.y, bb.z, bb.w, gs.x, gs.y, pxgx);
        }
        // the scans in key order, in two rounds (which kept pairs fit
        // depends on the first round's prefixes)
        uint32_t s1[3] = {cnt, keep ? 1u : 0u, keep ? cnt : 0u}, t1[3];
        block_exclusive_scan_multi<3>(s1, red4, t1);
        const uint32_t tot_cnt = t1[0], tot_keep = t1[1], tot_fcnt = t1[2];
        uint32_t start = carry_start + s1[0];
        if (c < C && F.pair_bounds_out) {
            // every pair's bounds in key order (stages 5-6 of the reference)
            if (c < F.pair_out_cap) {
                atag_cluster_bounds b;
                b.x_min = (uint16_t)bb.x; b.x_max = (uint16_t)bb.y;
                b.y_min = (uint16_t)bb.z; b.y_max = (uint16_t)bb.w;
                b.gx_sum = gs.x; b.gy_sum = gs.y;
                b.pxgx_pygy_sum = pxgx;
                b.start = start;
                b.count = cnt;
                F.pair_bounds_out[c] = b;
                if (F.pair_keys_out) F.pair_keys_out[c] = keys[c];
            } else {
                atomicOr(status, ATAG_DEVFLAG_PAIR_OVERFLOW);
            }
        }
        uint32_t cid = carry_cluster + s1[1];
        uint32_t fstart = carry_fstart + s1[2];
        const bool fits = keep && cid < F.cluster_cap && (unsigned long long)fstart + cnt <= F.cpoint_cap;
        const bool small = cnt <= small_max;
        uint32_t s2[4] = {fits && small ? 1u : 0u, fits && !small ? 1u : 0u, fits ? cnt : 0u,
                          fits ? (cnt + CE_RUN - 1) / CE_RUN : 0u}, t2[4];
        block_exclusive_scan_multi<4>(s2, red4, t2);
        const uint32_t tot_small = t2[0], tot_large = t2[1], tot_fit = t2[2], tot_runs = t2[3];
        uint32_t js = carry_small + s2[0];
        uint32_t jl = carry_large + s2[1];
        const uint32_t run0 = carry_runs + s2[3];
        if (fits) F.cluster_work[small ? js : F.cluster_cap - 1 - jl] = cid;
        if (keep) {
            if (!fits) {
                atomicOr(status, ATAG_DEVFLAG_CLUSTER_OVERFLOW);
            } else {
                F.pair_cluster[slot] = cid;
                F.cluster_keys[cid] = keys[c];
                atag_cluster_bounds b;
                b.x_min = (uint16_t)bb.x; b.x_max = (uint16_t)bb.y;
                b.y_min = (uint16_t)bb.z; b.y_max = (uint16_t)bb.w;
                b.gx_sum = gs.x; b.gy_sum = gs.y;
                b.pxgx_pygy_sum = pxgx;
                b.start = start;
                b.count = cnt;
                F.cluster_bounds[cid] = b;
                F.cluster_extents[cid] = atag_cluster_extents{fstart, cnt};
                F.cluster_center[cid] = make_float2(bounds_cx(bb.x, bb.y), bounds_cy(bb.z, bb.w));
                F.cluster_cursor[cid] = 0;
                F.cluster_runs[cid] = run0;
                F.peak_count[cid] = 0;
            }
        }
        carry_start += tot_cnt;
        carry_cluster += tot_keep;
        carry_fstart += tot_fcnt;
        carry_small += tot_small;
        carry_large += tot_large;
        carry_fit += tot_fit;
        carry_runs += tot_runs;
    }
    if (threadIdx.x == 0) {
        // clusters are assigned in order and the capacity checks are
        // monotone, so the clusters that fit are the prefix [0, nfit) and
        // their points the prefix [0, carry_fit) of the cluster point array
        const uint32_t nfit = carry_small + carry_large;
        F.counters[CNT_CLUSTERS] = nfit;
        F.counters[CNT_SMALL] = carry_small;
        F.counters[CNT_LARGE] = carry_large;
        F.counters[CNT_RUNS] = carry_runs;
        F.stats->width = F.width;
        F.stats->height = F.height;
        F.stats->n_points = F.counters[CNT_ALLPOINTS];
        F.stats->n_pairs = C;
        F.stats->n_clusters = nfit;
        F.stats->n_cluster_points = carry_fit;
    }
    batch_offsets(fs, a);
}

// ---------------------------------------------------------------------------
// 3. scatter points of surviving pairs into their cluster segments
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_scatter_points(const __grid_constant__ FrameSet fs) {
    if (fs.overlap) await_previous_kernel();
    const FrameDesc& F = fs.of_table(blockIdx.y);
    uint32_t n = F.counters[CNT_POINTS];
    if (n > F.point_cap) n = F.point_cap;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        uint32_t i = base + threadIdx.x;
        uint32_t cid = INVALID, packed = 0;
        if (i < n) {
            unsigned long long e = F.points[i];
            uint32_t slot = (uint32_t)(e >> 32);
            packed = (uint32_t)e;
            if (slot != INVALID) cid = F.pair_cluster[slot];
        }
        unsigned mask = __match_any_sync(0xffffffffu, cid);
        if (cid != INVALID) {
            int leader = __ffs(mask) - 1;
            uint32_t b = 0;
            if ((int)lane == leader) b = atomicAdd(F.cluster_cursor + cid, (uint32_t)__popc(mask));
            b = __shfl_sync(mask, b, leader);
            uint32_t rank = __popc(mask & ((1u << lane) - 1u));
            atag_cluster_extents ext = F.cluster_extents[cid];
            float2 ctr = F.cluster_center[cid];
            float theta = calc_theta(packed, ctr.x, ctr.y);
            uint32_t pos = ext.start + b + rank;
            F.sortbuf[pos] = ((unsigned long long)float_order_key(theta) << 32) | packed;
        }
    }
}

// ---------------------------------------------------------------------------
// 4. one cluster per CTA: sort by (theta, point), ClusterPoints and line-fit
// inputs; then one warp per run of points: the prefix sums
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t find_frame(const uint32_t* offsets, uint32_t n_frames, uint32_t item) {
    uint32_t lo = 0, hi = n_frames;  // offsets[lo] <= item < offsets[hi]
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (offsets[mid] <= item) lo = mid; else hi = mid;
    }
    return lo;
}

// Bucket of a sort key's theta half among nb = 4 nq buckets: a monotone
// function of the key, about uniform over a compact cluster.  calc_theta
// (boundary_point.h:48-61) is a quadrant's offset plus a ratio r >= 0 of
// tangent type, which may run into the next quadrant's values, so the four
// parts are cut by value.  Up to r = 64 a part's first 7/8 of buckets are linear
// in r / (1 + r) (the angle, nearly); beyond, points close to an axis of the
// cluster (long thin shapes) take the last 1/8 by the logarithm of r.  Every
// operation rounds to nearest, so each step and the whole are monotone.
struct Buckets {
    uint32_t nq, lin, sh;  // buckets per part, linear ones, log step
    float scale;
    __device__ __forceinline__ explicit Buckets(uint32_t nb) {
        nq = nb >> 2;
        lin = nq - (nq >> 3);
        sh = 24u + 6u - (31u - (uint32_t)__clz((int)nq));  // 14 octaves of r fit nq / 8 buckets
        scale = __fmul_rn((float)lin, 65.0f / 64.0f);
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t theta_key) const {
        const float th = float_from_order_key(theta_key);
        const uint32_t part = th < 0.0f ? 0u : th < 65536.0f ? 1u : th < 131072.0f ? 2u : 3u;
        const float r = __fsub_rn(th, ((float)part - 1.0f) * 65536.0f);
        uint32_t b;
        if (r < 64.0f) {
            const float g = __fsub_rn(1.0f, __frcp_rn(__fadd_rn(1.0f, r)));
            b = min((uint32_t)max(__float2int_rz(__fmul_rn(g, scale)), 0), lin - 1u);
        } else {
            b = lin + min((__float_as_uint(r) - __float_as_uint(64.0f)) >> sh, nq - lin - 1u);
        }
        return part * nq + b;
    }
};

constexpr uint32_t SPLIT_STEPS = 48, SPLIT_MIN = 512;

// Sort of one cluster per CTA by (theta, packed point), the reference's
// (cluster, slope) order (main.cpp:737-750) with ties fixed by the point, as
// a bucket sort: count the buckets, prefix the counts, place the keys bucket
// by bucket, then rank each key among its bucket's.  In compact clusters those
// are few (rounding of theta leaves up to ~25 equal ones in the largest): O(n),
// against the log2(threads) merge rounds, and radix passes in global memory
// above 16,384 keys, that it replaced.  On a thin slanted line theta takes few
// values, and thousands of keys share one.  Where the buckets of one warp alone
// would take SPLIT_STEPS comparisons per key of the cluster, the buckets are made
// anew, cut by MAX_NB / 4 of the keys themselves, evenly sampled and sorted: a
// key's bucket is then found by binary search, and whatever the shape a bucket
// holds 4 n / MAX_NB keys on average.  A line of 10,700 keys takes 72 us (471
// without, 90 by the merge sort), one of 15,200 keys 115 (1,235; 127), one of
// 31,700 keys, past the shared memory, 281 (8,289; 584).  With 32 to 128 steps a
// key these take about the same, lines of 1,650 keys 29 to 24; up to SPLIT_MIN
// keys, where all of them in one bucket cost some 5 us, nothing is counted.
// Bound by instruction issue and the latency of one CTA; sort and prefix sums of
// a lone 1080p frame 82 -> 42 us, of a 4K stress frame 343 -> 100 us, of 64 1080p
// frames 750 -> 492 us (stage alone, the prefix sums by a kernel of their own).
// Keys are placed in shared memory, or for clusters over `cap` keys (frames
// larger than 4K) in their segment of errbuf.  Results: ClusterPoints and, in
// the segment of sortbuf, each point's line-fit inputs in sorted order; and
// per run of CE_RUN points the moments of all earlier points, from which
// k_cluster_lines computes the prefix sums with any number of warps.
template <uint32_t THREADS, int KEEP, uint32_t MAX_NB, uint32_t MAX_RUNS>
__device__ __forceinline__ void cluster_sort(const FrameSet& fs, const uint32_t* __restrict__ work_offsets,
                                             uint32_t n_frames, uint32_t* __restrict__ work_counter, uint32_t cap) {
    constexpr uint32_t W = THREADS / 32;
    extern __shared__ unsigned long long smem_keys[];  // cap keys, then MAX_NB counters
    uint32_t* hist = reinterpret_cast<uint32_t*>(smem_keys + cap);
    __shared__ long long red_m[6][MAX_RUNS];
    __shared__ uint32_t red32[W];
    __shared__ uint32_t s_item;
    // of split clusters: MAX_NB / 4 counters, and the sorted samples
    constexpr uint32_t SPLIT = MAX_NB / 4;
    unsigned long long* cuts = reinterpret_cast<unsigned long long*>(hist + MAX_NB / 2);
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t total = work_offsets[n_frames];
    // a CTA's first cluster is its own index, later ones come from the queue
    for (uint32_t item = blockIdx.x; item < total;) {
        const uint32_t fidx = find_frame(work_offsets, n_frames, item);
        const FrameDesc& F = fs.get(fidx);
        const uint32_t j = item - work_offsets[fidx];
        const uint32_t cid = F.cluster_work[THREADS == CF_LARGE_THREADS ? F.cluster_cap - 1 - j : j];
        const atag_cluster_extents ext = F.cluster_extents[cid];
        const uint32_t n = ext.count, start = ext.start;
        unsigned long long* src = F.sortbuf + start;
        unsigned long long* X = n <= cap ? smem_keys : reinterpret_cast<unsigned long long*>(F.errbuf) + start;
        // about one bucket per key
        const uint32_t nb = min(max(256u, 1u << (32 - __clz((int)(n - 1u)))), MAX_NB);
        const Buckets theta_buckets(nb);
        auto by_theta = [&](unsigned long long k) { return theta_buckets((uint32_t)(k >> 32)); };
        auto by_cuts = [&](unsigned long long k) {  // the cuts above the first that are at most the key
            uint32_t b = 0;
#pragma unroll
            for (uint32_t step = SPLIT / 2; step; step >>= 1) b += cuts[b + step] <= k ? step : 0u;
            return b;
        };
        for (uint32_t i = threadIdx.x; i < nb; i += THREADS) hist[i] = 0u;
        if (threadIdx.x == 0) s_item = gridDim.x + atomicAdd(work_counter, 1u);
        __syncthreads();
        // KEEP keys per thread stay in registers with their buckets (all of a
        // small cluster's); the rest are read and bucketed twice
        unsigned long long key[KEEP];
        uint32_t bkt[KEEP];
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            const uint32_t i = threadIdx.x + u * THREADS;
            key[u] = i < n ? __ldcg(src + i) : 0ull;
        }
        // counts the buckets; a warp's part of them is [h0, h1).  False, where
        // the buckets may be made anew, if ranking would take too many steps.
        auto count = [&](auto bucket, uint32_t h0, uint32_t h1, bool may_split) {
#pragma unroll
            for (int u = 0; u < KEEP; u++) {
                const uint32_t i = threadIdx.x + u * THREADS;
                bkt[u] = bucket(key[u]);
                if (i < n) atomicAdd(&hist[bkt[u]], 1u);
            }
            for (uint32_t i = threadIdx.x + KEEP * THREADS; i < n; i += THREADS) atomicAdd(&hist[bucket(__ldcg(src + i))], 1u);
            __syncthreads();
            uint32_t sum = 0;
            for (uint32_t h = h0 + lane; h < h1; h += 32) sum += hist[h];
            sum = __reduce_add_sync(0xFFFFFFFFu, sum);
            if (lane == 0) red32[w] = sum;
            if (!may_split) {
                __syncthreads();
                return true;
            }
            uint32_t steps = 0;  // n^2 < 2^31
            for (uint32_t h = h0 + lane; h < h1; h += 32) steps += hist[h] * hist[h];
            return !__syncthreads_or(__reduce_add_sync(0xFFFFFFFFu, steps) > SPLIT_STEPS * n);
        };
        // prefixes the counts, places the keys and ranks each in its bucket
        auto order = [&](auto bucket, uint32_t h0, uint32_t h1) {
            uint32_t carry = __reduce_add_sync(0xFFFFFFFFu, lane < w ? red32[lane] : 0u);
            for (uint32_t h = h0 + lane; h < h1; h += 32) {
                const uint32_t v = hist[h];
                uint32_t x = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                    if ((int)lane >= o) x += y;
                }
                hist[h] = carry + x - v;
                carry += __shfl_sync(0xFFFFFFFFu, x, 31);
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < KEEP; u++)
                if (threadIdx.x + u * THREADS < n) X[atomicAdd(&hist[bkt[u]], 1u)] = key[u];
            for (uint32_t i = threadIdx.x + KEEP * THREADS; i < n; i += THREADS) {
                const unsigned long long k = __ldcg(src + i);
                X[atomicAdd(&hist[bucket(k)], 1u)] = k;
            }
            __syncthreads();
            // hist[b] is now the end of bucket b.  Two keys per thread and step,
            // so their image reads overlap.
            for (uint32_t i0 = threadIdx.x; i0 < n; i0 += 2 * THREADS) {
                unsigned long long k[2];
                uint32_t rank[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const uint32_t i = i0 + u * THREADS;
                    k[u] = 0ull;
                    rank[u] = INVALID;
                    if (i >= n) continue;
                    k[u] = X[i];
                    const uint32_t b = bucket(k[u]), lo = b ? hist[b - 1] : 0u, hi = hist[b];
                    uint32_t r = lo;
                    for (uint32_t q = lo; q < i; q++) r += X[q] <= k[u] ? 1u : 0u;
                    for (uint32_t q = i + 1; q < hi; q++) r += X[q] < k[u] ? 1u : 0u;
                    rank[u] = r;
                }
                unsigned long long v[2];
#pragma unroll
                for (int u = 0; u < 2; u++) v[u] = linefit_rxyw((uint32_t)k[u], F.width, F.height, F.grey);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    if (rank[u] == INVALID) continue;
                    const uint32_t packed = (uint32_t)k[u];
                    atag_cluster_point cp;
                    cp.packed_x = (uint16_t)packed;
                    cp.packed_y = (uint16_t)(packed >> 16);
                    cp.slope = float_from_order_key((uint32_t)(k[u] >> 32));
                    F.cluster_points[start + rank[u]] = cp;
                    __stcg(src + rank[u], v[u]);
                }
            }
        };
        // each warp takes a contiguous part of the buckets, in rows of 32
        const uint32_t per = max(nb / W, 32u), h0 = w * per, h1 = min(nb, h0 + per);
        if (count(by_theta, h0, h1, n > SPLIT_MIN)) {
            order(by_theta, h0, h1);
        } else {
            for (uint32_t i = threadIdx.x; i < SPLIT; i += THREADS) {
                hist[i] = 0u;
                cuts[i] = __ldcg(src + i * n / SPLIT);
            }
            __syncthreads();
            bitonic_sort_u64(cuts, SPLIT);
            static_assert(SPLIT % (32 * W) == 0, "rows of 32 buckets per warp");
            const uint32_t s0 = w * (SPLIT / W), s1 = s0 + SPLIT / W;
            count(by_cuts, s0, s1, false);
            order(by_cuts, s0, s1);
        }
        __syncthreads();
        // moments of each run of CE_RUN points: W, Mx and My fit 32 bits (W <=
        // 362, rx, ry <= 8193)
        const uint32_t nruns = (n + CE_RUN - 1) / CE_RUN;
        for (uint32_t r = w; r < nruns; r += W) {
            uint32_t mx = 0, my = 0, mw = 0;
            long long xx = 0, yy = 0, xy = 0;
            const uint32_t i1 = min(n, (r + 1) * CE_RUN);
            for (uint32_t i = r * CE_RUN + lane; i < i1; i += 32) {
                const Moment m = moment_of(__ldcg(src + i));
                mx += (uint32_t)m.Mx;
                my += (uint32_t)m.My;
                mw += (uint32_t)m.W;
                xx = wadd(xx, m.Mxx);
                yy = wadd(yy, m.Myy);
                xy = wadd(xy, m.Mxy);
            }
            mx = __reduce_add_sync(0xFFFFFFFFu, mx);
            my = __reduce_add_sync(0xFFFFFFFFu, my);
            mw = __reduce_add_sync(0xFFFFFFFFu, mw);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                xx = wadd(xx, __shfl_xor_sync(0xFFFFFFFFu, xx, o));
                yy = wadd(yy, __shfl_xor_sync(0xFFFFFFFFu, yy, o));
                xy = wadd(xy, __shfl_xor_sync(0xFFFFFFFFu, xy, o));
            }
            if (lane == 0) {
                red_m[0][r] = mx; red_m[1][r] = my; red_m[2][r] = xx;
                red_m[3][r] = yy; red_m[4][r] = xy; red_m[5][r] = mw;
            }
        }
        __syncthreads();
        // their exclusive prefixes, component c on warp c mod W
        for (uint32_t c = w; c < 6; c += W) {
            long long carry = 0;
            for (uint32_t r0 = 0; r0 < nruns; r0 += 32) {
                const uint32_t r = r0 + lane;
                const long long v = r < nruns ? red_m[c][r] : 0ll;
                long long x = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                    if ((int)lane >= o) x = wadd(x, y);
                }
                if (r < nruns) F.runs[F.cluster_runs[cid] + r].before[c] = wadd(carry, wsub(x, v));
                carry = wadd(carry, __shfl_sync(0xFFFFFFFFu, x, 31));
            }
        }
        for (uint32_t r = threadIdx.x; r < nruns; r += THREADS) {
            RunInfo& R = F.runs[F.cluster_runs[cid] + r];
            R.cluster = cid;
            R.first = r * CE_RUN;
        }
        item = s_item;
        __syncthreads();  // the shared memory is free for the next cluster
    }
}

__global__ void __launch_bounds__(CF_SMALL_THREADS, 4) k_cluster_sort_small(const __grid_constant__ FrameSet fs,
                                                                        const uint32_t* __restrict__ work_offsets,
                                                                        uint32_t n_frames,
                                                                        uint32_t* __restrict__ work_counter,
                                                                        uint32_t cap) {
    cluster_sort<CF_SMALL_THREADS, CF_SMALL_CAP / CF_SMALL_THREADS, CF_SMALL_NB, CF_SMALL_CAP / CE_RUN>(fs, work_offsets, n_frames, work_counter, cap);
}
__global__ void __launch_bounds__(CF_LARGE_THREADS, 1) k_cluster_sort_large(const __grid_constant__ FrameSet fs,
                                                                           const uint32_t* __restrict__ work_offsets,
                                                                           uint32_t n_frames,
                                                                           uint32_t* __restrict__ work_counter,
                                                                           uint32_t cap) {
    cluster_sort<CF_LARGE_THREADS, 4, CF_LARGE_NB, CF_MAX_RUNS>(fs, work_offsets, n_frames, work_counter, cap);
}

// ---------------------------------------------------------------------------
// 4b. the segmented inclusive scan of the moments (main.cpp:796-801) and
// fit_lines (fit_quad.cpp:153-375) in its cyclic form: the error of the window
// around each point, the 7-tap filter and the strict local maxima.
// One warp per run of up to CE_RUN consecutive points of one cluster.  It
// reads the line-fit inputs of the run and, for the errors, of 24 points on
// either side (cyclic), and scans them in chunks of 128: lane l has points 4 l
// .. 4 l + 3, one warp scan of the lanes' sums, then each lane adds its points
// one by one.  With the moments of the cluster's earlier runs that gives the
// run's LineFitPoints, and the scan itself, kept in shared memory, every
// window's moment: integer sums, so the same whatever they start from, and no
// prefix sum is read back from memory.  W, Mx and My stay below 2^32 over a run
// and its margins (W <= 362, coordinates <= 2^15).  Then lane l filters
// positions 8 l .. 8 l + 7 from 14 errors and compares with its neighbour
// lanes'.  Maxima are appended to their cluster's candidate list in the
// cluster's segment of errbuf (a cyclic sequence of n values has at most n/2
// strict maxima).  Bound by latency (128 registers and 50 KB of shared memory
// leave 16 warps per SM); as two kernels, the errors reading prefix sums back,
// 64 frames of 1080p took 125 + 197 us and a lone frame 10 + 30 us, now 277 and
// 20 us (with the cheaper hypotf and conversions in both: 125 + 235 and 10 + 16).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cyclic(int i, int n) {  // i in [-n, 3n): n is at least CE_MARGIN
    if (i < 0) i += n;
    while (i >= n) i -= n;
    return (uint32_t)i;
}

__device__ __forceinline__ void store_sector(void* p, long long a, long long b, long long c, long long d) {
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

struct ShortMoment {  // of at most a run and its margins
    uint32_t w, mx, my;
    unsigned long long xx, yy, xy;
};
__device__ __forceinline__ ShortMoment s_add(const ShortMoment& a, const ShortMoment& b) {
    return ShortMoment{a.w + b.w, a.mx + b.mx, a.my + b.my, a.xx + b.xx, a.yy + b.yy, a.xy + b.xy};
}
__device__ __forceinline__ ShortMoment s_sub(const ShortMoment& a, const ShortMoment& b) {
    return ShortMoment{a.w - b.w, a.mx - b.mx, a.my - b.my, a.xx - b.xx, a.yy - b.yy, a.xy - b.xy};
}
__device__ __forceinline__ ShortMoment s_shfl(const ShortMoment& a, int src) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    return ShortMoment{__shfl_sync(FULL, a.w, src), __shfl_sync(FULL, a.mx, src), __shfl_sync(FULL, a.my, src),
                       __shfl_sync(FULL, a.xx, src), __shfl_sync(FULL, a.yy, src), __shfl_sync(FULL, a.xy, src)};
}
// of one point's line-fit inputs (linefit_rxyw)
__device__ __forceinline__ ShortMoment s_of(unsigned long long v) {
    const uint32_t rx = (uint32_t)v & 0xFFFFu, ry = (uint32_t)v >> 16, w = (uint32_t)(v >> 32);
    const uint32_t ax = w * rx, ay = w * ry;
    return ShortMoment{w, ax, ay, (unsigned long long)ax * rx, (unsigned long long)ay * ry, (unsigned long long)ax * ry};
}

// fit_line's error (fit_quad.cpp:37-105) of a window of `count` <= 41 points:
// the same integers, in the widths they need
__device__ __forceinline__ float window_fit_error(const ShortMoment& m, uint32_t count) {
    const unsigned long long cxx = m.xx * m.w - (unsigned long long)m.mx * m.mx;
    const unsigned long long cyy = m.yy * m.w - (unsigned long long)m.my * m.my;
    const unsigned long long cxy = m.xy * m.w - (unsigned long long)m.mx * m.my;
    const float sdist = hypot_f(i64_to_f32_rn((long long)(cxx - cyy)), i64_to_f32_rn((long long)(2 * cxy)));
    const float num = __fsub_rn(i64_to_f32_rn((long long)(cxx + cyy)), sdist);
    const float eig = __fdiv_rn(num, (float)(8u * m.w * m.w));
    return __fmul_rn((float)count, eig);
}

constexpr uint32_t CE_MARGIN = 24;                           // window (20) and filter (3) reach, and a neighbour
// A run's margins go round the cluster at most once, and its windows reach at
// least two points to either side (fewer give no error, fit_quad.cpp:202-225).
static_assert(CE_MARGIN <= MIN_CLUSTER_POINTS && MIN_CLUSTER_POINTS / 12 >= 2, "smallest cluster of the window errors");
constexpr uint32_t CE_SPAN = CE_RUN + 2 * CE_MARGIN;         // points a warp scans
constexpr uint32_t CE_ERRS = CE_RUN + 8;                     // errors of positions -4 .. CE_RUN + 3
// Sums of the points before local index j at [CE_BASE + j]: the base keeps a
// lane's four sums (j = i + 1 .. i + 4, i a multiple of 4) 16-byte aligned.
constexpr uint32_t CE_BASE = 3;
struct RunSums {
    unsigned long long xx[CE_BASE + CE_SPAN + 5], yy[CE_BASE + CE_SPAN + 5], xy[CE_BASE + CE_SPAN + 5];
    uint32_t w[CE_BASE + CE_SPAN + 5], mx[CE_BASE + CE_SPAN + 5], my[CE_BASE + CE_SPAN + 5];
    float err[CE_ERRS + CE_ERRS / 8];  // error i at i + i / 8: lanes eight apart read distinct banks
    uint32_t pad_[3];
};
static_assert((CE_BASE + CE_SPAN + 5) % 4 == 0 && sizeof(RunSums) % 16 == 0, "16-byte aligned sums");

template <bool ERRORS>
__device__ __forceinline__ void cluster_run(const FrameDesc& F, const RunInfo& R, RunSums* S) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31, cid = R.cluster, first = R.first;
    const atag_cluster_extents ext = F.cluster_extents[cid];
    const uint32_t n = ext.count, len = min(CE_RUN, n - first);
    constexpr uint32_t M = ERRORS ? CE_MARGIN : 0u;
    const uint32_t span = len + 2 * M;  // local index i: point first - M + i (cyclic)
    const unsigned long long* in = F.sortbuf + ext.start;
    // a 32-byte sector per store where the array's alignment allows it (the
    // detector's own always does; a caller's array may not)
    const bool wide = (reinterpret_cast<uintptr_t>(F.line_fit) & 31u) == 0;
    atag_line_fit_point* out = F.line_fit + ext.start + first;
    ShortMoment carry{0, 0, 0, 0ull, 0ull, 0ull}, start{0, 0, 0, 0ull, 0ull, 0ull};
    if (ERRORS && lane == 0) {
        S->w[CE_BASE] = S->mx[CE_BASE] = S->my[CE_BASE] = 0u;
        S->xx[CE_BASE] = S->yy[CE_BASE] = S->xy[CE_BASE] = 0ull;
    }
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < span; c0 += 128) {
        const uint32_t i0 = c0 + 4 * lane;
        unsigned long long v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t i = i0 + q;
            v[q] = i < span ? __ldcg(in + (ERRORS ? cyclic((int)(first + i) - (int)M, (int)n) : first + i)) : 0ull;
        }
        ShortMoment sum = s_of(v[0]);
#pragma unroll
        for (int q = 1; q < 4; q++) sum = s_add(sum, s_of(v[q]));
        ShortMoment incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const ShortMoment t{__shfl_up_sync(FULL, incl.w, o),  __shfl_up_sync(FULL, incl.mx, o),
                                __shfl_up_sync(FULL, incl.my, o), __shfl_up_sync(FULL, incl.xx, o),
                                __shfl_up_sync(FULL, incl.yy, o), __shfl_up_sync(FULL, incl.xy, o)};
            if ((int)lane >= o) incl = s_add(incl, t);
        }
        ShortMoment at = s_add(carry, s_sub(incl, sum));  // of the points before this lane's
        carry = s_add(carry, s_shfl(incl, 31));
        // the sums before the run itself: after the last margin point
        if (ERRORS && c0 == 0) start = s_shfl(s_add(at, sum), (int)(M / 4 - 1));
        ShortMoment p[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            at = s_add(at, s_of(v[q]));
            p[q] = at;
            const uint32_t i = i0 + q;
            if ((int)i < (int)M || i - M >= len) continue;
            const ShortMoment d = s_sub(at, start);
            const long long Mx = wadd(R.before[0], d.mx), My = wadd(R.before[1], d.my), W = wadd(R.before[5], d.w);
            const long long Mxx = wadd(R.before[2], (long long)d.xx), Myy = wadd(R.before[3], (long long)d.yy);
            const long long Mxy = wadd(R.before[4], (long long)d.xy);
            atag_line_fit_point* o = out + (i - M);
            if (wide) {
                store_sector(o, Mx, My, Mxx, Myy);
                store_sector(reinterpret_cast<char*>(o) + 32, Mxy, W, 0ll, 0ll);
            } else {
                store_moment(o, Moment{Mx, My, Mxx, Myy, Mxy, W});
            }
        }
        if (ERRORS && i0 < span) {
            const uint32_t j = CE_BASE + i0 + 1;
            *reinterpret_cast<uint4*>(S->w + j) = make_uint4(p[0].w, p[1].w, p[2].w, p[3].w);
            *reinterpret_cast<uint4*>(S->mx + j) = make_uint4(p[0].mx, p[1].mx, p[2].mx, p[3].mx);
            *reinterpret_cast<uint4*>(S->my + j) = make_uint4(p[0].my, p[1].my, p[2].my, p[3].my);
#pragma unroll
            for (int q = 0; q < 4; q += 2) {
                *reinterpret_cast<ulonglong2*>(S->xx + j + q) = make_ulonglong2(p[q].xx, p[q + 1].xx);
                *reinterpret_cast<ulonglong2*>(S->yy + j + q) = make_ulonglong2(p[q].yy, p[q + 1].yy);
                *reinterpret_cast<ulonglong2*>(S->xy + j + q) = make_ulonglong2(p[q].xy, p[q + 1].xy);
            }
        }
    }
    if (!ERRORS) return;
    __syncwarp();
    // error i: position first - 4 + i, the window of k points on either side
    const uint32_t k = min(20u, n / 12u);
    constexpr uint32_t ILP = 3;
    for (uint32_t i0 = lane; i0 < len + 8; i0 += 32 * ILP) {
#pragma unroll
        for (uint32_t u = 0; u < ILP; u++) {
            const uint32_t i = i0 + 32 * u;
            if (i >= len + 8) break;
            const uint32_t lo = CE_BASE + (M - 4) + i - k, hi = lo + 2 * k + 1;
            const ShortMoment m{S->w[hi] - S->w[lo],   S->mx[hi] - S->mx[lo], S->my[hi] - S->my[lo],
                                S->xx[hi] - S->xx[lo], S->yy[hi] - S->yy[lo], S->xy[hi] - S->xy[lo]};
            S->err[i + (i >> 3)] = window_fit_error(m, 2 * k + 1);
        }
    }
    __syncwarp();
    // cyclic 7-tap filter (fit_quad.cpp:296-324): output o is position
    // first + o, from errors o + 1 .. o + 7
    auto filter = [&](const float* e) {
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < 7; j++) acc = __fadd_rn(acc, __fmul_rn(e[j], filter_tap(j)));
        return acc;
    };
    auto err_at = [&](uint32_t i) { return S->err[i + (i >> 3)]; };
    float f[10];  // outputs 8 l - 1 .. 8 l + 8
    {
        float e[14];
#pragma unroll
        for (int j = 0; j < 14; j++) e[j] = err_at(min(8 * lane + 1 + j, CE_ERRS - 1));
#pragma unroll
        for (int o = 0; o < 8; o++) f[1 + o] = filter(e + o);
        // the outputs before the run (lane 0) and past a full one (lane 31)
        const uint32_t b = lane == 0 ? 0u : CE_RUN + 1u;
#pragma unroll
        for (int j = 0; j < 7; j++) e[j] = err_at(b + j);
        const float edge = filter(e);
        f[0] = __shfl_up_sync(FULL, f[8], 1);
        f[9] = __shfl_down_sync(FULL, f[1], 1);
        if (lane == 0) f[0] = edge;
        if (lane == 31) f[9] = edge;
    }
    // strict local maxima (fit_quad.cpp:341-371) with error != 0
    // (main.cpp:832-835); global point 0 is never a corner (the first
    // work-group's first output is x = 1, fit_quad.cpp:182-190)
    unsigned long long* cand = reinterpret_cast<unsigned long long*>(F.errbuf) + ext.start;
#pragma unroll
    for (int o = 0; o < 8; o++) {
        const uint32_t li = first + 8 * lane + o;
        const float cur = f[1 + o];
        if (8 * lane + o < len && cur > f[o] && cur > f[o + 2] && cur != 0.0f && !(cid == 0 && li == 0)) {
            const uint32_t at = atomicAdd(F.peak_count + cid, 1u);
            cand[at] = ((unsigned long long)float_order_key(cur) << 32) | (uint32_t)(~li);
        }
    }
    __syncwarp();
}

// Items go round the CTAs first, so that a few still use every SM.
constexpr int CE_WARPS = 4;
static_assert(CE_LINES_SMEM == CE_WARPS * sizeof(RunSums), "dynamic shared memory of k_cluster_lines");
__global__ void __launch_bounds__(32 * CE_WARPS, 4) k_cluster_lines(const __grid_constant__ FrameSet fs,
                                                                    const uint32_t* __restrict__ run_offsets,
                                                                    uint32_t n_frames) {
    extern __shared__ __align__(16) unsigned char smem_runs[];
    const uint32_t wid = threadIdx.x >> 5, total = run_offsets[n_frames];
    RunSums* S = reinterpret_cast<RunSums*>(smem_runs) + wid;
    for (uint32_t item = blockIdx.x + gridDim.x * wid; item < total; item += gridDim.x * CE_WARPS) {
        const uint32_t fidx = find_frame(run_offsets, n_frames, item);
        const FrameDesc& F = fs.of_table(fidx);
        cluster_run<true>(F, F.runs[item - run_offsets[fidx]], S);
    }
}
// the stage entry point: prefix sums only
__global__ void __launch_bounds__(32 * CE_WARPS, 4) k_cluster_prefix(const __grid_constant__ FrameSet fs,
                                                                     const uint32_t* __restrict__ run_offsets) {
    const FrameDesc& F = fs.get(0);
    const uint32_t total = run_offsets[1];
    for (uint32_t item = blockIdx.x + gridDim.x * (threadIdx.x >> 5); item < total; item += gridDim.x * CE_WARPS)
        cluster_run<false>(F, F.runs[item], nullptr);
}

// ---------------------------------------------------------------------------
// 5. peak extents (D10-D12), do_indexing + corners, ordered quads
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_peaks_scan(const __grid_constant__ FrameSet fs, BatchOffsets a) {
    if (fs.overlap) await_previous_kernel();
    const FrameDesc& F = fs.of_table(blockIdx.x);
    __shared__ uint32_t red[33];
    const uint32_t C = F.counters[CNT_CLUSTERS];
    uint32_t carry_q = 0, carry_k = 0;
    for (uint32_t c0 = 0; c0 < C; c0 += blockDim.x) {
        uint32_t c = c0 + threadIdx.x;
        uint32_t k = c < C ? F.peak_count[c] : 0u;
        uint32_t tq, tk;
        uint32_t q = carry_q + block_exclusive_scan_u32(k ? 1u : 0u, red, &tq);
        uint32_t s = carry_k + block_exclusive_scan_u32(k, red, &tk);
        if (k) {
            F.peak_clusters[q] = c;
            F.peak_extents[q] = atag_peak_extents{s, k};
        }
        carry_q += tq;
        carry_k += tk;
    }
    if (threadIdx.x == 0) {
        F.counters[CNT_PEAKCLU] = carry_q;
        F.stats->n_corners = carry_k;
        F.stats->n_peak_clusters = carry_q;
    }
    batch_offsets(fs, a);
}

// The 10 best corner candidates of a cluster by (error desc, index asc), one
// per lane from lane 0 (0 past the last): the corner sort of main.cpp:856-863
// restricted to what do_indexing reads (fit_quad.cpp:411-414 uses at most 10
// corners).
__device__ __forceinline__ unsigned long long best_candidates(const unsigned long long* cand, uint32_t n) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr int KEEP = 4;  // per lane in registers; clusters with more candidates than fit read the rest each time
    const uint32_t lane = threadIdx.x & 31, take = n < 10u ? n : 10u;
    unsigned long long c[KEEP], mine = 0, last = ~0ull;
#pragma unroll
    for (int u = 0; u < KEEP; u++) c[u] = lane + 32u * u < n ? cand[lane + 32u * u] : 0ull;
    for (uint32_t j = 0; j < take; j++) {
        unsigned long long best = 0;
#pragma unroll
        for (int u = 0; u < KEEP; u++)
            if (c[u] < last && c[u] > best) best = c[u];
        for (uint32_t i = lane + 32u * KEEP; i < n; i += 32) {
            const unsigned long long key = cand[i];
            if (key < last && key > best) best = key;
        }
        const uint32_t hi = __reduce_max_sync(FULL, (uint32_t)(best >> 32));
        const uint32_t lo = __reduce_max_sync(FULL, (uint32_t)(best >> 32) == hi ? (uint32_t)best : 0u);
        last = (unsigned long long)hi << 32 | lo;
        if (lane == j) mine = last;
    }
    return mine;
}

// One warp per cluster with peaks: its 10 best corners, the combination
// search, and the corners of the chosen four on lanes of their own.  Bound by
// the latency of one warp: the clusters go round the CTAs first, so that a
// lone frame's ~100 use every SM.  A lone 1080p frame's selection and search
// took 12 + 29 us as a kernel each with serial corners (25 now), 64 frames
// 30 + 133 us (82 now).
__global__ void __launch_bounds__(256) k_index_quads(const __grid_constant__ FrameSet fs,
                                                     const uint32_t* work_offsets, uint32_t n_frames,
                                                     PipelineParams p) {
    if (fs.overlap) await_previous_kernel();
    __shared__ SegmentTable T[8];  // one per warp
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t total = work_offsets[n_frames];
    for (uint32_t item = blockIdx.x + gridDim.x * wid; item < total; item += gridDim.x * 8) {
        const uint32_t fidx = find_frame(work_offsets, n_frames, item);
        const FrameDesc& F = fs.of_table(fidx);
        const uint32_t q = item - work_offsets[fidx];
        const uint32_t cid = F.peak_clusters[q], count = F.peak_count[cid];
        const atag_cluster_extents ce = F.cluster_extents[p.compat_peak_index ? q : cid];
        const unsigned long long key = best_candidates(
            reinterpret_cast<const unsigned long long*>(F.errbuf) + F.cluster_extents[cid].start, count);
        if (lane < min(count, 10u)) {
            atag_corner c;
            c.line_fit_point_index = ~(uint32_t)key;
            c.cluster_index = (uint16_t)cid;
            c.error = float_from_order_key((uint32_t)(key >> 32));
            F.peaks[(size_t)cid * 10 + lane] = c;
        }
        atag_fitted_quad* fq = F.fitted + q;
        QuadSide side;
        const int chosen = index_one_cluster(count, ~(uint32_t)key, F.line_fit + ce.start, ce.count, p.max_line_fit_mse,
                                             p.cos_critical_f, T[wid], fq, side);
        if (chosen < 0) {
            // no combination: the quad stays zero (main.cpp:318-319)
            for (uint32_t k = lane; k < sizeof(atag_fitted_quad) / 4; k += 32) reinterpret_cast<uint32_t*>(fq)[k] = 0u;
            if (lane == 0) F.quad_ok[q] = 0;
        } else {
            float line[4] = {0.0f, 0.0f, 0.0f, 0.0f}, cx, cy, e, mse;
            if (lane < 4) fit_line(side.m, side.points, line, &e, &mse);
            const bool any = __any_sync(0xFFFFFFFFu, lane < 4 && side.index != 0);
            const bool ok = __shfl_sync(0xFFFFFFFFu, (int)quad_corners8(line, p, cx, cy), 0) && any;
            atag_quad_corners& qc = F.quad_tmp[q];
            if (lane < 4) {
                qc.corners[lane][0] = cx;
                qc.corners[lane][1] = cy;
            } else if (lane == 4) {
                qc.reversed_border = (uint8_t)p.reversed_border;
                qc.pad_[0] = qc.pad_[1] = qc.pad_[2] = 0;
                qc.blob_index = q;
                F.quad_ok[q] = ok ? 1u : 0u;
            }
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(1024) k_compact_quads(const __grid_constant__ FrameSet fs) {
    if (fs.overlap) await_previous_kernel();
    const FrameDesc& F = fs.of_table(blockIdx.x);
    __shared__ uint32_t red[33];
    const uint32_t Cp = F.counters[CNT_PEAKCLU];
    uint32_t carry = 0, nfit = 0;
    for (uint32_t c0 = 0; c0 < Cp; c0 += blockDim.x) {
        uint32_t q = c0 + threadIdx.x;
        uint32_t ok = q < Cp ? F.quad_ok[q] : 0u;
        uint32_t fit = 0;
        if (q < Cp) {
            const atag_fitted_quad& fq = F.fitted[q];
            fit = (fq.indices[0] | fq.indices[1] | fq.indices[2] | fq.indices[3]) != 0;
        }
        uint32_t tot, tf;
        uint32_t pos = carry + block_exclusive_scan_u32(ok, red, &tot);
        block_exclusive_scan_u32(fit, red, &tf);
        if (ok) {
            if (pos < F.quad_cap) F.quads[pos] = F.quad_tmp[q];
        }
        carry += tot;
        nfit += tf;
    }
    if (threadIdx.x == 0) {
        if (carry > F.quad_cap) atomicOr(F.counters + CNT_STATUS, ATAG_DEVFLAG_QUAD_OVERFLOW);
        F.stats->n_fitted = nfit;
        F.stats->n_quads = carry < F.quad_cap ? carry : F.quad_cap;
        F.stats->status = F.counters[CNT_STATUS];
    }
}

#define BOUNDARY_KERNELS(SUFFIX, BEFORE)                                                                        \
    __global__ void __launch_bounds__(BP_W / 4 * 8, 16)                                                         \
        k_boundaries_pairs_r8##SUFFIX(const __grid_constant__ FrameSet fs, uint32_t min_size) {                 \
        BEFORE;                                                                                                 \
        boundaries_pairs_impl<8>(fs, min_size);                                                                 \
    }                                                                                                           \
    __global__ void __launch_bounds__(BP_W / 4 * 16, 8)                                                         \
        k_boundaries_pairs_r16##SUFFIX(const __grid_constant__ FrameSet fs, uint32_t min_size) {                \
        BEFORE;                                                                                                 \
        boundaries_pairs_impl<16>(fs, min_size);                                                                \
    }
BOUNDARY_KERNELS(, )
BOUNDARY_KERNELS(_overlapped, await_previous_kernel())
#undef BOUNDARY_KERNELS

}  // namespace atag
