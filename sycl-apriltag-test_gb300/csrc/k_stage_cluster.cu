// k_stage_cluster.cu — kernels of the stage entry points that stand in for
// the reference's oneDPL glue between its device functions:
//   atag_cluster       stages 4-11 (src/main.cpp:467-801), from the dense
//                      boundary planes that find_boundaries writes to the
//                      line-fit prefix sums that fit_lines reads;
//   atag_corner_peaks  stages 13-15 (src/main.cpp:832-907), from fit_lines'
//                      dense corner array to do_indexing's inputs.
// atag_cluster shares the fused detector's pair table, filter and cluster
// sorts (k_cluster.cu); only the entry and exit over the dense planes are
// here: the planes are read twice (sums per pair, then the points of the
// surviving clusters), so no compacted point list is ever written.
#include "atag_kernels.cuh"
#include "atag_pairs.cuh"

namespace atag {

// The planes are read in groups of PP_GROUP entries per warp, PP_UNROLL of
// them at once so that their loads are in flight together.
constexpr uint32_t PP_UNROLL = 4, PP_GROUP = 32 * PP_UNROLL;
constexpr uint32_t PP_LC = 32;  // pair table of a CTA; more pairs go straight to the frame's

struct PlanePairs {
    unsigned long long key[PP_LC], pxgx[PP_LC];
    uint32_t cnt[PP_LC], xmin[PP_LC], xmax[PP_LC], ymin[PP_LC], ymax[PP_LC];
    int gx[PP_LC], gy[PP_LC];
};

__device__ __forceinline__ int plane_pairs_insert(PlanePairs& T, unsigned long long key) {
    uint32_t h = hash_key(key) & (PP_LC - 1);
    for (uint32_t p = 0; p < PP_LC; p++) {
        const unsigned long long k = atomicCAS(&T.key[h], EMPTY_KEY, key);
        if (k == EMPTY_KEY || k == key) return (int)h;
        h = (h + 1) & (PP_LC - 1);
    }
    return -1;
}

// Stages 4 and 6: copy_if(point != 0) and reduce_by_segment of
// ClusterBounds::inital_from_point per pair key (cluster_bounds.h:27-45).
// The sort by key that separates them in the reference only orders the
// pairs, which k_pairs_finalize does on the distinct keys.  A CTA takes one
// stretch of the planes; a warp keeps the sums of one pair in registers, a
// point per lane, while its entries are of that pair, then adds them to the
// CTA's table, which goes to the frame's at the end.  Most points of a frame
// are of the pair of its two largest components: merged per warp and entry
// group into the frame's table, their atomics on one slot took 277 us for
// 1292 x 964 (30 now).
__global__ void __launch_bounds__(256) k_planes_pairs(const __grid_constant__ FrameSet fs,
                                                      const uint32_t* __restrict__ points,
                                                      const unsigned long long* __restrict__ keys, uint32_t n) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const FrameDesc& F = fs.get(0);
    uint32_t* status = F.counters + CNT_STATUS;
    __shared__ PlanePairs T;
    for (uint32_t i = threadIdx.x; i < PP_LC; i += blockDim.x) {
        T.key[i] = EMPTY_KEY;
        T.pxgx[i] = 0ull;
        T.cnt[i] = T.xmax[i] = T.ymax[i] = 0u;
        T.xmin[i] = T.ymin[i] = FULL;
        T.gx[i] = T.gy[i] = 0;
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    unsigned long long cur = EMPTY_KEY;
    uint32_t cnt = 0, xmn = FULL, xmx = 0, ymn = FULL, ymx = 0, found = 0;
    int gx = 0, gy = 0, px = 0;
    auto to_frame = [&](unsigned long long key, uint32_t c, uint32_t x0, uint32_t x1, uint32_t y0, uint32_t y1, int sx,
                        int sy, unsigned long long sp) {
        const uint32_t gs = global_insert(F, key);
        if (gs == INVALID) atomicOr(status, ATAG_DEVFLAG_PAIR_OVERFLOW);
        else global_flush(F, key, gs, c, x0, x1, y0, y1, sx, sy, sp);
    };
    auto flush = [&]() {
        if (cnt == 0) return;
        const uint32_t x0 = __reduce_min_sync(FULL, xmn), x1 = __reduce_max_sync(FULL, xmx);
        const uint32_t y0 = __reduce_min_sync(FULL, ymn), y1 = __reduce_max_sync(FULL, ymx);
        const int sx = __reduce_add_sync(FULL, gx), sy = __reduce_add_sync(FULL, gy), sp = __reduce_add_sync(FULL, px);
        if (lane != 0) return;
        const unsigned long long spx = (unsigned long long)(long long)sp;
        const int t = plane_pairs_insert(T, cur);
        if (t < 0) {
            to_frame(cur, cnt, x0, x1, y0, y1, sx, sy, spx);
            return;
        }
        atomicAdd(&T.cnt[t], cnt);
        atomicMin(&T.xmin[t], x0);
        atomicMax(&T.xmax[t], x1);
        atomicMin(&T.ymin[t], y0);
        atomicMax(&T.ymax[t], y1);
        atomicAdd(&T.gx[t], sx);
        atomicAdd(&T.gy[t], sy);
        atomicAdd(&T.pxgx[t], spx);
    };
    const uint32_t groups = (n + PP_GROUP - 1) / PP_GROUP, per = (groups + gridDim.x - 1) / gridDim.x;
    const uint32_t g0 = blockIdx.x * per, g1 = min(groups, g0 + per);
    for (uint32_t g = g0 + (threadIdx.x >> 5); g < g1; g += warps) {
        uint32_t p[PP_UNROLL];
        unsigned long long k[PP_UNROLL];
#pragma unroll
        for (uint32_t u = 0; u < PP_UNROLL; u++) {
            const uint32_t i = g * PP_GROUP + 32 * u + lane;
            p[u] = i < n ? __ldg(points + i) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < PP_UNROLL; u++)
            k[u] = p[u] ? __ldg(keys + (g * PP_GROUP + 32 * u + lane)) : EMPTY_KEY;
#pragma unroll
        for (uint32_t u = 0; u < PP_UNROLL; u++) {
            const bool v = p[u] != 0u;
            unsigned pend = __ballot_sync(FULL, v);
            if (!pend) continue;
            found += (uint32_t)__popc(pend);
            const uint32_t xd = bp_xd(p[u]), yd = bp_yd(p[u]);
            const int dx = bp_gx(p[u]), dy = bp_gy(p[u]);
            // the current pair's points first, so that it is left once
            unsigned m = __ballot_sync(FULL, v && k[u] == cur);
            while (true) {
                if (m) {
                    pend &= ~m;
                    cnt += (uint32_t)__popc(m);
                    if ((m >> lane) & 1u) {
                        xmn = min(xmn, xd);
                        xmx = max(xmx, xd);
                        ymn = min(ymn, yd);
                        ymx = max(ymx, yd);
                        gx += dx;
                        gy += dy;
                        px += (int)xd * dx + (int)yd * dy;
                    }
                }
                // (a lane's and a warp's sums of up to 16384 points fit 32 bits)
                if (!pend && cnt < 16384u - 32u) break;
                flush();
                if (pend) cur = __shfl_sync(FULL, k[u], __ffs(pend) - 1);
                cnt = xmx = ymx = 0;
                xmn = ymn = FULL;
                gx = gy = px = 0;
                if (!pend) break;
                m = __ballot_sync(FULL, v && k[u] == cur);
            }
        }
    }
    flush();
    if (lane == 0 && found) atomicAdd(F.counters + CNT_ALLPOINTS, found);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < PP_LC; i += blockDim.x)
        if (T.key[i] != EMPTY_KEY)
            to_frame(T.key[i], T.cnt[i], T.xmin[i], T.xmax[i], T.ymin[i], T.ymax[i], T.gx[i], T.gy[i], T.pxgx[i]);
}

// Stage 7: each point of a pair that passed the filter goes to its
// cluster's segment with its calc_theta key (main.cpp:621-675); the
// cluster sorts then order each segment by (slope, point).  A lane looks a
// key up only when it differs from its last one, and points of dropped pairs
// (most) take no part after that.
__global__ void __launch_bounds__(256) k_planes_scatter(const __grid_constant__ FrameSet fs,
                                                        const uint32_t* __restrict__ points,
                                                        const unsigned long long* __restrict__ keys, uint32_t n) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const FrameDesc& F = fs.get(0);
    const uint32_t lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const uint32_t groups = (n + PP_GROUP - 1) / PP_GROUP, per = (groups + gridDim.x - 1) / gridDim.x;
    const uint32_t g0 = blockIdx.x * per, g1 = min(groups, g0 + per);
    unsigned long long last = EMPTY_KEY;
    uint32_t last_cid = INVALID;
    for (uint32_t g = g0 + (threadIdx.x >> 5); g < g1; g += warps) {
        uint32_t p[PP_UNROLL];
        unsigned long long k[PP_UNROLL];
#pragma unroll
        for (uint32_t u = 0; u < PP_UNROLL; u++) {
            const uint32_t i = g * PP_GROUP + 32 * u + lane;
            p[u] = i < n ? __ldg(points + i) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < PP_UNROLL; u++)
            k[u] = p[u] ? __ldg(keys + (g * PP_GROUP + 32 * u + lane)) : EMPTY_KEY;
#pragma unroll
        for (uint32_t u = 0; u < PP_UNROLL; u++) {
            uint32_t cid = INVALID;
            if (p[u]) {
                if (k[u] != last) {
                    const uint32_t slot = global_lookup(F, k[u]);
                    last = k[u];
                    last_cid = slot != INVALID ? F.pair_cluster[slot] : INVALID;
                }
                cid = last_cid;
            }
            if (!__any_sync(FULL, cid != INVALID)) continue;
            const unsigned mask = __match_any_sync(FULL, cid);
            if (cid != INVALID) {
                const int leader = __ffs(mask) - 1;
                uint32_t b = 0;
                if ((int)lane == leader) b = atomicAdd(F.cluster_cursor + cid, (uint32_t)__popc(mask));
                b = __shfl_sync(mask, b, leader);
                const uint32_t rank = __popc(mask & ((1u << lane) - 1u));
                const atag_cluster_extents ext = F.cluster_extents[cid];
                const float2 ctr = F.cluster_center[cid];
                const float theta = calc_theta(p[u], ctr.x, ctr.y);
                if (b + rank < ext.count)
                    F.sortbuf[ext.start + b + rank] = ((unsigned long long)float_order_key(theta) << 32) | p[u];
            }
        }
    }
}

// The 16-bit cluster index of every sorted point (main.cpp:641), the
// filtered keys if asked, and the counters.  One warp per cluster.
__global__ void __launch_bounds__(256) k_stage_cluster_out(const __grid_constant__ FrameSet fs,
                                                           uint16_t* cluster_indices,
                                                           unsigned long long* cluster_keys_out) {
    const FrameDesc& F = fs.get(0);
    const uint32_t C = F.counters[CNT_CLUSTERS];
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint32_t c = blockIdx.x * wpb + (threadIdx.x >> 5); c < C; c += gridDim.x * wpb) {
        const atag_cluster_extents ext = F.cluster_extents[c];
        for (uint32_t k = lane; k < ext.count; k += 32) cluster_indices[ext.start + k] = (uint16_t)c;
        if (lane == 0 && cluster_keys_out) cluster_keys_out[c] = F.cluster_keys[c];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        F.stats->n_corners = 0;
        F.stats->n_peak_clusters = 0;
        F.stats->n_fitted = 0;
        F.stats->n_quads = 0;
        F.stats->status = F.counters[CNT_STATUS];
    }
}

// ---------------------------------------------------------------------------
// Stages 13-15: copy_if(error != 0) over the dense corner array, sort by
// (cluster ascending, error descending) and one PeakExtents per cluster
// with corners.  fit_lines writes a cluster's corners inside its extent, so
// the compaction and the sort run per cluster: counts, an exclusive scan
// over the clusters, then each cluster's corners sorted in shared memory.
// The reference's sort leaves ties unordered; here they go by position.
// ---------------------------------------------------------------------------
// Bound by the latency of the loads.  Clusters of up to PK_WARP points take a
// warp each, larger ones a CTA of 1024 threads, PK_UNROLL points per thread at
// once.  Clusters go round the CTAs first, then their warps, so that a few use
// every SM.  With a warp for clusters of any size the counts of 1292 x 964 took
// 68 us (9 now), the sort on 256 threads 37 (19 on 1024); with a CTA for clusters
// of any size 65,535 clusters of 24 points took 887 us in all (107 now, 671 on
// warps and 256 threads), 4,000 of them 69 (17, 57).
constexpr int PK_UNROLL = 4;
constexpr uint32_t PK_WARP = 32 * PK_UNROLL * 2, PK_WARPS = 32;

__global__ void __launch_bounds__(32 * PK_WARPS) k_peaks_count(const atag_corner* __restrict__ found,
                                                     const atag_cluster_extents* __restrict__ ext,
                                                     uint32_t n_clusters, uint32_t* __restrict__ counts) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    __shared__ uint32_t red[33], s_large[PK_WARPS];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    auto count = [&](const atag_cluster_extents& e, uint32_t first, uint32_t step) {
        uint32_t k = 0;
#pragma unroll PK_UNROLL
        for (uint32_t i = first; i < e.count; i += step) k += found[(size_t)e.start + i].error != 0.0f ? 1u : 0u;
        return k;
    };
    for (uint32_t c0 = blockIdx.x; c0 < n_clusters; c0 += gridDim.x * PK_WARPS) {
        const uint32_t c = c0 + gridDim.x * wid;
        uint32_t large = INVALID;
        if (c < n_clusters) {
            const atag_cluster_extents e = ext[c];
            if (e.count > PK_WARP) {
                large = c;
            } else {
                const uint32_t k = __reduce_add_sync(FULL, count(e, lane, 32));
                if (lane == 0) counts[c] = k;
            }
        }
        if (lane == 0) s_large[wid] = large;
        __syncthreads();
        for (unsigned m = __ballot_sync(FULL, s_large[lane] != INVALID); m; m &= m - 1) {
            const uint32_t cl = s_large[__ffs(m) - 1];
            const uint32_t k = block_sum_u32(count(ext[cl], threadIdx.x, blockDim.x), red);
            if (threadIdx.x == 0) counts[cl] = k;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(1024) k_peaks_offsets(const uint32_t* __restrict__ counts, uint32_t n_clusters,
                                                        uint32_t* __restrict__ offsets,
                                                        atag_peak_extents* __restrict__ peak_extents,
                                                        uint32_t extents_cap, uint32_t corner_cap,
                                                        uint32_t* __restrict__ d_counts) {
    __shared__ uint32_t red[33];
    uint32_t carry_q = 0, carry_k = 0;
    for (uint32_t c0 = 0; c0 < n_clusters; c0 += blockDim.x) {
        const uint32_t c = c0 + threadIdx.x;
        const uint32_t k = c < n_clusters ? counts[c] : 0u;
        uint32_t tq, tk;
        const uint32_t q = carry_q + block_exclusive_scan_u32(k ? 1u : 0u, red, &tq);
        const uint32_t s = carry_k + block_exclusive_scan_u32(k, red, &tk);
        if (c < n_clusters) offsets[c] = s;
        if (k && q < extents_cap) peak_extents[q] = atag_peak_extents{s, k};
        carry_q += tq;
        carry_k += tk;
    }
    if (threadIdx.x == 0) {
        d_counts[0] = carry_k;
        d_counts[1] = carry_q;
        d_counts[2] = (carry_k > corner_cap || carry_q > extents_cap) ? ATAG_DEVFLAG_QUAD_OVERFLOW : 0u;
    }
}

__global__ void __launch_bounds__(32 * PK_WARPS) k_peaks_sort(const atag_corner* __restrict__ found,
                                                    const atag_cluster_extents* __restrict__ ext,
                                                    uint32_t n_clusters, const uint32_t* __restrict__ counts,
                                                    const uint32_t* __restrict__ offsets,
                                                    atag_corner* __restrict__ out, uint32_t corner_cap,
                                                    uint32_t* __restrict__ d_counts) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    extern __shared__ unsigned long long pk_keys[];
    __shared__ uint32_t s_n, s_large[PK_WARPS];
    static_assert(PK_WARPS * PK_WARP <= PK_SORT_CAP, "a warp's share of the keys");
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // key: error descending (complemented order key), then position
    auto key_of = [](float err, uint32_t i) { return ((unsigned long long)(~float_order_key(err)) << 32) | i; };
    for (uint32_t c0 = blockIdx.x; c0 < n_clusters; c0 += gridDim.x * PK_WARPS) {
        const uint32_t cw = c0 + gridDim.x * wid, kw = cw < n_clusters ? counts[cw] : 0u;
        uint32_t large = INVALID;
        if (kw) {
            const atag_cluster_extents e = ext[cw];
            if (e.count > PK_WARP) {
                large = cw;
            } else {
                // keys listed by ballots, each corner put at its key's rank
                unsigned long long* keys = pk_keys + wid * PK_WARP;
                uint32_t n = 0;
#pragma unroll PK_UNROLL
                for (uint32_t i0 = 0; i0 < e.count; i0 += 32) {
                    const uint32_t i = i0 + lane;
                    const float err = i < e.count ? found[(size_t)e.start + i].error : 0.0f;
                    const unsigned m = __ballot_sync(FULL, err != 0.0f);
                    if (err != 0.0f) keys[n + (uint32_t)__popc(m & ((1u << lane) - 1u))] = key_of(err, i);
                    n += (uint32_t)__popc(m);
                }
                __syncwarp();
                const uint32_t off = offsets[cw];
                for (uint32_t j = lane; j < n; j += 32) {
                    const unsigned long long key = keys[j];
                    uint32_t r = 0;
                    for (uint32_t q = 0; q < n; q++) r += keys[q] < key ? 1u : 0u;
                    if (off + r < corner_cap) out[off + r] = found[(size_t)e.start + (uint32_t)key];
                }
            }
        }
        if (lane == 0) s_large[wid] = large;
        __syncthreads();
        for (unsigned m = __ballot_sync(FULL, s_large[lane] != INVALID); m; m &= m - 1) {
            const uint32_t c = s_large[__ffs(m) - 1], k = counts[c];
            if (k > PK_SORT_CAP) {
                // more corners than a cluster of valid points can have
                if (threadIdx.x == 0) atomicOr(d_counts + 2, ATAG_DEVFLAG_SORT_OVERFLOW);
                continue;
            }
            const atag_cluster_extents e = ext[c];
            if (threadIdx.x == 0) s_n = 0;
            __syncthreads();
            for (uint32_t i0 = threadIdx.x; i0 < e.count; i0 += PK_UNROLL * blockDim.x) {
                float err[PK_UNROLL];
#pragma unroll
                for (int u = 0; u < PK_UNROLL; u++) {
                    const uint32_t i = i0 + u * blockDim.x;
                    err[u] = i < e.count ? found[(size_t)e.start + i].error : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < PK_UNROLL; u++) {
                    if (err[u] == 0.0f) continue;
                    const uint32_t at = atomicAdd(&s_n, 1u);
                    if (at < k) pk_keys[at] = key_of(err[u], i0 + u * blockDim.x);
                }
            }
            __syncthreads();
            bitonic_sort_u64(pk_keys, k);
            const uint32_t off = offsets[c];
            for (uint32_t j = threadIdx.x; j < k; j += blockDim.x)
                if (off + j < corner_cap) out[off + j] = found[(size_t)e.start + (uint32_t)pk_keys[j]];
            __syncthreads();
        }
        __syncthreads();
    }
}

}  // namespace atag
