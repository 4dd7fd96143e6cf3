// k_quads.cu — drop-in kernels for the reference's fit_lines and do_indexing,
// and the corner intersection of process_fitted_quads moved to the device.
#include <cooperative_groups.h>

#include "atag_kernels.cuh"
#include "atag_quads.cuh"

namespace atag {

// ---------------------------------------------------------------------------
// fit_lines (fit_quad.cpp:153-375), restated warp-per-work-group: 32 lanes
// hold points x = 24 g - 3 ... 24 g + 28 and lanes 4..27 decide corners.
// The work-group barriers become __syncwarp.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_fit_lines_windowed(const atag_line_fit_point* __restrict__ points,
                                                            const uint16_t* __restrict__ cidx,
                                                            const atag_cluster_extents* __restrict__ extents,
                                                            size_t n, atag_corner* __restrict__ found) {
    constexpr int WG = 32, PPE = 3, EO = 4;
    __shared__ uint16_t s_ci[4][WG];
    __shared__ atag_cluster_extents s_ce[4][WG];
    __shared__ float s_es[4][WG], s_ed[4][WG], s_fs[4][WG], s_fd[4][WG];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t group = (size_t)blockIdx.x * 4 + wid;
    const size_t groups = (n + 23) / 24;
    if (group >= groups) return;
    const long long x = (long long)group * (WG - 2 * EO) + lane - PPE;
    const long long xc = x < 0 ? 0 : (x > (long long)n - 1 ? (long long)n - 1 : x);
    const uint16_t ci = cidx[xc];
    const atag_cluster_extents ce = extents[ci];
    s_ci[wid][lane] = ci;
    s_ce[wid][lane] = ce;
    __syncwarp();
    s_es[wid][lane] = window_error(points, ce.start, ce.count, x);
    int their = lane;
    if (lane >= EO && s_ci[wid][lane - EO] != ci) their = lane - EO;
    if (lane < WG - EO && s_ci[wid][lane + EO] != ci) their = lane + EO;
    if (their != lane) {
        atag_cluster_extents te = s_ce[wid][their];
        s_ed[wid][lane] = window_error(points, te.start, te.count, x);
    } else {
        s_ed[wid][lane] = __int_as_float(0x7fc00000);
    }
    __syncwarp();
    if (lane >= PPE && lane < WG - PPE) {
        float acc = 0.0f, dacc = 0.0f;
#pragma unroll
        for (int i = 0; i < 7; i++) {
            int t = lane + i - PPE;
            float f = filter_tap(i);
            if (s_ci[wid][t] == ci) {
                acc = __fadd_rn(acc, __fmul_rn(s_es[wid][t], f));
                dacc = __fadd_rn(dacc, __fmul_rn(s_ed[wid][t], f));
            } else {
                dacc = __fadd_rn(dacc, __fmul_rn(s_es[wid][t], f));
                acc = __fadd_rn(acc, __fmul_rn(s_ed[wid][t], f));
            }
        }
        s_fs[wid][lane] = acc;
        s_fd[wid][lane] = dacc;
    }
    __syncwarp();
    if (lane < EO || lane >= WG - EO) return;
    if (x < 0 || x >= (long long)n) return;
    const float cur = s_fs[wid][lane];
    const bool gb = cur > (s_ci[wid][lane - 1] == ci ? s_fs : s_fd)[wid][lane - 1];
    const bool ga = cur > (s_ci[wid][lane + 1] == ci ? s_fs : s_fd)[wid][lane + 1];
    if (gb && ga) {
        atag_corner c;
        c.line_fit_point_index = (uint32_t)(x - ce.start);
        c.cluster_index = ci;
        c.error = cur;
        found[x] = c;
    }
}

// ---------------------------------------------------------------------------
// do_indexing (fit_quad.cpp:392-535): one warp per peak extent;
// cluster_extents is indexed by the extent's position, exactly as the
// reference does.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_do_indexing(const atag_peak_extents* __restrict__ extents, size_t count,
                                                     const atag_corner* __restrict__ corners,
                                                     const atag_line_fit_point* __restrict__ points,
                                                     const atag_cluster_extents* __restrict__ cluster_extents,
                                                     float max_mse, float cos_critical,
                                                     atag_fitted_quad* __restrict__ fitted) {
    __shared__ SegmentTable T[4];  // one per warp
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (size_t q = blockIdx.x + (size_t)gridDim.x * wid; q < count; q += (size_t)gridDim.x * 4) {
        const atag_peak_extents pe = extents[q];
        const atag_cluster_extents ce = cluster_extents[q];
        // fewer than four corners make no quad and are not read
        const uint32_t used = pe.count < 4u ? 0u : min(pe.count, 10u);
        const uint32_t idx = lane < used ? corners[pe.start + lane].line_fit_point_index : 0u;
        QuadSide side;
        index_one_cluster(pe.count, idx, points + ce.start, ce.count, max_mse, cos_critical, T[wid], fitted + q, side);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// process_fitted_quads (main.cpp:1035-1162) up to tag decoding, on one cluster
// of PQ_CTAS thread blocks: eight lanes per quad, and an ordered compaction
// that reads the other blocks' counts from their shared memory.  Bound by the
// FP64 chain of a quad (lines, corners, lengths, angles), which one block's SM
// runs for few quads at a time: 65 quads took 38 us on one block with a thread
// each, 28 with eight lanes each, 11 on the cluster.
// ---------------------------------------------------------------------------
__global__ void __cluster_dims__(PQ_CTAS, 1, 1) __launch_bounds__(128)
    k_process_quads(const atag_fitted_quad* __restrict__ fitted, size_t count, PipelineParams p,
                    atag_quad_corners* __restrict__ out, size_t cap, uint32_t* __restrict__ count_out) {
    constexpr uint32_t PER = 16;  // quads of a block and round
    constexpr unsigned FULL = 0xFFFFFFFFu;
    namespace cg = cooperative_groups;
    cg::cluster_group blocks = cg::this_cluster();
    __shared__ uint32_t ok_mask[2];  // by round parity: which of the block's quads stand
    const uint32_t g = threadIdx.x & 7, local = threadIdx.x >> 3, rank = blocks.block_rank(), lane = threadIdx.x & 31;
    uint32_t base = 0, round = 0;
    for (size_t c0 = 0; c0 < count; c0 += PQ_CTAS * PER, round ^= 1) {
        const size_t i = c0 + rank * PER + local;
        float line[4] = {0.0f, 0.0f, 0.0f, 0.0f}, cx, cy, e, mse;
        bool any = false;
        if (i < count) {
            const atag_fitted_quad& fq = fitted[i];
            any = (fq.indices[0] | fq.indices[1] | fq.indices[2] | fq.indices[3]) != 0;
            if (any && g < 4) fit_line(load_moment(&fq.moments[g]), fq.num_in_moments[g], line, &e, &mse);
        }
        const bool ok = quad_corners8(line, p, cx, cy) && any;
        if (threadIdx.x == 0) ok_mask[round] = 0;
        __syncthreads();
        if (ok && g == 0) atomicOr(&ok_mask[round], 1u << local);
        // the masks of all blocks; this round's are rewritten two rounds on,
        // after every block has passed the next round's barrier
        blocks.sync();
        const uint32_t mask = lane < PQ_CTAS ? *blocks.map_shared_rank(&ok_mask[round], lane) : 0u;
        const uint32_t n = (uint32_t)__popc(mask);
        const uint32_t before = __reduce_add_sync(FULL, lane < rank ? n : 0u), total = __reduce_add_sync(FULL, n);
        const uint32_t mine = __shfl_sync(FULL, mask, (int)rank);
        const size_t at = (size_t)base + before + (uint32_t)__popc(mine & ((1u << local) - 1u));
        if (ok && at < cap) {
            atag_quad_corners& qc = out[at];
            if (g < 4) {
                qc.corners[g][0] = cx;
                qc.corners[g][1] = cy;
            } else if (g == 4) {
                qc.reversed_border = (uint8_t)p.reversed_border;
                qc.pad_[0] = qc.pad_[1] = qc.pad_[2] = 0;
                qc.blob_index = (uint32_t)i;
            }
        }
        base += total;
    }
    if (rank == 0 && threadIdx.x == 0) *count_out = base < cap ? base : (uint32_t)cap;
    blocks.sync();  // no block leaves while another may read its masks
}

}  // namespace atag
