// atag_quads.cuh — the combination search of do_indexing and the corner
// intersection of process_fitted_quads, shared by the drop-in kernels and
// the fused per-cluster pipeline.
#pragma once

#include "atag_kernels.cuh"

namespace atag {

// The 210 sets of 4 of 10 peak ranks as bit masks, numbered as the reference
// numbers its combinations (combinadics.h:36-53).
struct CombinationMasks {
    uint16_t mask[210];
};
constexpr CombinationMasks combination_masks() {
    CombinationMasks M{};
    const uint32_t c4[10] = {0, 0, 0, 0, 1, 5, 15, 35, 70, 126};
    const uint32_t c3[10] = {0, 0, 0, 1, 4, 10, 20, 35, 56, 84};
    const uint32_t c2[10] = {0, 0, 1, 3, 6, 10, 15, 21, 28, 36};
    for (uint32_t n = 0; n < 210; n++) {
        uint32_t num = n, a = 9, b = 9, c = 9;
        while (a > 0 && c4[a] > num) a--;
        num -= c4[a];
        while (b > 0 && c3[b] > num) b--;
        num -= c3[b];
        while (c > 0 && c2[c] > num) c--;
        num -= c2[c];
        M.mask[n] = (uint16_t)((1u << a) | (1u << b) | (1u << c) | (1u << num));
    }
    return M;
}
static __device__ const CombinationMasks COMBINATIONS = combination_masks();

// do_indexing for one peak cluster on one warp.  The 210 combinations of
// up to 10 peaks only ever fit the 90 ordered segments between two of those
// peaks, so each segment is fitted once (the same get_moment/fit_line
// arithmetic as the per-combination form, hence the same bits) and every
// combination sums four table entries in the reference's order
// (fit_quad.cpp:404-503).  The peaks are put in line-fit index order first
// (sort_4, fit_quad.cpp:377-389,437), so a combination is four ascending
// positions, and the 21 prefix sums all segments come from are read once.
// The choice is the reference's: the lowest total error, then the smallest
// combination number within 0.1 of it (fit_quad.cpp:501-519).  Lane i < 4
// writes side i of *out and keeps it in `side`; every lane returns the chosen
// number, or -1.
struct SegmentTable {
    float err[10][10], mse[10][10], lp[10][10][4];  // by position; lp for a < b
    Moment at[10], before[10], last;                // prefix sums at and before the peaks, and the cluster's last
    uint32_t idx[10];                               // line_fit_point_index by position
};

struct QuadSide {
    Moment m;
    uint16_t points, index;  // as atag_fitted_quad stores them
};

// get_moment (fit_quad.cpp:15-35) from position a to position b
__device__ __forceinline__ Moment segment_moment(const SegmentTable& T, uint32_t a, uint32_t b, uint32_t ccount,
                                                 unsigned long long* total) {
    const unsigned long long i0 = T.idx[a], i1 = T.idx[b];
    *total = 0;
    if (i0 == i1) return Moment{0, 0, 0, 0, 0, 0};
    if (i0 < i1) {
        *total = i1 - i0 + 1;
        return m_sub(T.at[b], T.before[a]);
    }
    *total = (unsigned long long)ccount - i0 + i1 + 1;
    return m_add(m_sub(T.last, T.before[a]), T.at[b]);
}

// The four ascending positions of a set of ranks; order: rank r's position in
// bits 4 r .. 4 r + 3.
__device__ __forceinline__ void positions_of(uint32_t ranks, unsigned long long order, uint32_t (&p)[4]) {
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        m |= 1u << ((uint32_t)(order >> (4 * (__ffs(ranks) - 1))) & 15u);
        ranks &= ranks - 1;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        p[j] = __ffs(m) - 1;
        m &= m - 1;
    }
}

// `corner_index`: rank r's line_fit_point_index on lane r.
__device__ __forceinline__ int index_one_cluster(uint32_t count, uint32_t corner_index,
                                                 const atag_line_fit_point* __restrict__ cpts, uint32_t ccount,
                                                 float max_mse, float cos_critical, SegmentTable& T,
                                                 atag_fitted_quad* out, QuadSide& side) {
    constexpr int PER = (210 + 31) / 32;  // combinations per lane
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t m = count < 10u ? count : 10u;
    const uint32_t ncomb = n_choose_4(m);
    if (ncomb == 0) return -1;
    // rank -> position (ties, which only a caller's corners can have, by rank)
    uint32_t mypos = 0;
    for (uint32_t j = 0; j < m; j++) {
        const uint32_t o = __shfl_sync(FULL, corner_index, (int)j);
        mypos += (o < corner_index || (o == corner_index && j < lane)) ? 1u : 0u;
    }
    unsigned long long order = 0;
    for (uint32_t j = 0; j < m; j++) order |= (unsigned long long)__shfl_sync(FULL, mypos, (int)j) << (4 * j);
    if (lane < m) {
        T.idx[mypos] = corner_index;
        T.at[mypos] = load_moment(cpts + corner_index);
        T.before[mypos] = corner_index > 0 ? load_moment(cpts + corner_index - 1) : Moment{0, 0, 0, 0, 0, 0};
    }
    if (lane == 31 && ccount > 0) T.last = load_moment(cpts + (ccount - 1));
    __syncwarp();
    // forward segments (with line parameters) first, then backward ones
    const uint32_t half = m * (m - 1) / 2;
    for (uint32_t s = lane; s < 2 * half; s += 32) {
        // s mod half -> the pair lo < hi
        const bool back = s >= half;
        uint32_t r = back ? s - half : s, lo = 0, n = m - 1;
        while (r >= n) {
            r -= n;
            n--;
            lo++;
        }
        const uint32_t hi = lo + 1 + r, a = back ? hi : lo, b = back ? lo : hi;
        unsigned long long nim;
        const Moment mo = segment_moment(T, a, b, ccount, &nim);
        float e, mse;
        fit_line(mo, nim, back ? nullptr : T.lp[a][b], &e, &mse);
        T.err[a][b] = e;
        T.mse[a][b] = mse;
    }
    __syncwarp();
    float errs[PER];
    uint32_t low_key = float_order_key(__int_as_float(0x7f800000));
#pragma unroll
    for (int t = 0; t < PER; t++) {
        const uint32_t n = lane + 32u * t;
        float err = __int_as_float(0x7f800000);
        if (n < ncomb) {
            uint32_t p[4];
            positions_of(COMBINATIONS.mask[n], order, p);
            float total = 0.0f;
            bool valid = true;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t a = p[j], b = p[(j + 1) & 3];
                valid &= T.mse[a][b] <= max_mse;
                total = __fadd_rn(total, T.err[a][b]);
            }
            const float* p01 = T.lp[p[0]][p[1]];
            const float* p12 = T.lp[p[1]][p[2]];
            const float dot = __fadd_rn(__fmul_rn(p01[2], p12[2]), __fmul_rn(p01[3], p12[3]));
            valid &= fabsf(dot) <= cos_critical;
            if (valid && !isnan(total)) err = total;
        }
        errs[t] = err;
        low_key = min(low_key, float_order_key(err));
    }
    low_key = __reduce_min_sync(FULL, low_key);
    const float lowest = float_from_order_key(low_key);
    if (isinf(lowest) && lowest > 0) return -1;
    uint32_t first = 0xFFFFFFFFu;
#pragma unroll
    for (int t = PER - 1; t >= 0; t--)  // (double)(err - lowest) < 0.1, in float
        if (__fsub_rn(errs[t], lowest) < 0x1.99999ap-4f) first = lane + 32u * t;
    const uint32_t chosen = __reduce_min_sync(FULL, first);
    if (chosen == 0xFFFFFFFFu) return -1;
    uint32_t p[4];
    positions_of(COMBINATIONS.mask[chosen], order, p);
    if (lane < 4) {
        const uint32_t a = lane == 0 ? p[0] : (lane == 1 ? p[1] : (lane == 2 ? p[2] : p[3]));
        const uint32_t b = lane == 0 ? p[1] : (lane == 1 ? p[2] : (lane == 2 ? p[3] : p[0]));
        unsigned long long nim;
        side.m = segment_moment(T, a, b, ccount, &nim);
        side.points = (uint16_t)nim;
        side.index = (uint16_t)T.idx[a];
        store_moment(&out->moments[lane], side.m);
        out->num_in_moments[lane] = side.points;
        out->indices[lane] = side.index;
    }
    return (int)chosen;
}

// process_fitted_quads body (main.cpp:1042-1161) for one FittedQuad on a group
// of 8 lanes: lane i < 4 of the group passes line i (centroid, normal) of the
// quad's sides and gets corner i in (cx, cy).  Corners, side lengths and angles
// are computed one per lane; on one thread their FP64 divisions and square
// roots were the longest serial chain of a lone frame's last stages.  Every
// lane of the group returns whether the quad stands.
__device__ __forceinline__ bool quad_corners8(const float (&line)[4], const PipelineParams& p, float& cx, float& cy) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int g = threadIdx.x & 7, base = (threadIdx.x & 31) & ~7;
    auto of = [&](float v, int i) { return __shfl_sync(FULL, v, base + i); };
    bool ok = true;
    {
        const int j = (g + 1) & 3;
        const float l0 = of(line[0], j), l1 = of(line[1], j), l2 = of(line[2], j), l3 = of(line[3], j);
        const double A00 = (double)line[3], A01 = -(double)l3, A10 = -(double)line[2], A11 = (double)l2;
        const double B0 = (double)__fadd_rn(-line[0], l0), B1 = (double)__fadd_rn(-line[1], l1);
        const double det = __dsub_rn(__dmul_rn(A00, A11), __dmul_rn(A10, A01));
        const double W00 = __ddiv_rn(A11, det), W01 = __ddiv_rn(-A01, det);
        if (g < 4 && fabs(det) < 0.001) ok = false;
        const double L0 = __dadd_rn(__dmul_rn(W00, B0), __dmul_rn(W01, B1));
        cx = __double2float_rn(__dadd_rn((double)line[0], __dmul_rn(L0, A00)));
        cy = __double2float_rn(__dadd_rn((double)line[1], __dmul_rn(L0, A10)));
    }
    {
        // the triangles 0 1 2 and 2 3 0: lengths 01, 12, 20 on lanes 0-2 and
        // 23, 30, 02 on lanes 3-5
        const int from = g < 3 ? g : (g < 5 ? g - 1 : 0), to = g < 2 ? g + 1 : (g == 2 ? 0 : (g == 3 ? 3 : (g == 4 ? 0 : 2)));
        const float fx = of(cx, from), fy = of(cy, from), tx = of(cx, to), ty = of(cy, to);
        const float len = hypot_f(__fsub_rn(tx, fx), __fsub_rn(ty, fy));
        float area = 0.0f;
#pragma unroll
        for (int k = 0; k < 6; k += 3) {
            const float a = of(len, k), b = of(len, k + 1), c = of(len, k + 2);
            const float pp = __fdiv_rn(__fadd_rn(__fadd_rn(a, b), c), 2.0f);
            float t = __fmul_rn(pp, __fsub_rn(pp, a));
            t = __fmul_rn(t, __fsub_rn(pp, b));
            t = __fmul_rn(t, __fsub_rn(pp, c));
            area = __fadd_rn(area, __fsqrt_rn(t));
        }
        if ((double)area < p.min_area) ok = false;
    }
    {
        const int i1 = (g + 1) & 3, i2 = (g + 2) & 3;
        const float x1 = of(cx, i1), y1 = of(cy, i1), x2 = of(cx, i2), y2 = of(cy, i2);
        const float dx1 = __fsub_rn(x1, cx), dy1 = __fsub_rn(y1, cy), dx2 = __fsub_rn(x2, x1), dy2 = __fsub_rn(y2, y1);
        const float num = __fadd_rn(__fmul_rn(dx1, dx2), __fmul_rn(dy1, dy2));
        const float s1 = __fadd_rn(__fmul_rn(dx1, dx1), __fmul_rn(dy1, dy1));
        const float s2 = __fadd_rn(__fmul_rn(dx2, dx2), __fmul_rn(dy2, dy2));
        const float cosd = __fdiv_rn(num, __fsqrt_rn(__fmul_rn(s1, s2)));
        if (g < 4 && (fabs((double)cosd) > p.cos_critical_d || __fmul_rn(dx1, dy2) < __fmul_rn(dy1, dx2))) ok = false;
    }
    const unsigned bad = __ballot_sync(FULL, !ok);
    return ((bad >> base) & 0xFFu) == 0u;
}

}  // namespace atag
