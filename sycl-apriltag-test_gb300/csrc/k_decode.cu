// k_decode.cu — reading tags: each quad's bit grid matched against a code
// family that the caller describes the way the AprilTag library describes
// its families (bits at per-bit cell coordinates).
//
// The reference hands each quad to the AprilTag library's quad_decode_task
// with tag36h11 and the detector defaults plus quad_decimate = 1
// (src/quad_decoding.cpp:46-75).  The library is not in the reference tree;
// this kernel follows its published decoding algorithm (Olson 2011; Wang &
// Olson 2016; Krogius, Haggenmiller & Olson 2019) with its documented
// defaults (edge refinement on, decode sharpening 0.25):
//   1. edge refinement: per edge, max(16, |edge| / 8) points along it; at
//      each, quarter-pixel positions -r .. r along the outward normal
//      (r = quad_decimate + 1), the grey step between the pixels one pixel
//      either side (truncated coordinates - 0.5) weighted by its square
//      where it rises outward, gives the edge's offset; a line through the
//      offset points; corners at the intersections of adjacent lines
//      (kept when the 2x2 determinant is at most 1e-3);
//   2. homography of the tag square [-1, 1]^2 onto the quad (closed form,
//      Heckbert 1989);
//   3. grey models: least-squares planes over the white ring just outside
//      the black border and over the border, nearest-pixel samples, one per
//      cell along each side; rejected when white minus black at the centre
//      is below min_contrast;
//   4. each bit: bilinear sample at its cell centre (pixel centres at
//      +0.5) minus the models' mean, on a total_width^2 grid, sharpened by
//      decode_sharpening times the 4-neighbour Laplacian; bit = value > 0;
//   5. decision margin = min(mean value of the white bits, mean magnitude
//      of the black bits), counts starting at 1;
//   6. the code and quarter turn with the smallest Hamming distance
//      (ties: fewer turns, lower index), accepted at most max_hamming with a
//      non-negative decision margin.
// Beyond the library: a quad wound the other way is read with corners 0, 3,
// 2, 1 (flagged); the refinement's normal points outward by the quad's
// signed area; a projection behind the camera (z <= 0) or a corner that is not
// finite marks the quad degenerate.
//
// One warp per quad, FP64 throughout: lanes take the refinement's points,
// the grey-model samples, the bits and the codes.  FP64 issues at 2 lanes per
// clock and SM on this GPU (a warp instruction holds a scheduler's share of
// the pipe for about 64 clocks, whatever its active lanes), so the kernel is
// bound by its FP64 instruction count and is arranged around it:
//   * the four edges are refined side by side, eight lanes each, so edge set-up,
//     line fit and corner intersection are issued once, not four times, and
//     the sums reduce over eight lanes;
//   * positions along an edge's normal step in exact integers (Q50), but for
//     those on pixel borders; each grey value is fetched once (the step at n
//     pairs offsets n + 1 and n - 1), and weights and grey-model sums are
//     integers, exact;
//   * the edge's direction comes from square roots, not atan2/sin/cos;
//   * both grey models are solved at once, on even and odd lanes.
// 4,096 quads against 587 codes: 4,072 FP64 warp instructions per quad and
// 1,178 us before; 615 and 229 us now (597 and 219 without the FP64 positions
// on pixel borders and the quotients and cell centres of `project`).
#include <vector>

#include "atag_edge_samples.cuh"
#include "atag_internal.h"
#include "atag_kernels.cuh"

namespace atag {
namespace {

constexpr int DECODE_WARPS = 4;
constexpr int MAX_TW = 16;  // total_width limit: the value grid lives in shared memory
// Cells -1 .. width_at_border (the white ring's) and those of the bits, which
// start at (width_at_border - total_width) / 2 >= -6: bit cells are int8, so
// widths are at most 2 * 127 + MAX_TW.
constexpr int CELL_BASE = 8, MAX_CELLS = CELL_BASE + 2 * 127 + MAX_TW + 2;

struct FamilyDesc {
    int8_t bit_x[64], bit_y[64];
    uint8_t perm[64];  // one quarter turn: bit i takes bit perm[i]
    int nbits, width_at_border, total_width, reversed_border;
    uint32_t n_codes, max_hamming;
};

struct DecodeParams {
    double sharpening, min_contrast;
    int refine, quad_decimate;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// unit square -> quad, bottom-right element 1
struct Homography {
    double a, b, c, d, e, f, g, h;
};

__device__ __forceinline__ bool homography_ok(const double* px, const double* py, double* den) {
    const double dx1 = px[1] - px[2], dx2 = px[3] - px[2], dy1 = py[1] - py[2], dy2 = py[3] - py[2];
    *den = dx1 * dy2 - dx2 * dy1;
    const double ref = fabs(dx1) + fabs(dx2) + fabs(dy1) + fabs(dy2);
    return fabs(*den) > 1e-12 * ref * ref;
}
__device__ __forceinline__ Homography make_homography(const double* px, const double* py, double den) {
    Homography H;
    const double sx = px[0] - px[1] + px[2] - px[3], sy = py[0] - py[1] + py[2] - py[3];
    const double dx1 = px[1] - px[2], dx2 = px[3] - px[2], dy1 = py[1] - py[2], dy2 = py[3] - py[2];
    H.g = (sx * dy2 - dx2 * sy) / den;
    H.h = (dx1 * sy - sx * dy1) / den;
    H.a = px[1] - px[0] + H.g * px[1];
    H.b = px[3] - px[0] + H.h * px[3];
    H.c = px[0];
    H.d = py[1] - py[0] + H.g * py[1];
    H.e = py[3] - py[0] + H.h * py[3];
    H.f = py[0];
    return H;
}

// unit-square coordinates -> pixel; false behind the camera
__device__ __forceinline__ bool project(const Homography& H, double u, double v, double* x, double* y) {
    const double z = H.g * u + H.h * v + 1.0;
    if (!(z > 0.0)) return false;
    *x = (H.a * u + H.b * v + H.c) / z;
    *y = (H.d * u + H.e * v + H.f) / z;
    return true;
}

__device__ __forceinline__ double det3(double a00, double a01, double a02, double a10, double a11, double a12,
                                       double a20, double a21, double a22) {
    return a00 * (a11 * a22 - a12 * a21) - a01 * (a10 * a22 - a12 * a20) + a02 * (a10 * a21 - a11 * a20);
}

// Least-squares plane of the grey values over integer coordinates (a, b) =
// width_at_border * (tx, ty), from its exact integer sums a^2, ab, a, b^2, b,
// n, av, bv, v; min_det = 1e-12 in tag coordinates.
struct Plane {
    double c0, c1, c2;
    bool ok;
};
__device__ __forceinline__ Plane solve_plane(const int* s, double min_det) {
    const double A00 = s[0], A01 = s[1], A02 = s[2], A11 = s[3], A12 = s[4], A22 = s[5];
    const double B0 = s[6], B1 = s[7], B2 = s[8];
    Plane P{0.0, 0.0, 0.0, false};
    const double d = det3(A00, A01, A02, A01, A11, A12, A02, A12, A22);
    P.ok = s[5] >= 3 && fabs(d) > min_det;
    if (!P.ok) return P;
    P.c0 = det3(B0, A01, A02, B1, A11, A12, B2, A12, A22) / d;
    P.c1 = det3(A00, B0, A02, A01, B1, A12, A02, B2, A22) / d;
    P.c2 = det3(A00, A01, B0, A01, A11, B1, A02, A12, B2) / d;
    return P;
}

// C's conversion of a double to int (toward zero), as a double-range test
__device__ __forceinline__ bool trunc_in(double v, int n, int* out) {
    const double t = trunc(v);
    if (!(t >= 0.0 && t < (double)n)) return false;
    *out = (int)t;
    return true;
}

// Grey values along one refinement point's normal: offset k quarter pixels,
// the pixel at the truncated coordinate - 0.5; -1 outside the image.  Within
// 4,000 px of the origin positions are Q50 integers: an FP64 point from 4 px
// on converts exactly, and steps without rounding error.  A coordinate within
// 2^-32 px of a pixel's border, where the FP64 sum's rounding (below 2^-40)
// may fall on the other side of it, is taken from that sum, as beyond 4,000 px:
// quads along the axes with corners on whole pixels put many points there.
struct NormalWalk {
    const uint8_t* __restrict__ img;
    int w, h;
    size_t pitch;
    bool fixed;
    long long X, Y, NX, NY;  // Q50 position - 0.5, Q52 normal
    double x0, y0, nx, ny;
    __device__ __forceinline__ static bool at_border(long long v) { return (uint32_t)(v >> 18) + 1u <= 1u; }
    __device__ __forceinline__ int at(int k) const {
        int ix, iy;
        // k / 4 * n in Q50: k * Q52 >> 4
        const long long x = X + ((k * NX) >> 4), y = Y + ((k * NY) >> 4);
        if (fixed && !at_border(x) && !at_border(y)) {
            // truncation toward zero takes (-1, 0) to 0
            constexpr long long ONE = 1ll << 50;
            if (x <= -ONE || y <= -ONE) return -1;
            ix = x < 0 ? 0 : (int)(x >> 50);
            iy = y < 0 ? 0 : (int)(y >> 50);
            if (ix >= w || iy >= h) return -1;
        } else {
            const double n = 0.25 * k;
            if (!trunc_in(x0 + n * nx - 0.5, w, &ix) || !trunc_in(y0 + n * ny - 0.5, h, &iy)) return -1;
        }
        return img[(size_t)iy * pitch + ix];
    }
};

// Step 1 on the quad's warp: lanes 8 e .. 8 e + 7 take edge e's points.
__device__ void refine_edges(const uint8_t* __restrict__ img, int w, int h, size_t pitch, double* px, double* py,
                             bool reversed, int quad_decimate) {
    const int lane = threadIdx.x & 31, e = lane >> 3, sub = lane & 7;
    // this lane's edge: corner e -> corner e + 1
    const double ax = e == 0 ? px[0] : e == 1 ? px[1] : e == 2 ? px[2] : px[3];
    const double ay = e == 0 ? py[0] : e == 1 ? py[1] : e == 2 ? py[2] : py[3];
    const double bx = e == 0 ? px[1] : e == 1 ? px[2] : e == 2 ? px[3] : px[0];
    const double by = e == 0 ? py[1] : e == 1 ? py[2] : e == 2 ? py[3] : py[0];
    double nx = by - ay, ny = -(bx - ax);
    const double mag = sqrt(nx * nx + ny * ny);
    nx /= mag;
    ny /= mag;
    if (reversed) {
        nx = -nx;
        ny = -ny;
    }
    const int nsamples = edge_sample_count(mag);
    SampleRange S{0, nsamples};
    if (__any_sync(0xFFFFFFFFu, nsamples > EDGE_SAMPLES_WHOLE))
        S = edge_sample_range(ax, ay, bx, by, nsamples, quad_decimate + 2, w, h);
    const int r4 = 4 * (quad_decimate + 1);  // search range in quarter pixels
    // FP64 positions where a corner is far out or two coincide (warp-uniform)
    constexpr double FAR = 4000.0;
    NormalWalk W{img, w, h, pitch, false, 0, 0, 0, 0, 0.0, 0.0, nx, ny};
    W.fixed = __all_sync(0xFFFFFFFFu, fabs(ax) < FAR && fabs(ay) < FAR && mag > 0.0);
    if (W.fixed) {
        W.NX = __double2ll_rn(nx * 0x1p52);
        W.NY = __double2ll_rn(ny * 0x1p52);
    }
    // sums about the edge's midpoint
    const double mx = 0.5 * (ax + bx), my = 0.5 * (ay + by);
    double m[5] = {0, 0, 0, 0, 0};  // x, y, xx, xy, yy
    int count = 0;
    for (int s = S.lo + sub; s < S.hi; s += 8) {
        const double alpha = (1.0 + s) / (nsamples + 1);
        W.x0 = alpha * ax + (1.0 - alpha) * bx;
        W.y0 = alpha * ay + (1.0 - alpha) * by;
        if (W.fixed) {
            W.X = __double2ll_rn((W.x0 - 0.5) * 0x1p50);
            W.Y = __double2ll_rn((W.y0 - 0.5) * 0x1p50);
        }
        // the step at position n quarter pixels from -r4 to r4 pairs offsets
        // n + 4 and n - 4: each offset is fetched once, 8 kept
        int ring[8];
#pragma unroll
        for (int u = 0; u < 8; u++) ring[u] = W.at(u - r4 - 4);
        int Mn = 0, Mc = 0;
        for (int k0 = -r4; k0 <= r4; k0 += 8)
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int n = k0 + u;
                if (n > r4) break;
                const int g2 = ring[u], g1 = W.at(n + 4);
                ring[u] = g1;
                const int d = g1 - g2;
                if (g1 < 0 || g2 < 0 || d < 0) continue;
                Mn += d * d * n;
                Mc += d * d;
            }
        if (Mc == 0) continue;
        const double n0 = 0.25 * (double)Mn / (double)Mc;
        const double dx = W.x0 - mx + n0 * nx, dy = W.y0 - my + n0 * ny;
        m[0] += dx;
        m[1] += dy;
        m[2] += dx * dx;
        m[3] += dx * dy;
        m[4] += dy * dy;
        count++;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 5; k++) m[k] += __shfl_xor_sync(0xFFFFFFFFu, m[k], o);
        count += __shfl_xor_sync(0xFFFFFFFFu, count, o);
    }
    // the line through the offset points: centroid and normal direction
    // (cos th, sin th), th = atan2(-2 Cxy, Cyy - Cxx) / 2, from the half-angle
    // vector (R + h, c), or (|c|, +-(R - h)) for h < 0
    const double inv = 1.0 / (double)max(count, 1);
    const double Ex = m[0] * inv, Ey = m[1] * inv;
    // products rounded before they are subtracted: one point's covariance is 0
    const double c = __dmul_rn(Ex, Ey) - m[3] * inv;
    const double hh = 0.5 * ((m[4] * inv - __dmul_rn(Ey, Ey)) - (m[2] * inv - __dmul_rn(Ex, Ex)));
    const double R = sqrt(hh * hh + c * c);
    double lc = hh >= 0.0 ? R + hh : fabs(c), ls = hh >= 0.0 ? c : copysign(R - hh, c);
    const double len = sqrt(lc * lc + ls * ls);
    lc = len == 0.0 ? 1.0 : lc / len;
    ls = len == 0.0 ? 0.0 : ls / len;
    const double lx = mx + Ex, ly = my + Ey;
    // corner e + 1: this edge's line with the next edge's
    const int nxt = (lane + 8) & 31;
    const double c2 = __shfl_sync(0xFFFFFFFFu, lc, nxt), s2 = __shfl_sync(0xFFFFFFFFu, ls, nxt);
    const double B0 = __shfl_sync(0xFFFFFFFFu, lx, nxt) - lx, B1 = __shfl_sync(0xFFFFFFFFu, ly, nxt) - ly;
    const int count2 = __shfl_sync(0xFFFFFFFFu, count, nxt);
    const double det = ls * c2 - lc * s2;
    double qx = bx, qy = by;
    if (count > 0 && count2 > 0 && fabs(det) > 0.001) {
        const double L0 = (c2 * B0 + s2 * B1) / det;
        qx = lx + L0 * ls;
        qy = ly - L0 * lc;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        px[(i + 1) & 3] = __shfl_sync(0xFFFFFFFFu, qx, 8 * i);
        py[(i + 1) & 3] = __shfl_sync(0xFFFFFFFFu, qy, 8 * i);
    }
}

// A code from its bits' ballots: bit i of the tag is code bit n - 1 - i.
__device__ __forceinline__ unsigned long long code_of(unsigned lo, unsigned hi, int n) {
    return __brevll((unsigned long long)hi << 32 | lo) >> (64 - n);
}
__device__ __forceinline__ unsigned long long rotate_code(unsigned long long c, const FamilyDesc& F) {
    const int lane = threadIdx.x & 31, n = F.nbits;
    const bool b0 = lane < n && ((c >> (n - 1 - F.perm[lane])) & 1ull);
    const bool b1 = lane + 32 < n && ((c >> (n - 1 - F.perm[min(lane + 32, 63)])) & 1ull);
    const unsigned lo = __ballot_sync(0xFFFFFFFFu, b0), hi = __ballot_sync(0xFFFFFFFFu, b1);
    return code_of(lo, hi, n);
}

__global__ void __launch_bounds__(32 * DECODE_WARPS) k_decode_quads(
    const uint8_t* __restrict__ img, int w, int h, size_t pitch, const uint8_t* __restrict__ quads, size_t stride,
    uint32_t n, const unsigned long long* __restrict__ codes, const __grid_constant__ FamilyDesc F,
    DecodeParams prm, atag_decoded* __restrict__ out) {
    __shared__ double s_vals[DECODE_WARPS][MAX_TW * MAX_TW];
    // unit-square coordinate of each cell's centre, by way of the tag coordinate
    // and its roundings: a quad along the axes puts many samples on the borders
    // between pixels, where the last bit chooses the pixel
    __shared__ double s_centre[MAX_CELLS];
    for (int i = threadIdx.x; i < CELL_BASE + max(F.width_at_border, F.total_width) + 2; i += blockDim.x) {
        const double t = 2.0 * (((double)(i - CELL_BASE) + 0.5) / F.width_at_border - 0.5);
        s_centre[i] = 0.5 * (t + 1.0);
    }
    __syncthreads();
    const double* centre = s_centre + CELL_BASE;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t q = blockIdx.x * DECODE_WARPS + wid;
    if (q >= n) return;  // warp-uniform
    double* vals = s_vals[wid];
    const float* cf = reinterpret_cast<const float*>(quads + (size_t)q * stride);
    double px[4], py[4];
    bool finite = true;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        finite &= isfinite(cf[2 * i]) && isfinite(cf[2 * i + 1]);
        px[i] = (double)cf[2 * i];
        py[i] = (double)cf[2 * i + 1];
    }
    atag_decoded R;
    memset(&R, 0, sizeof R);
    R.id = -1;
    R.hamming = 0xFFFFFFFFu;
    double area2 = 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++) area2 += px[i] * py[(i + 1) & 3] - px[(i + 1) & 3] * py[i];
    if (area2 < 0.0) {
        double t = px[1];
        px[1] = px[3];
        px[3] = t;
        t = py[1];
        py[1] = py[3];
        py[3] = t;
        R.status |= ATAG_DECODE_REORDERED;
    }
    auto finish = [&]() {
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                R.corners[i][0] = (float)px[i];
                R.corners[i][1] = (float)py[i];
            }
            out[q] = R;
        }
    };
    // With finite corners every projected coordinate below is finite (z is 1
    // plus bounded terms, so not denormal); homography_ok itself never reads
    // corner 0.
    double den;
    bool ok = finite && homography_ok(px, py, &den);
    if (ok && prm.refine) {
        refine_edges(img, w, h, pitch, px, py, F.reversed_border != 0, prm.quad_decimate);
        ok = homography_ok(px, py, &den);
    }
    if (!ok) {
        R.status |= ATAG_DECODE_DEGENERATE;
        finish();
        return;
    }
    const Homography H = make_homography(px, py, den);
    // 3. grey models: 8 sides x W samples, lanes over them; coordinates are
    // half cells, hx = 2 (x0 + i), so that tx = (hx - W) / W and the sums
    // over hx - W are integers
    const int Wb = F.width_at_border, T = F.total_width;
    int sums[2][9];  // black, white
#pragma unroll
    for (int k = 0; k < 9; k++) sums[0][k] = sums[1][k] = 0;
    bool behind = false;
    for (int k = lane; k < 8 * Wb; k += 32) {
        const int pat = k / Wb, i = k % Wb;
        // the eight sides in the order left out/in, right out/in, top out/in,
        // bottom out/in; the outer ones are white
        const bool white = (pat & 1) == 0, vertical = pat < 4;
        const int edge = (pat & 2) ? 2 * Wb + (white ? 1 : -1) : (white ? -1 : 1);
        const int hx = vertical ? edge : 2 * i + 1, hy = vertical ? 2 * i + 1 : edge;
        double x, y;
        if (!project(H, centre[hx >> 1], centre[hy >> 1], &x, &y)) {
            behind = true;
            continue;
        }
        // (-1, 0) truncates to 0; the conversion saturates and takes NaN to
        // INT_MIN, which the unsigned test rejects too
        const int ix = __double2int_rz(x), iy = __double2int_rz(y);
        if ((unsigned)ix >= (unsigned)w || (unsigned)iy >= (unsigned)h) continue;
        const int v = img[(size_t)iy * pitch + ix], ta = hx - Wb, tb = hy - Wb;
        const int t[9] = {ta * ta, ta * tb, ta, tb * tb, tb, 1, ta * v, tb * v, v};
#pragma unroll
        for (int j = 0; j < 9; j++) {
            sums[0][j] += white ? 0 : t[j];
            sums[1][j] += white ? t[j] : 0;
        }
    }
    if (__any_sync(0xFFFFFFFFu, behind)) {
        R.status |= ATAG_DECODE_DEGENERATE;
        finish();
        return;
    }
    // even lanes solve the black model, odd lanes the white one
    int mine[9];
#pragma unroll
    for (int j = 0; j < 9; j++) {
        const int b = __reduce_add_sync(0xFFFFFFFFu, sums[0][j]), wt = __reduce_add_sync(0xFFFFFFFFu, sums[1][j]);
        mine[j] = (lane & 1) ? wt : b;
    }
    const double W2 = (double)Wb * Wb;
    const Plane P = solve_plane(mine, 1e-12 * W2 * W2);
    if (!__all_sync(0xFFFFFFFFu, P.ok)) {
        R.status |= ATAG_DECODE_LOW_CONTRAST;
        finish();
        return;
    }
    const double black = __shfl_sync(0xFFFFFFFFu, P.c2, 0), white = __shfl_sync(0xFFFFFFFFu, P.c2, 1);
    R.white = (float)white;
    R.black = (float)black;
    const double contrast = F.reversed_border ? black - white : white - black;
    if (!(contrast >= prm.min_contrast)) {
        R.status |= ATAG_DECODE_LOW_CONTRAST;
        finish();
        return;
    }
    // the models' mean, which the bits are compared with
    const double t0 = 0.5 * (P.c0 + __shfl_xor_sync(0xFFFFFFFFu, P.c0, 1));
    const double t1 = 0.5 * (P.c1 + __shfl_xor_sync(0xFFFFFFFFu, P.c1, 1));
    const double t2 = 0.5 * (black + white);
    // 4. bit values on the total_width grid; lane i has bits i and i + 32
    const int m = (Wb - T) / 2, nb = F.nbits;
    for (int k = lane; k < T * T; k += 32) vals[k] = 0.0;
    __syncwarp();
    int cell[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int i = lane + 32 * j;
        if (i >= nb) continue;
        const int bx = F.bit_x[i], by = F.bit_y[i], hx = 2 * bx + 1, hy = 2 * by + 1;
        cell[j] = (by - m) * T + (bx - m);
        double x, y;
        if (!project(H, centre[bx], centre[by], &x, &y)) {
            behind = true;
            continue;
        }
        // bilinear, pixel centres at +0.5; outside the image the value stays 0
        x -= 0.5;
        y -= 0.5;
        const int x1 = __double2int_rd(x), y1 = __double2int_rd(y);
        if (x1 < 0 || y1 < 0 || x1 >= w || y1 >= h) continue;
        const double fx = x - (double)x1, fy = y - (double)y1;
        const int x2 = x1 + (fx > 0.0 ? 1 : 0), y2 = y1 + (fy > 0.0 ? 1 : 0);
        if (x2 >= w || y2 >= h) continue;
        const uint8_t *r1 = img + (size_t)y1 * pitch, *r2 = img + (size_t)y2 * pitch;
        const int v1 = r1[x1], v2 = r1[x2], v3 = r2[x1], v4 = r2[x2];
        const double top = (double)v1 + fx * (double)(v2 - v1), bottom = (double)v3 + fx * (double)(v4 - v3);
        vals[cell[j]] = top + fy * (bottom - top) - (t0 * (hx - Wb) + t1 * (hy - Wb) + t2);
    }
    if (__any_sync(0xFFFFFFFFu, behind)) {
        R.status |= ATAG_DECODE_DEGENERATE;
        finish();
        return;
    }
    __syncwarp();
    // sharpening, the bits and their scores
    double ws = 0.0, bs = 0.0;
    unsigned bal[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
        bool bit = false;
        if (lane + 32 * j < nb) {
            const int k = cell[j], y = k / T, x = k % T;
            const double v0 = vals[k];
            double acc = 4.0 * v0;
            if (y > 0) acc -= vals[k - T];
            if (y + 1 < T) acc -= vals[k + T];
            if (x > 0) acc -= vals[k - 1];
            if (x + 1 < T) acc -= vals[k + 1];
            const double v = v0 + prm.sharpening * acc;
            bit = v > 0.0;
            if (bit) ws += v;
            else bs -= v;
        }
        bal[j] = __ballot_sync(0xFFFFFFFFu, bit);
    }
    const int nwhite = __popc(bal[0]) + __popc(bal[1]);
    ws = warp_sum(ws);
    bs = warp_sum(bs);
    const double margin = fmin(ws / (nwhite + 1.0), bs / (nb - nwhite + 1.0));
    const unsigned long long code = code_of(bal[0], bal[1], nb);
    R.code = code;
    R.decision_margin = (float)margin;
    // 6. nearest code over the four quarter turns: (distance, turns, index)
    unsigned long long best = ~0ull;
    const unsigned long long r1 = rotate_code(code, F), r2 = rotate_code(r1, F), r3 = rotate_code(r2, F);
    for (uint32_t i = lane; i < F.n_codes; i += 32) {
        const unsigned long long c = codes[i];
        // least distance, then fewest turns: distance * 4 + turns
        const uint32_t d0 = 4u * __popcll(code ^ c), d1 = 4u * __popcll(r1 ^ c) + 1u, d2 = 4u * __popcll(r2 ^ c) + 2u,
                       d3 = 4u * __popcll(r3 ^ c) + 3u;
        const unsigned long long key = ((unsigned long long)min(min(d0, d1), min(d2, d3)) << 32) | i;
        best = key < best ? key : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xFFFFFFFFu, best, o);
        best = v < best ? v : best;
    }
    if (best != ~0ull) {
        R.hamming = (uint32_t)(best >> 34);
        const uint32_t turns = (uint32_t)(best >> 32) & 3u;
        if (R.hamming <= F.max_hamming && margin >= 0.0) {
            R.id = (int32_t)(uint32_t)best;
            R.rotation = turns;
            double rx[4], ry[4];
            for (int i = 0; i < 4; i++) {
                rx[i] = px[(i + turns) & 3];
                ry[i] = py[(i + turns) & 3];
            }
            for (int i = 0; i < 4; i++) {
                px[i] = rx[i];
                py[i] = ry[i];
            }
        }
    }
    finish();
}

}  // namespace
}  // namespace atag

using namespace atag;

extern "C" void atag_decode_params_default(atag_decode_params* p) {
    p->decode_sharpening = 0.25f;
    p->refine_edges = 1;
    p->quad_decimate = 1;
    p->min_contrast = 0.0f;
}

extern "C" atag_status atag_decode_quads(const uint8_t* d_image, size_t width, size_t height, size_t pitch,
                                         const float* d_corners, size_t corner_stride, size_t n_quads,
                                         const atag_tag_family* family, const atag_decode_params* params,
                                         atag_decoded* d_out, atag_stream_t stream) {
    atag_status st = atag_init();
    if (st) return st;
    if (!family) return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: null family");
    if (n_quads == 0) return ATAG_OK;
    if (!d_image || !d_corners || !d_out || (family->n_codes && !family->d_codes) || !family->h_bit_x ||
        !family->h_bit_y)
        return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: null pointer");
    if (width < 2 || height < 2 || width > (size_t)INT32_MAX || height > (size_t)INT32_MAX)
        return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: image smaller than 2x2 or too large");
    if (pitch == 0) pitch = width;
    if (pitch < width) return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: pitch below width");
    if (corner_stride < 8 * sizeof(float) || corner_stride % 4)
        return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: corner stride below 32 bytes or not a multiple of 4");
    if (reinterpret_cast<uintptr_t>(d_corners) % 4 || reinterpret_cast<uintptr_t>(d_out) % 8 ||
        reinterpret_cast<uintptr_t>(family->d_codes) % 8)
        return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: misaligned corners, codes or output");
    if (n_quads > (size_t)UINT32_MAX || family->n_codes > (1u << 24))
        return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: too many quads or codes");
    const int nb = (int)family->nbits, W = (int)family->width_at_border, T = (int)family->total_width;
    if (nb < 1 || nb > 64 || W < 3 || T < 1 || T > MAX_TW || (W - T) % 2 != 0)
        return set_error(ATAG_ERR_INVALID_ARGUMENT,
                         "decode_quads: family needs 1..64 bits, width_at_border >= 3, total_width <= 16 with "
                         "total_width - width_at_border even");
    FamilyDesc F;
    memset(&F, 0, sizeof F);
    F.nbits = nb;
    F.width_at_border = W;
    F.total_width = T;
    F.reversed_border = family->reversed_border ? 1 : 0;
    F.n_codes = family->n_codes;
    F.max_hamming = family->max_hamming;
    const int m = (W - T) / 2;
    // every bit's cell must lie on the grid, be used once, and a quarter turn
    // must carry the bit cells onto bit cells (the families are symmetric)
    std::vector<int> at((size_t)T * T, -1);
    for (int i = 0; i < nb; i++) {
        const int x = family->h_bit_x[i], y = family->h_bit_y[i];
        if (x - m < 0 || x - m >= T || y - m < 0 || y - m >= T || at[(size_t)(y - m) * T + (x - m)] >= 0)
            return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: bit cell off the tag grid or used twice");
        at[(size_t)(y - m) * T + (x - m)] = i;
        F.bit_x[i] = (int8_t)x;
        F.bit_y[i] = (int8_t)y;
    }
    for (int i = 0; i < nb; i++) {
        const int sx = W - 1 - F.bit_y[i], sy = F.bit_x[i];
        const int j = (sx - m >= 0 && sx - m < T && sy - m >= 0 && sy - m < T) ? at[(size_t)(sy - m) * T + (sx - m)] : -1;
        if (j < 0) return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: the bit layout is not symmetric under quarter turns");
        F.perm[i] = (uint8_t)j;
    }
    atag_decode_params p;
    if (params) p = *params; else atag_decode_params_default(&p);
    if (p.quad_decimate < 1 || p.quad_decimate > 8)
        return set_error(ATAG_ERR_INVALID_ARGUMENT, "decode_quads: quad_decimate must be 1..8");
    DecodeParams prm{(double)p.decode_sharpening, (double)p.min_contrast, p.refine_edges ? 1 : 0, p.quad_decimate};
    const uint32_t n = (uint32_t)n_quads;
    k_decode_quads<<<(n + DECODE_WARPS - 1) / DECODE_WARPS, 32 * DECODE_WARPS, 0, (cudaStream_t)stream>>>(
        d_image, (int)width, (int)height, pitch, reinterpret_cast<const uint8_t*>(d_corners), corner_stride, n,
        reinterpret_cast<const unsigned long long*>(family->d_codes), F, prm, d_out);
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ATAG_OK : set_error(ATAG_ERR_CUDA, cudaGetErrorString(e));
}
