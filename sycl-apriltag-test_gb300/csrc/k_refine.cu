// k_refine.cu — subpixel corner refinement: forward and hand-written adjoint.
//
// The reference stops at the corners of process_fitted_quads
// (src/main.cpp:1035-1162); this stage (new, no counterpart there) refines
// them on an FP32 image the way AprilTag refines edges:
//
//   for each edge e = corner a -> corner b (d = (b-a)/|b-a|, n = (-d_y, d_x)):
//     for j in 0..15:  p_j = a + t_j (b - a),  t_j = (j + 0.5) / 16
//       4 taps across the edge: v_jk = I(p_j + u_k n), u = (-1.5,-0.5,0.5,1.5)
//       (bilinear, clamped to the image: 64 samples per edge)
//       g_m = v_j(m+1) - v_jm, w_m = g_m^2, Omega_j = sum w_m,
//       o_j = (sum w_m c_m) / (Omega_j + eps), c = (-1, 0, 1)
//       edge point q_j = p_j + o_j n with weight W_j = Omega_j + eps
//     weighted line fit of (q_j, W_j): moments in FP32 about the edge
//     midpoint, covariance eigen-solve in FP64: centroid m_e, direction
//     u_e = (cos phi, sin phi), phi = atan2(2 cxy, cxx - cyy) / 2,
//     residual r_e = sum_j W_j d_j^2, d_j the distance of q_j to the line
//     (= S0 * lambda_min, computed in a second pass without cancellation)
//   refined corner i = intersection of lines of edges i-1 and i (FP64).
//
// Forward writes the refined corners, the residuals and the 256 sampled
// intensities per quad; backward recomputes the forward and propagates
// dL/d(refined corners) and dL/d(residuals) to dL/d(corners), dL/d(samples)
// and, optionally, dL/d(image) (scattered through the bilinear weights).
//
// A warp takes an edge (two samples per lane); the FP64 part of an edge (the
// eigen-solve, the intersections and their adjoints) has no lane-level
// parallelism, and on this GPU FP64 issues at 2 lanes per clock and SM
// whether a warp's lanes do different work or the same.  So the edges' moments
// go through shared memory, and one warp of the CTA takes all of its edges'
// FP64 parts at once, lane = edge (up to 32 edges of 8 quads).  With every
// lane of every edge's warp solving its own edge redundantly, the FP64 pipe
// was 80-85% busy: 4,096 quads took 167 us forward and 339 us backward, and
// take 22 and 64 us now (single launches, cold caches).
#include <algorithm>

#include "atag_internal.h"
#include "atag_kernels.cuh"

namespace atag {
namespace {

constexpr int RF_POS = 16, RF_TAPS = 4;
constexpr float RF_EPS = 1e-6f;
__device__ __constant__ float RF_U[4] = {-1.5f, -0.5f, 0.5f, 1.5f};

struct Bilinear {
    float v, gx, gy;  // value and its spatial gradient
};

// Pixel sources: an FP32 image, or the detector's u8 grey frame read as
// value / 255 (the same numbers as the FP32-normalised image).
struct F32Image {
    const float* __restrict__ p;
    __device__ __forceinline__ float operator[](size_t i) const { return __ldg(p + i); }
};
struct U8Image {
    const uint8_t* __restrict__ p;
    __device__ __forceinline__ float operator[](size_t i) const { return __fdiv_rn((float)__ldg(p + i), 255.0f); }
};

template <class Img>
__device__ __forceinline__ Bilinear bilinear(const Img& img, int w, int h, float x, float y) {
    const float xc = fminf(fmaxf(x, 0.0f), (float)(w - 1)), yc = fminf(fmaxf(y, 0.0f), (float)(h - 1));
    const bool inx = x > 0.0f && x < (float)(w - 1), iny = y > 0.0f && y < (float)(h - 1);
    int x0 = (int)floorf(xc), y0 = (int)floorf(yc);
    x0 = min(x0, w - 2);
    y0 = min(y0, h - 2);
    const float fx = xc - (float)x0, fy = yc - (float)y0;
    const float i00 = img[(size_t)y0 * w + x0], i01 = img[(size_t)y0 * w + x0 + 1];
    const float i10 = img[(size_t)(y0 + 1) * w + x0], i11 = img[(size_t)(y0 + 1) * w + x0 + 1];
    Bilinear b;
    b.v = (1.0f - fy) * ((1.0f - fx) * i00 + fx * i01) + fy * ((1.0f - fx) * i10 + fx * i11);
    b.gx = inx ? (1.0f - fy) * (i01 - i00) + fy * (i11 - i10) : 0.0f;
    b.gy = iny ? (1.0f - fx) * (i10 - i00) + fx * (i11 - i01) : 0.0f;
    return b;
}

__device__ __forceinline__ void bilinear_scatter(float* __restrict__ gimg, int w, int h, float x, float y, float g) {
    const float xc = fminf(fmaxf(x, 0.0f), (float)(w - 1)), yc = fminf(fmaxf(y, 0.0f), (float)(h - 1));
    int x0 = min((int)floorf(xc), w - 2), y0 = min((int)floorf(yc), h - 2);
    const float fx = xc - (float)x0, fy = yc - (float)y0;
    atomicAdd(gimg + (size_t)y0 * w + x0, g * (1.0f - fx) * (1.0f - fy));
    atomicAdd(gimg + (size_t)y0 * w + x0 + 1, g * fx * (1.0f - fy));
    atomicAdd(gimg + (size_t)(y0 + 1) * w + x0, g * (1.0f - fx) * fy);
    atomicAdd(gimg + (size_t)(y0 + 1) * w + x0 + 1, g * fx * fy);
}

constexpr int RF_WARPS = 4, RF_QUADS = 8, RF_EDGES = 4 * RF_QUADS;

// The fitted line of an edge, FP64.
struct EdgeLine {
    double mx, my, ux, uy;                          // line
    double S0, Sx, Sy, Sxx, Syy, Sxy;               // moments about (ox, oy)
    double cxx, cyy, cxy;
};

// What an edge's warp hands to the FP64 lane, and what it gets back.
struct EdgeSums {
    float m6[6], ox, oy, dx, dy, nx, ny;
    float pad_;  // 13 words: lanes of the FP64 warp read distinct banks
};
struct EdgeFit {
    float cs, cn, c0;      // distance of q_j to the line: sa cs + o cn - c0
    float nux, nuy;        // its normal
};

struct LaneState {
    // position j = lane / 2 owns taps 2*(lane&1) .. +1
    float dx, dy, nx, ny, len, t;
    Bilinear s[2];
    float sx[2], sy[2];
    // position-level values (valid on even lanes)
    float v[4], gd[3], w[3], Om, Nn, o, W;
    float sa;              // (t_j - 1/2) |b - a|: q_j - midpoint = sa d + o n
};

// FP32 part of an edge on its warp: samples, edge points and the moments of
// the line fit (in S, written by lane 0).
template <class Img>
__device__ __forceinline__ void edge_samples(const Img& img, int iw, int ih, float ax, float ay, float bx, float by,
                                             LaneState& L, EdgeSums& S) {
    const int lane = threadIdx.x & 31, j = lane >> 1, half = lane & 1;
    const float Dx = bx - ax, Dy = by - ay;
    L.len = fmaxf(sqrtf(Dx * Dx + Dy * Dy), 1e-6f);
    L.dx = Dx / L.len;
    L.dy = Dy / L.len;
    L.nx = -L.dy;
    L.ny = L.dx;
    L.t = ((float)j + 0.5f) / (float)RF_POS;
    const float px = ax + L.t * Dx, py = ay + L.t * Dy;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float u = RF_U[2 * half + i];
        L.sx[i] = px + u * L.nx;
        L.sy[i] = py + u * L.ny;
        L.s[i] = bilinear(img, iw, ih, L.sx[i], L.sy[i]);
    }
    // gather the 4 taps of position j on its even lane
    const float o0 = __shfl_xor_sync(0xffffffffu, L.s[0].v, 1), o1 = __shfl_xor_sync(0xffffffffu, L.s[1].v, 1);
    L.v[0] = half ? o0 : L.s[0].v;
    L.v[1] = half ? o1 : L.s[1].v;
    L.v[2] = half ? L.s[0].v : o0;
    L.v[3] = half ? L.s[1].v : o1;
    L.Om = 0.0f;
    L.Nn = 0.0f;
#pragma unroll
    for (int m = 0; m < 3; m++) {
        L.gd[m] = L.v[m + 1] - L.v[m];
        L.w[m] = L.gd[m] * L.gd[m];
        L.Om += L.w[m];
        L.Nn += L.w[m] * (float)(m - 1);
    }
    L.o = L.Nn / (L.Om + RF_EPS);
    L.W = L.Om + RF_EPS;  // a contrast-free edge falls back to the unrefined line
    // moments about the edge midpoint, one contribution per position; the
    // point is taken relative to the midpoint in the edge's own frame
    // ((j - 7.5) / 16 is exact), not as a difference of image coordinates
    const float ox = 0.5f * (ax + bx), oy = 0.5f * (ay + by);
    L.sa = ((float)j - 0.5f * (RF_POS - 1)) / (float)RF_POS * L.len;
    const float X = L.sa * L.dx + L.o * L.nx, Y = L.sa * L.dy + L.o * L.ny, Wc = half ? 0.0f : L.W;
    float m6[6] = {Wc, Wc * X, Wc * Y, Wc * X * X, Wc * Y * Y, Wc * X * Y};
#pragma unroll
    for (int k = 0; k < 6; k++)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) m6[k] += __shfl_xor_sync(0xffffffffu, m6[k], off);
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 6; k++) S.m6[k] = m6[k];
        S.ox = ox; S.oy = oy;
        S.dx = L.dx; S.dy = L.dy; S.nx = L.nx; S.ny = L.ny;
    }
}

// FP64 part of an edge on one lane: the eigen-solve of the 2x2 covariance.
// The direction of the larger eigenvalue, (cos phi, sin phi) with phi =
// atan2(2 cxy, cxx - cyy) / 2, follows without trigonometry from the
// eigenvector (R + h, cxy) or, for h < 0, (|cxy|, +-(R - h)), h = (cxx - cyy)
// / 2, R = sqrt(h^2 + cxy^2): both components are sums of terms of one sign.
__device__ __forceinline__ void solve_line(const EdgeSums& S, EdgeLine& E, EdgeFit& fit) {
    E.S0 = fmax((double)S.m6[0], 1e-30);
    E.Sx = S.m6[1]; E.Sy = S.m6[2]; E.Sxx = S.m6[3]; E.Syy = S.m6[4]; E.Sxy = S.m6[5];
    const double mx = E.Sx / E.S0, my = E.Sy / E.S0;
    E.cxx = E.Sxx / E.S0 - mx * mx;
    E.cyy = E.Syy / E.S0 - my * my;
    E.cxy = E.Sxy / E.S0 - mx * my;
    const double h = 0.5 * (E.cxx - E.cyy);
    const double R = sqrt(h * h + E.cxy * E.cxy);
    const double vx = h >= 0.0 ? R + h : fabs(E.cxy), vy = h >= 0.0 ? E.cxy : copysign(R - h, E.cxy);
    const double len = sqrt(vx * vx + vy * vy);
    E.mx = (double)S.ox + mx;
    E.my = (double)S.oy + my;
    E.ux = len == 0.0 ? 1.0 : vx / len;
    E.uy = len == 0.0 ? 0.0 : vy / len;
    // residual sum W_j d_j^2 of the perpendicular distances to the fitted
    // line, in a second pass (S0 * lambda_min from the moments would
    // cancel), in the edge frame: d_j = sa (d.nu) + o (n.nu) - (m.nu), whose
    // terms are small where the line runs along the edge
    const double nux = -E.uy, nuy = E.ux;
    fit.nux = (float)nux;
    fit.nuy = (float)nuy;
    fit.cs = (float)((double)S.dx * nux + (double)S.dy * nuy);
    fit.cn = (float)((double)S.nx * nux + (double)S.ny * nuy);
    fit.c0 = (float)(mx * nux + my * nuy);
}

// Intersection of line A (m_A + alpha u_A) with line B, FP64.
struct Crossing {
    double cx, cy, alpha, P, Q, Dx, Dy;
};
__device__ __forceinline__ Crossing intersect(double amx, double amy, double aux, double auy, const EdgeLine& B) {
    Crossing X;
    X.Dx = B.mx - amx;
    X.Dy = B.my - amy;
    X.P = B.ux * X.Dy - B.uy * X.Dx;
    X.Q = B.ux * auy - B.uy * aux;
    X.alpha = X.P / X.Q;
    X.cx = amx + X.alpha * aux;
    X.cy = amy + X.alpha * auy;
    return X;
}
// Lane 4 q + i of the FP64 warp: corner i of quad q, the crossing of lines
// i - 1 (A, fetched from its lane) and i (B, this lane's).
__device__ __forceinline__ Crossing corner_of(const EdgeLine& E, double* aux, double* auy) {
    const int lane = threadIdx.x & 31, prev = (lane & ~3) | ((lane + 3) & 3);
    const double amx = __shfl_sync(0xffffffffu, E.mx, prev), amy = __shfl_sync(0xffffffffu, E.my, prev);
    *aux = __shfl_sync(0xffffffffu, E.ux, prev);
    *auy = __shfl_sync(0xffffffffu, E.uy, prev);
    return intersect(amx, amy, *aux, *auy, E);
}

// Quads per CTA: four CTAs per SM put one FP64 warp on each of its four
// schedulers (the FP64 warp's index turns with the CTA), and few quads spread
// over the SMs one by one.
inline unsigned refine_quads_per_cta(size_t n) {
    const size_t slots = 4 * (size_t)device_sms();
    return (unsigned)std::min<size_t>(RF_QUADS, (n + slots - 1) / slots);
}

}  // namespace

__global__ void __launch_bounds__(32 * RF_WARPS) k_refine_forward(const float* __restrict__ img, int iw, int ih,
                                                        const float* __restrict__ corners, int nq, int qpc,
                                                        float* __restrict__ refined, float* __restrict__ residual,
                                                        float* __restrict__ samples) {
    __shared__ EdgeSums sums[RF_EDGES];
    __shared__ EdgeFit fits[RF_EDGES];
    __shared__ float pos[RF_EDGES][RF_POS][3];  // sa, o, W of each position
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t q0 = (size_t)blockIdx.x * qpc;
    const int ne = 4 * min(qpc, nq - (int)q0);
    for (int k = warp; k < ne; k += RF_WARPS) {
        const int e = k & 3, e1 = (e + 1) & 3, j = lane >> 1, half = lane & 1;
        const float* c = corners + (q0 + (k >> 2)) * 8;
        LaneState L;
        edge_samples(F32Image{img}, iw, ih, c[2 * e], c[2 * e + 1], c[2 * e1], c[2 * e1 + 1], L, sums[k]);
        if (samples) {
            float* s = samples + (q0 * 4 + k) * (RF_POS * RF_TAPS) + j * RF_TAPS + 2 * half;
            s[0] = L.s[0].v;
            s[1] = L.s[1].v;
        }
        if (!half) {
            pos[k][j][0] = L.sa;
            pos[k][j][1] = L.o;
            pos[k][j][2] = L.W;
        }
    }
    __syncthreads();
    if (warp == (blockIdx.x & (RF_WARPS - 1))) {
        EdgeLine E;
        EdgeFit fit;
        solve_line(sums[min(lane, ne - 1)], E, fit);
        double aux, auy;
        const Crossing X = corner_of(E, &aux, &auy);
        if (lane < ne) {
            fits[lane] = fit;
            refined[q0 * 8 + 2 * lane] = (float)X.cx;
            refined[q0 * 8 + 2 * lane + 1] = (float)X.cy;
        }
    }
    if (!residual) return;
    __syncthreads();
    for (int k = warp; k < ne; k += RF_WARPS) {
        const int j = lane >> 1, half = lane & 1;
        const float sa = pos[k][j][0], o = pos[k][j][1], W = pos[k][j][2];
        const EdgeFit f = fits[k];
        const float dist = sa * f.cs + o * f.cn - f.c0;
        float rr = half ? 0.0f : W * dist * dist;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) rr += __shfl_xor_sync(0xffffffffu, rr, off);
        if (lane == 0) residual[q0 * 4 + k] = rr;
    }
}

// Refinement of the detector's own quads, in place, as the last stage of a
// detect call: the frame's u8 grey image, read as value / 255, gives the
// same refined corners as atag_refine_forward on the FP32-normalised image.
// A corner whose two edge lines are nearly parallel (|sin| of their angle
// at most 1e-3) keeps its unrefined position.  Frame blockIdx.x; its quads
// blockIdx.y, blockIdx.y + gridDim.y, ...
__global__ void __launch_bounds__(32 * RF_WARPS) k_refine_detected(const __grid_constant__ FrameSet fs) {
    if (fs.overlap) await_previous_kernel();
    __shared__ EdgeSums sums[4];
    const FrameDesc& F = fs.of_table(blockIdx.x);
    const uint32_t nq = min(F.stats->n_quads, F.quad_cap);
    const U8Image img{F.grey};
    const int e = threadIdx.x >> 5, lane = threadIdx.x & 31, e1 = (e + 1) & 3;
    for (uint32_t q = blockIdx.y; q < nq; q += gridDim.y) {
        atag_quad_corners* qc = F.quads + q;
        const float ax = qc->corners[e][0], ay = qc->corners[e][1], bx = qc->corners[e1][0], by = qc->corners[e1][1];
        LaneState L;
        edge_samples(img, (int)F.width, (int)F.height, ax, ay, bx, by, L, sums[e]);
        __syncthreads();  // also: every warp has read the corners
        if (e == (int)(blockIdx.y & (RF_WARPS - 1))) {
            EdgeLine E;
            EdgeFit fit;
            solve_line(sums[lane & 3], E, fit);
            double aux, auy;
            const Crossing X = corner_of(E, &aux, &auy);
            if (lane < 4 && fabs(X.Q) > 1e-3 && isfinite(X.cx) && isfinite(X.cy)) {
                qc->corners[lane][0] = (float)X.cx;
                qc->corners[lane][1] = (float)X.cy;
            }
        }
        __syncthreads();
    }
}

// What the FP64 lane of an edge hands back for the adjoint: the adjoints of
// its moments, of the origin (through the centroid) and of its residual.
struct EdgeAdjoint {
    double gS0, gSx, gSy, gSxx, gSyy, gSxy;
    float gox, goy, gr;
};

__global__ void __launch_bounds__(32 * RF_WARPS) k_refine_backward(const float* __restrict__ img, int iw, int ih,
                                                         const float* __restrict__ corners, int nq, int qpc,
                                                         const float* __restrict__ g_refined,
                                                         const float* __restrict__ g_residual,
                                                         float* __restrict__ g_corners, float* __restrict__ g_samples,
                                                         float* __restrict__ g_image) {
    __shared__ EdgeSums sums[RF_EDGES];
    __shared__ EdgeFit fits[RF_EDGES];
    __shared__ EdgeAdjoint adj[RF_EDGES];
    __shared__ float gc[RF_EDGES][2];       // adjoints of the input corners
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, j = lane >> 1, half = lane & 1;
    const size_t q0 = (size_t)blockIdx.x * qpc;
    const int ne = 4 * min(qpc, nq - (int)q0);
    if (threadIdx.x < 2 * RF_EDGES) (&gc[0][0])[threadIdx.x] = 0.0f;
    // pass 0 gathers the moments of the CTA's edges; pass 1, with their
    // adjoints, repeats an edge's FP32 forward (its pixels are in L1) rather
    // than keeping its lanes' states
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
        for (int k = warp; k < ne; k += RF_WARPS) {
            const int e = k & 3, e1 = (e + 1) & 3;
            const float* c = corners + (q0 + (k >> 2)) * 8;
            LaneState L;
            edge_samples(F32Image{img}, iw, ih, c[2 * e], c[2 * e + 1], c[2 * e1], c[2 * e1 + 1], L, sums[k]);
            if (pass == 0) continue;
            const EdgeFit f = fits[k];
            const EdgeAdjoint& G = adj[k];
            const float dist = L.sa * f.cs + L.o * f.cn - f.c0;
            // moments -> edge point q_j and weight W_j (even lanes own position j)
            const float X = L.sa * L.dx + L.o * L.nx, Y = L.sa * L.dy + L.o * L.ny;
            const float grf = G.gr;
            float gW = (float)(G.gS0 + G.gSx * X + G.gSy * Y + G.gSxx * X * X + G.gSyy * Y * Y + G.gSxy * X * Y) +
                       grf * dist * dist;
            float gqx = (float)(L.W * (G.gSx + 2.0 * G.gSxx * X + G.gSxy * Y)) + grf * 2.0f * L.W * dist * f.nux;
            float gqy = (float)(L.W * (G.gSy + 2.0 * G.gSyy * Y + G.gSxy * X)) + grf * 2.0f * L.W * dist * f.nuy;
            // X = q_x - o_x with q = p + o n and o the midpoint (the forward
            // evaluates the same quantity as sa d_x + o n_x)
            float gox = -gqx, goy = -gqy;
            float gpx = gqx, gpy = gqy;
            const float go = gqx * L.nx + gqy * L.ny;
            float gnx = L.o * gqx, gny = L.o * gqy;
            const float den_o = L.Om + RF_EPS;
            const float gN = go / den_o;
            const float gOm = gW - go * L.Nn / (den_o * den_o);
            float gv[4] = {0, 0, 0, 0};
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const float gw = gN * (float)(m - 1) + gOm;
                const float ggd = 2.0f * L.gd[m] * gw;
                gv[m + 1] += ggd;
                gv[m] -= ggd;
            }
            if (half) {  // only even lanes carry position-level adjoints
                gpx = gpy = gnx = gny = gox = goy = 0.0f;
                gv[0] = gv[1] = gv[2] = gv[3] = 0.0f;
            }
            if (lane == 0) {  // the line's centroid is origin + S_x / S_0: direct path to the origin
                gox += G.gox;
                goy += G.goy;
            }
            // hand the adjoints of taps 2, 3 to the odd lane
            const float t2 = __shfl_xor_sync(0xffffffffu, gv[2], 1), t3 = __shfl_xor_sync(0xffffffffu, gv[3], 1);
            const float gs0 = half ? t2 : gv[0], gs1 = half ? t3 : gv[1];
            if (g_samples) {
                float* s = g_samples + (q0 * 4 + k) * (RF_POS * RF_TAPS) + j * RF_TAPS + 2 * half;
                s[0] = gs0;
                s[1] = gs1;
            }
            // samples -> sample positions -> p_j, n
            const float gsv[2] = {gs0, gs1};
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float u = RF_U[2 * half + i];
                const float gx = gsv[i] * L.s[i].gx, gy = gsv[i] * L.s[i].gy;
                gpx += gx;
                gpy += gy;
                gnx += u * gx;
                gny += u * gy;
                if (g_image) bilinear_scatter(g_image, iw, ih, L.sx[i], L.sy[i], gsv[i]);
            }
            // p = a + t (b - a); origin = (a + b) / 2; n = (-d_y, d_x), d = (b - a) / |b - a|
            float gax = (1.0f - L.t) * gpx + 0.5f * gox, gay = (1.0f - L.t) * gpy + 0.5f * goy;
            float gbx = L.t * gpx + 0.5f * gox, gby = L.t * gpy + 0.5f * goy;
            const float gdx = gny, gdy = -gnx;
            const float dd = L.dx * gdx + L.dy * gdy;
            const float gDx = (gdx - L.dx * dd) / L.len, gDy = (gdy - L.dy * dd) / L.len;
            gax -= gDx; gay -= gDy; gbx += gDx; gby += gDy;
            float acc[4] = {gax, gay, gbx, gby};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
            if (lane == 0) {  // two edges add to each corner
                atomicAdd(&gc[k][0], acc[0]);
                atomicAdd(&gc[k][1], acc[1]);
                atomicAdd(&gc[(k & ~3) | e1][0], acc[2]);
                atomicAdd(&gc[(k & ~3) | e1][1], acc[3]);
            }
        }
        __syncthreads();
        if (pass == 0) {
            if (warp == (blockIdx.x & (RF_WARPS - 1))) {
                EdgeLine E;
                EdgeFit fit;
                const int k = min(lane, ne - 1);
                solve_line(sums[k], E, fit);
                // adjoint of corner i (this lane), the crossing of lines A = i - 1
                // (the lane before in its quad) and B = i (this lane's own)
                double aux, auy;
                const Crossing C = corner_of(E, &aux, &auy);
                const double gcx = g_refined ? (double)g_refined[q0 * 8 + 2 * k] : 0.0;
                const double gcy = g_refined ? (double)g_refined[q0 * 8 + 2 * k + 1] : 0.0;
                const double ga = gcx * aux + gcy * auy;
                const double gP = ga / C.Q, gQ = -ga * C.P / (C.Q * C.Q);
                const double gDx = -gP * E.uy, gDy = gP * E.ux;
                // Q = uBx uAy - uBy uAx, P = uBx Dy - uBy Dx
                double gmx_a = gcx - gDx, gmy_a = gcy - gDy;
                double gux_a = C.alpha * gcx - gQ * E.uy, guy_a = C.alpha * gcy + gQ * E.ux;
                // line i's adjoints: as B of its own corner, as A of the next lane's
                const int next = (lane & ~3) | ((lane + 1) & 3);
                gmx_a = __shfl_sync(0xffffffffu, gmx_a, next);
                gmy_a = __shfl_sync(0xffffffffu, gmy_a, next);
                gux_a = __shfl_sync(0xffffffffu, gux_a, next);
                guy_a = __shfl_sync(0xffffffffu, guy_a, next);
                const double gmx0 = gDx + gmx_a, gmy0 = gDy + gmy_a;
                const double gux = gP * C.Dy + gQ * auy + gux_a, guy = -gP * C.Dx - gQ * aux + guy_a;
                // line adjoint -> moment adjoints
                const double gphi = -E.uy * gux + E.ux * guy;
                const double Xc = E.cxx - E.cyy, Yc = 2.0 * E.cxy, den = Xc * Xc + Yc * Yc;
                double gcxx = 0, gcyy = 0, gcxy = 0;
                if (den > 1e-300) {
                    const double s = gphi / den;
                    gcxy = s * Xc;
                    gcxx = -0.5 * s * Yc;
                    gcyy = 0.5 * s * Yc;
                }
                // the residual's gradient needs no path through the line: the line
                // minimises sum W d^2, so only q_j and W_j move it (envelope theorem)
                const double is = 1.0 / E.S0, mx = E.Sx * is, my = E.Sy * is;
                const double gmx = gmx0 - 2.0 * mx * gcxx - my * gcxy;
                const double gmy = gmy0 - 2.0 * my * gcyy - mx * gcxy;
                if (lane < ne) {
                    fits[lane] = fit;
                    EdgeAdjoint G;
                    G.gSxx = gcxx * is;
                    G.gSyy = gcyy * is;
                    G.gSxy = gcxy * is;
                    G.gSx = gmx * is;
                    G.gSy = gmy * is;
                    G.gS0 = -(E.Sxx * gcxx + E.Syy * gcyy + E.Sxy * gcxy + E.Sx * gmx + E.Sy * gmy) * (is * is);
                    G.gox = (float)gmx0;
                    G.goy = (float)gmy0;
                    G.gr = g_residual ? g_residual[q0 * 4 + lane] : 0.0f;
                    adj[lane] = G;
                }
            }
            __syncthreads();
        }
    }
    if (threadIdx.x < 2 * ne) g_corners[q0 * 8 + threadIdx.x] = (&gc[0][0])[threadIdx.x];
}

}  // namespace atag

using namespace atag;

extern "C" atag_status atag_refine_forward(const float* d_image, size_t width, size_t height, const float* d_corners,
                                           size_t n_quads, float* d_refined, float* d_residual, float* d_samples,
                                           atag_stream_t stream) {
    atag_status st = atag_init();
    if (st) return st;
    if (!d_image || !d_corners || !d_refined) return set_error(ATAG_ERR_INVALID_ARGUMENT, "refine_forward: null pointer");
    if (width < 2 || height < 2) return set_error(ATAG_ERR_INVALID_ARGUMENT, "refine_forward: image smaller than 2x2");
    if (n_quads == 0) return ATAG_OK;
    if (n_quads > (size_t)INT32_MAX) return set_error(ATAG_ERR_INVALID_ARGUMENT, "refine_forward: too many quads");
    const unsigned qpc = refine_quads_per_cta(n_quads);
    k_refine_forward<<<(unsigned)((n_quads + qpc - 1) / qpc), 32 * RF_WARPS, 0, (cudaStream_t)stream>>>(
        d_image, (int)width, (int)height, d_corners, (int)n_quads, (int)qpc, d_refined, d_residual, d_samples);
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ATAG_OK : set_error(ATAG_ERR_CUDA, cudaGetErrorString(e));
}

extern "C" atag_status atag_refine_backward(const float* d_image, size_t width, size_t height, const float* d_corners,
                                            size_t n_quads, const float* d_grad_refined, const float* d_grad_residual,
                                            float* d_grad_corners, float* d_grad_samples, float* d_grad_image,
                                            atag_stream_t stream) {
    atag_status st = atag_init();
    if (st) return st;
    if (!d_image || !d_corners || !d_grad_corners)
        return set_error(ATAG_ERR_INVALID_ARGUMENT, "refine_backward: null pointer");
    if (width < 2 || height < 2) return set_error(ATAG_ERR_INVALID_ARGUMENT, "refine_backward: image smaller than 2x2");
    if (n_quads == 0) return ATAG_OK;
    if (n_quads > (size_t)INT32_MAX) return set_error(ATAG_ERR_INVALID_ARGUMENT, "refine_backward: too many quads");
    const unsigned qpc = refine_quads_per_cta(n_quads);
    k_refine_backward<<<(unsigned)((n_quads + qpc - 1) / qpc), 32 * RF_WARPS, 0, (cudaStream_t)stream>>>(
        d_image, (int)width, (int)height, d_corners, (int)n_quads, (int)qpc, d_grad_refined, d_grad_residual,
        d_grad_corners, d_grad_samples, d_grad_image);
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ATAG_OK : set_error(ATAG_ERR_CUDA, cudaGetErrorString(e));
}
