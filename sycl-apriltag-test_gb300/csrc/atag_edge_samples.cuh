// atag_edge_samples.cuh — the points at which tag reading looks for an edge:
// how many an edge has, and which of them can meet the image.  Corners come
// from the caller (or from corner refinement, where nearly parallel lines meet
// anywhere), so neither the number nor its product with anything may overflow,
// and the work has to stay bounded by the image.
#pragma once
#include <cmath>

namespace atag {

// max(16, length / 8), kept where s + 8 and count + 1 stay below 2^31.
__host__ __device__ __forceinline__ int edge_sample_count(double length) {
    return (int)fmax(16.0, fmin(length / 8.0, 2147483600.0));
}

// Edges of up to this many points (32,768 px) are walked whole.
constexpr int EDGE_SAMPLES_WHOLE = 4096;

// The points [lo, hi) of `count` that can come within `reach` px of a w x h
// image; point s lies at alpha a + (1 - alpha) b, alpha = (1 + s) / (count +
// 1).  The others read no pixel.  A longer edge's points are at least 7.9 px
// apart, so about (w + h + 4 reach) / 7.9 are left, whatever its length.  The
// margin covers the rounding of the points and of this arithmetic; lo is a
// multiple of 8, which keeps each point on the lane that it has in a whole walk.
struct SampleRange {
    int lo, hi;
};
__host__ __device__ __forceinline__ SampleRange edge_sample_range(double ax, double ay, double bx, double by, int count,
                                                                  int reach, int w, int h) {
    double a0 = 0.0, a1 = 1.0;
    for (int axis = 0; axis < 2; axis++) {
        const double a = axis ? ay : ax, b = axis ? by : bx, d = a - b;
        const double margin = reach + 1.0 + 0x1p-40 * (fabs(a) + fabs(b));
        const double low = -margin - b, high = (axis ? h : w) + margin - b;
        if (d == 0.0) {
            if (low > 0.0 || high < 0.0) return SampleRange{0, 0};
            continue;
        }
        const double t0 = low / d, t1 = high / d;
        a0 = fmax(a0, fmin(t0, t1));
        a1 = fmin(a1, fmax(t0, t1));
    }
    if (a0 > a1) return SampleRange{0, 0};
    const double n1 = (double)count + 1.0;
    const int lo = (int)fmax(0.0, floor(a0 * n1) - 2.0), hi = (int)fmin((double)count, ceil(a1 * n1) + 1.0);
    return SampleRange{lo & ~7, hi};
}

}  // namespace atag
