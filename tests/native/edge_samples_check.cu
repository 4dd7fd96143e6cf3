// Checks atag_edge_samples.cuh on the host: every point of an edge that can
// meet the image is in the range, the range's size is bounded by the image
// whatever the edge's length, and counts stay where s + 8 does not overflow.
// Prints "<edges> <failures>" and exits non-zero on a failure.
#include <cfloat>
#include <cstdio>
#include <random>

#include "../../sycl-apriltag-test_gb300/csrc/atag_edge_samples.cuh"

using namespace atag;

static long long edges = 0, bad = 0;

static void check(float fax, float fay, float fbx, float fby, int reach, int w, int h) {
    const double ax = fax, ay = fay, bx = fbx, by = fby;
    const double length = std::sqrt((bx - ax) * (bx - ax) + (by - ay) * (by - ay));
    const int n = edge_sample_count(length);
    const SampleRange R = edge_sample_range(ax, ay, bx, by, n, reach, w, h);
    edges++;
    bool ok = n >= 16 && n <= 0x7FFFFFFF - 16 && R.lo >= 0 && R.lo % 8 == 0 && R.hi <= n;
    const double most = (w + h + 4.0 * reach + 8.0 + 4 * 0x1p-40 * length) / 7.5 + 24.0;
    if (n > 16 && R.hi - R.lo > most) ok = false;
    // all points of short edges, a spread of the long ones' and those about the range
    const long long step = n > 200000 ? n / 100000 : 1;
    auto point = [&](long long s) {
        if (s < 0 || s >= n) return;
        const double alpha = (1.0 + s) / (n + 1.0);
        const double x = alpha * ax + (1.0 - alpha) * bx, y = alpha * ay + (1.0 - alpha) * by;
        const bool meets = x > -0.5 - reach && x < w + 0.5 + reach && y > -0.5 - reach && y < h + 0.5 + reach;
        if (meets && !(s >= R.lo && s < R.hi)) ok = false;
    };
    for (long long s = 0; s < n; s += step) point(s);
    for (long long d = -3000; d <= 3000; d++) {
        point(R.lo + d);
        point(R.hi + d);
    }
    if (!ok && bad++ < 10)
        printf("a=(%a, %a) b=(%a, %a) reach %d image %d x %d: count %d, range [%d, %d)\n", fax, fay, fbx, fby, reach, w,
               h, n, R.lo, R.hi);
}

int main() {
    std::mt19937 rng(7);
    auto uniform = [&](double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); };
    const int sizes[][2] = {{2, 2}, {640, 480}, {3840, 2160}, {20000, 30}};
    for (double far : {1e3, 3e4, 1e5, 1e6, 1e9, 1.6e10, 1.8e10, 1e15, 1e30, 1e38})
        for (const auto& z : sizes)
            for (int k = 0; k < 40; k++) {
                const int reach = 3 + k % 8;
                const double inx = uniform(-20, z[0] + 20), iny = uniform(-20, z[1] + 20), t = uniform(0, 6.2832);
                const float fx = (float)(inx + far * std::cos(t)), fy = (float)(iny + far * std::sin(t));
                check((float)inx, (float)iny, fx, fy, reach, z[0], z[1]);             // one end far out
                check((float)(2 * inx - fx), (float)(2 * iny - fy), fx, fy, reach, z[0], z[1]);  // through the image
                check((float)inx, (float)iny, (float)inx, fy, reach, z[0], z[1]);     // along a column
                check(fx, fy, (float)(fx + uniform(-far, far)), (float)(fy + uniform(-far, far)), reach, z[0], z[1]);
            }
    check(-FLT_MAX, -FLT_MAX, FLT_MAX, FLT_MAX, 3, 640, 480);
    check(FLT_MAX, 0.0f, FLT_MAX, 1.0f, 3, 640, 480);
    check(5.0f, 5.0f, 5.0f, 5.0f, 3, 640, 480);
    printf("%lld %lld\n", edges, bad);
    return bad ? 1 : 0;
}
