// Host check of the subdivision's fixed-point error test (spline.cuh):
// wherever chord_test decides, it is errorSq(k) < tolerance^2 in f64.
// Curves of all sizes and places, their subcurves down to the leaves, and
// knots set on the tolerance's edge, with degenerate chords and control
// points at the chord's ends.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "spline.cuh"

using namespace z2dg;

static long long tests = 0, decided = 0, wrong = 0;

static bool check(const Knots &k, const Tol &t) {
    const bool exact = error_sq(k) < t.d;
    const int r = chord_test(k, t);
    tests++;
    if (r >= 0) {
        decided++;
        if ((r != 0) != exact) wrong++;
    }
    return exact;
}

static double half(double a, double b) { return a + (b - a) / 2; }

static void split(Knots k, const Tol &t, int depth) {
    if (check(k, t) || depth == 0) return;
    const double abx = half(k.ax, k.bx), aby = half(k.ay, k.by), bcx = half(k.bx, k.cx), bcy = half(k.by, k.cy);
    const double cdx = half(k.cx, k.dx), cdy = half(k.cy, k.dy), ex = half(abx, bcx), ey = half(aby, bcy);
    const double gx = half(bcx, cdx), gy = half(bcy, cdy), fx = half(ex, gx), fy = half(ey, gy);
    split(Knots{k.ax, k.ay, abx, aby, ex, ey, fx, fy}, t, depth - 1);
    split(Knots{fx, fy, gx, gy, cdx, cdy, k.dx, k.dy}, t, depth - 1);
}

int main(int argc, char **argv) {
    const long n = argc > 1 ? atol(argv[1]) : 60000;
    std::mt19937_64 rng(11);
    auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); };
    for (long i = 0; i < n; i++) {
        const double size = std::exp(uni(-5.0, 9.0)), far = std::exp(uni(-3.0, 17.0)), tol = std::exp(uni(-6.0, 1.0));
        const double ox = uni(-far, far), oy = uni(-far, far);
        auto at = [&](double o) { return o + uni(-size, size); };
        Knots k{at(ox), at(oy), at(ox), at(oy), at(ox), at(oy), at(ox), at(oy)};
        const int kind = (int)(rng() % 8);
        if (kind == 1) k.dx = k.ax, k.dy = k.ay;
        if (kind == 2) k.dx = k.ax, k.dy = std::nextafter(k.ay, 1e9);
        if (kind == 3) k.bx = k.dx, k.by = k.dy;
        if (kind == 4) k.ax = 0.0, k.by = -0.0, k.cx = 1e-310, k.cy = -1e-40;
        split(k, make_tol(tol, k), 9);
        // control points at the tolerance from the chord, or from its end
        const double cx = k.dx - k.ax, cy = k.dy - k.ay, len = std::sqrt(cx * cx + cy * cy);
        if (!(len > 0)) continue;
        for (int j = 0; j < 16; j++) {
            const double f = (j & 1) ? uni(-0.5, 1.0) : uni(0.98, 1.02), e = tol * (1.0 + uni(-1.0, 1.0) * std::exp(uni(-30.0, -2.0)));
            Knots q = k;
            q.bx = k.ax + f * cx - e * cy / len;
            q.by = k.ay + f * cy + e * cx / len;
            if (j & 2) q.cx = half(k.ax, k.dx), q.cy = half(k.ay, k.dy);
            else q.cx = k.dx + e * cx / len, q.cy = k.dy + e * cy / len;
            check(q, make_tol(tol, q));
        }
    }
    printf("tests %lld decided %.5f wrong %lld\n", tests, (double)decided / (double)tests, wrong);
    return wrong ? 1 : 0;
}
