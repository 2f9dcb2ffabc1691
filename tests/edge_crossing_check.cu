// Host check of the f32 crossings (fill.cuh): wherever crossing_f32 decides,
// xi + its integer is round(x_start + x_inc * ((sr + 0.5) - top)) in f64.
// Random edges (short and long, steep and flat, on and around half-integer
// crossings, negative and large coordinates), every active sample row of the
// short ones and 64 of the long ones.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "fill.cuh"

using namespace z2dg;

int main(int argc, char **argv) {
    const long n = argc > 1 ? atol(argv[1]) : 2000000;
    std::mt19937_64 rng(7);
    auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); };
    long long rows = 0, decided = 0, wrong = 0, bad_fields = 0;
    for (long i = 0; i < n; i++) {
        const double size = std::exp(uni(-3.0, 10.0)), far = std::exp(uni(0.0, 18.5));
        double ax = uni(-far, far), ay = uni(-far, far), bx = ax + uni(-size, size), by = ay + uni(-size, size);
        const int kind = (int)(rng() % 5);
        auto snap = [](double v, double g) { return std::round(v * g) / g; };
        if (kind == 1) ax = snap(ax, 2), bx = snap(bx, 2), ay = snap(ay, 2), by = snap(by, 2);
        if (kind == 2) ax = snap(ax, 8), bx = snap(bx, 8), ay = snap(ay, 8), by = snap(by, 8);
        if (kind == 3) ay = snap(ay, 1) + 0.5, by = snap(by, 1) + 0.5;
        if (kind == 4) bx = ax;
        if (ay == by) continue;
        DEdge e{};
        const bool down = ay < by;
        e.top = down ? ay : by;
        e.x_start = down ? ax : bx;
        e.x_inc = down ? (bx - ax) / (by - ay) : (ax - bx) / (ay - by);
        if (!edge_fields(e, down)) e.rt = (int32_t)std::round(e.top);
        e.rb = (int32_t)std::round(down ? by : ay);
        if (e.rt != (int32_t)std::round(e.top) || edge_dir(e) != (down ? -1 : 1)) bad_fields++;
        const int32_t step = std::max(1, (e.rb - e.rt) / 64);
        for (int32_t sr = e.rt; sr < e.rb; sr += step) {
            // as the rasteriser asks: a pixel row of 4 sample rows
            const int32_t sub0 = sr & ~3, hi = std::min(e.rb - sub0, 4), rel = sub0 - e.rt;
            const float t = ((float)rel + (float)(sr - sub0)) + fabsf(e.fdt);
            const float limit = crossing_limit(e.fxi, (float)(rel + hi));
            int32_t v;
            rows++;
            if (!crossing_f32(e.fx, e.fxi, t, limit, v)) continue;
            decided++;
            const int32_t X = (int32_t)std::round(e.x_start + (e.x_inc * (((double)sr + 0.5) - e.top)));
            if (e.xi + (v - kRoundMagicBits) != X) wrong++;
        }
    }
    printf("rows %lld decided %lld wrong %lld bad_fields %lld\n", rows, decided, wrong, bad_fields);
    return wrong == 0 && bad_fields == 0 && decided * 10 > rows * 9 ? 0 : 1;
}
