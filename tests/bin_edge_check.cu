// Host check of the bins' edge records (raster.cuh): for every band of 16 (or
// 4) sample rows that an edge touches, the record's rows are those on which
// the edge is active, and wherever crossing_f32 decides a row from the
// record as a pixel row of the band evaluates it, xi plus its integer is
// round(x_start + x_inc * ((sr + 0.5) - top)) in f64.  Random edges (short and
// long, steep and flat, on and around half-integer crossings, negative and
// large coordinates), with every band of the short ones and some 64 of the long.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "raster.cuh"

using namespace z2dg;

int main(int argc, char **argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    std::mt19937_64 rng(23);
    auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); };
    long long rows = 0, decided = 0, wrong = 0;
    for (long i = 0; i < n; i++) {
        const double size = std::exp(uni(-3.0, 10.0)), far = std::exp(uni(0.0, 18.5));
        double ax = uni(-far, far), ay = uni(-far, far), bx = ax + uni(-size, size), by = ay + uni(-size, size);
        const int kind = (int)(rng() % 5), sc = (rng() & 1) ? 4 : 1;
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
        const int32_t band = kTileRows * sc;
        const int32_t b0 = (int32_t)std::floor((double)e.rt / band), b1 = (int32_t)std::floor((double)(e.rb - 1) / band);
        const int32_t step = std::max(1, (b1 - b0) / 64);
        for (int32_t b = b0; b <= b1; b += step) {
            const int32_t row = b * band;
            const BinEdge B = bin_edge(e.xi, e.fx, e.fxi, e.fdt, e.rt, e.rb, 0, row, band);
            if (((int32_t)B.rows < 0) != down) wrong++;
            for (int32_t s = 0; s < band; s++) {
                const int32_t sr = row + s, off = s / sc * sc;
                if ((((B.rows >> s) & 1u) != 0) != (sr >= e.rt && sr < e.rb)) wrong++;
                if (sr < e.rt || sr >= e.rb) continue;
                rows++;
                int32_t m;
                const float v0 = fmaf(B.fxi, B.t + (float)off, B.fx);
                if (!crossing_f32(v0, B.fxi, (float)(s - off), B.limit, m)) continue;
                decided++;
                const double x = e.x_start + e.x_inc * (((double)sr + 0.5) - e.top);
                if ((double)m + (double)B.c != std::round(x)) wrong++;
            }
        }
    }
    printf("rows %lld decided %.6f wrong %lld\n", rows, (double)decided / (double)rows, wrong);
    return wrong ? 1 : 0;
}
