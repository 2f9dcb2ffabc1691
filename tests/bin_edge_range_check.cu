// Host check of the bins' edge records (raster.cuh) at the ends of the sample
// rows' range: an edge that reaches beyond 2^31 sample rows has its range
// saturated there, and a record's rows are still those with rt <= sr < rb.
// Where the edge's other fields fit f32, a decided crossing is the rounded f64
// value however far below the edge's first row the band lies.  Built with the
// undefined behaviour sanitizer: the subtractions must not overflow.
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "raster.cuh"

using namespace z2dg;

int main() {
    const int32_t lo = INT32_MIN, hi = INT32_MAX;
    const int32_t ends[] = {lo, lo + 1, lo + 100, -(1 << 26), -17, -1, 0, 1, 3, 16, 1000, 1 << 26, hi - 100, hi - 1, hi};
    const int32_t rows[] = {0, 4, 16, 992, 1 << 20, 1 << 26, 1 << 30, hi - 127, hi - 31, hi - 15};
    long long wrong = 0, decided = 0, tests = 0;
    for (int32_t rt : ends)
        for (int32_t rb : ends)
            for (int32_t row : rows)
                for (int32_t n : {kTileRows, 4 * kTileRows}) {
                    if (rt >= rb) continue;
                    for (bool down : {false, true}) {
                        DEdge e{};
                        e.top = (double)rt + 0.25;  // round(top) = rt
                        e.x_start = 100.25;
                        e.x_inc = 1e-6;
                        if (!edge_fields(e, down)) e.rt = rt;
                        const BinEdge B = bin_edge(e.xi, e.fx, e.fxi, e.fdt, rt, rb, 7, row, n);
                        tests++;
                        if (e.rt != rt || ((int32_t)B.rows < 0) != down || B.id != 7) wrong++;
                        for (int32_t s = 0; s < n; s++) {
                            const int64_t sr = (int64_t)row + s;
                            const bool active = sr >= rt && sr < rb;
                            if ((((B.rows >> s) & 1u) != 0) != active) wrong++;
                            int32_t m;
                            const float v0 = fmaf(B.fxi, B.t + (float)(s & ~3), B.fx);
                            if (!active || !crossing_f32(v0, B.fxi, (float)(s & 3), B.limit, m)) continue;
                            decided++;
                            const double x = e.x_start + e.x_inc * (((double)sr + 0.5) - e.top);
                            if ((double)m + (double)B.c != std::round(x)) wrong++;
                        }
                    }
                }
    printf("records %lld decided %lld wrong %lld\n", tests, decided, wrong);
    return wrong == 0 && decided > 0 ? 0 : 1;
}
