// spline.cuh -- Bezier subdivision of z2d's Spline.zig on the device,
// shared by the fill flattener (fill.cu) and the stroker (stroke_gpu.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "f64_int.cuh"
#include "fill.cuh"

namespace z2dg {

__host__ __device__ __forceinline__ bool pt_eq(double ax, double ay, double bx, double by) {
    return f64_eq(ax, bx) && f64_eq(ay, by);
}

struct Knots {
    double ax, ay, bx, by, cx, cy, dx, dy;
};

// Spline.Knots.errorSq (Spline.zig:83-123)
__host__ __device__ __forceinline__ double error_sq(const Knots &k) {
    double bx = k.bx - k.ax, by = k.by - k.ay, cx = k.cx - k.ax, cy = k.cy - k.ay;
    if (k.ax != k.dx || k.ay != k.dy) {
        const double dx = k.dx - k.ax, dy = k.dy - k.ay;
        const double dd = dx * dx + dy * dy;
        const double bd = bx * dx + by * dy;
        if (bd >= dd) {
            bx -= dx;
            by -= dy;
        } else {
            bx -= bd / dd * dx;
            by -= bd / dd * dy;
        }
        const double cd = cx * dx + cy * dy;
        if (cd >= dd) {
            cx -= dx;
            cy -= dy;
        } else {
            cx -= cd / dd * dx;
            cy -= cd / dd * dy;
        }
    }
    const double be = bx * bx + by * by, ce = cx * cx + cy * cy;
    return be > ce ? be : ce;
}
// f64 -> f32 by truncating the mantissa (relative error < 2^-23) with
// integer operations only, so that no FP64 instruction is spent on it.
// False outside f32's normal range (zero excepted).
__host__ __device__ __forceinline__ float f32_from(uint32_t b) {
    float f;
    memcpy(&f, &b, 4);
    return f;
}
__host__ __device__ __forceinline__ bool f32_trunc(double v, float &out) {
    const uint64_t b = f64_bits(v);
    const uint32_t hi = (uint32_t)(b >> 32);
    const uint32_t sign = hi & 0x80000000u;
    if ((b << 1) == 0ull) {
        out = f32_from(sign);
        return true;
    }
    const int32_t fe = (int32_t)((hi >> 20) & 0x7FFu) - 1023 + 127;
    if (fe <= 0 || fe >= 255) return false;
    out = f32_from(sign | ((uint32_t)fe << 23) | ((uint32_t)(b >> 29) & 0x7FFFFFu));
    return true;
}

// The decision errorSq(k) < tol2 of Spline.decomposeInto, taken in f32 when
// that is safe.  GB300 runs f64 at a small fraction of its f32 rate, and the
// error test is most of the subdivision's f64 work.  Every f32 quantity
// carries an absolute error bound built from first-order rounding analysis
// with slack: each input's own bound, each operation u (u = 2^-24),
// propagated through the projection and the squared norms.
// Returns 1 / 0 when the f32 value is farther than its bound from tol2 and,
// on the projection branches, from the branch condition; -1 otherwise (the
// caller then evaluates errorSq in f64).
__device__ __forceinline__ int error_sq_lt_f32_core(float bx, float by, float cx, float cy, float ebx, float eby,
                                                    float ecx, float ecy, bool proj, float dx, float dy, float edx,
                                                    float edy, float tol2f, float tol2e) {
    const float U = 5.9604644775390625e-8f;  // 2^-24
    if (proj) {
        const float dd = dx * dx + dy * dy;
        // the inputs' errors carried through the squares, then the roundings
        const float edd = 2.0f * fabsf(dx) * edx + edx * edx + 2.0f * fabsf(dy) * edy + edy * edy + 3.0f * U * dd;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float &px = i ? cx : bx, &py = i ? cy : by;
            float &epx = i ? ecx : ebx, &epy = i ? ecy : eby;
            const float t1 = px * dx, t2 = py * dy;
            const float pd = t1 + t2;
            const float epd = fabsf(dx) * epx + fabsf(px) * edx + epx * edx + fabsf(dy) * epy + fabsf(py) * edy +
                              epy * edy + 2.0f * U * (fabsf(t1) + fabsf(t2));
            const float diff = pd - dd;
            const float m = 1.125f * (epd + edd) + 2.0f * U * fabsf(diff) + 1e-30f;
            if (diff > m) {  // pd >= dd: subtract the whole chord
                const float nx = px - dx, ny = py - dy;
                epx = epx + edx + 2.0f * U * fabsf(nx);
                epy = epy + edy + 2.0f * U * fabsf(ny);
                px = nx;
                py = ny;
            } else if (diff < -m && dd > 0.0f) {  // subtract the projection onto the chord
                const float t = pd / dd;
                const float et = (epd + fabsf(t) * edd) / dd * 1.125f + 2.0f * U * fabsf(t) + 1e-30f;
                const float rx = t * dx, ry = t * dy;
                const float nx = px - rx, ny = py - ry;
                epx = epx + fabsf(dx) * et + fabsf(t) * edx + 2.0f * U * (fabsf(rx) + fabsf(nx));
                epy = epy + fabsf(dy) * et + fabsf(t) * edy + 2.0f * U * (fabsf(ry) + fabsf(ny));
                px = nx;
                py = ny;
            } else {
                return -1;
            }
        }
    }
    const float be = bx * bx + by * by, ce = cx * cx + cy * cy;
    const float ebe = 2.0f * fabsf(bx) * ebx + 2.0f * fabsf(by) * eby + ebx * ebx + eby * eby + 4.0f * U * be;
    const float ece = 2.0f * fabsf(cx) * ecx + 2.0f * fabsf(cy) * ecy + ecx * ecx + ecy * ecy + 4.0f * U * ce;
    const float e = be > ce ? be : ce;
    const float E = 1.25f * (ebe > ece ? ebe : ece) + 4.0f * U * e + 1e-30f + tol2e;
    if (!(E < 1e30f)) return -1;
    if (e + E < tol2f) return 1;
    if (e - E > tol2f) return 0;
    return -1;
}
// From the exact f64 differences b - a, c - a, d - a (truncation error < 2u
// of each).
__device__ __forceinline__ int error_sq_lt_f32(double bx64, double by64, double cx64, double cy64, bool proj,
                                               double dx64, double dy64, float tol2f, float tol2e) {
    const float U = 5.9604644775390625e-8f;  // 2^-24
    float bx, by, cx, cy, dx = 0.0f, dy = 0.0f;
    if (!f32_trunc(bx64, bx) || !f32_trunc(by64, by) || !f32_trunc(cx64, cx) || !f32_trunc(cy64, cy)) return -1;
    if (proj && (!f32_trunc(dx64, dx) || !f32_trunc(dy64, dy))) return -1;
    return error_sq_lt_f32_core(bx, by, cx, cy, 2.0f * U * fabsf(bx), 2.0f * U * fabsf(by), 2.0f * U * fabsf(cx),
                                2.0f * U * fabsf(cy), proj, dx, dy, 2.0f * U * fabsf(dx), 2.0f * U * fabsf(dy), tol2f,
                                tol2e);
}
// From the knots' coordinates, truncated to f32 (error < 2u of each) and
// subtracted in f32 (one more rounding): no f64 instruction at all, at the
// price of wider bounds (the coordinates' size instead of the differences').
// Serves the curves whose coordinates do not take chord_test's fixed point.
__device__ __forceinline__ int error_sq_lt_f32_pts(double ax64, double ay64, double bx64, double by64, double cx64,
                                                   double cy64, double dx64, double dy64, bool proj, float tol2f,
                                                   float tol2e) {
    const float U = 5.9604644775390625e-8f;  // 2^-24
    float ax, ay, pbx, pby, pcx, pcy, pdx = 0.0f, pdy = 0.0f;
    if (!f32_trunc(ax64, ax) || !f32_trunc(ay64, ay) || !f32_trunc(bx64, pbx) || !f32_trunc(by64, pby) ||
        !f32_trunc(cx64, pcx) || !f32_trunc(cy64, pcy))
        return -1;
    if (proj && (!f32_trunc(dx64, pdx) || !f32_trunc(dy64, pdy))) return -1;
    const float bx = pbx - ax, by = pby - ay, cx = pcx - ax, cy = pcy - ay, dx = pdx - ax, dy = pdy - ay;
    const float eax = 2.0f * U * fabsf(ax), eay = 2.0f * U * fabsf(ay);
    return error_sq_lt_f32_core(bx, by, cx, cy, eax + 2.0f * U * fabsf(pbx) + U * fabsf(bx),
                                eay + 2.0f * U * fabsf(pby) + U * fabsf(by), eax + 2.0f * U * fabsf(pcx) + U * fabsf(cx),
                                eay + 2.0f * U * fabsf(pcy) + U * fabsf(cy), proj, dx, dy,
                                eax + 2.0f * U * fabsf(pdx) + U * fabsf(dx), eay + 2.0f * U * fabsf(pdy) + U * fabsf(dy),
                                tol2f, tol2e);
}

// The squared tolerance of a subdivision, in f64, as a truncated f32 with its
// error bound, and as a bracket in the curve's fixed-point units (chord_test).
struct Tol {
    double d;
    float f, e;
    bool f_ok;
    float lo, hi;
    uint32_t shift0;
};

__host__ __device__ __forceinline__ Tol make_tol(double tol) {
    Tol t;
    t.d = tol * tol;  // decomposeInto's tolerance argument (Spline.zig:52)
    t.f = 0.0f;
    t.f_ok = f32_trunc(t.d, t.f);
    t.e = 4.0f * 5.9604644775390625e-8f * t.f;
    t.lo = -1.0f;  // the bracket that decides nothing
    t.hi = f32_from(0x7F800000u);
    t.shift0 = 0;
    return t;
}
// One curve's tolerance.  The fixed-point unit is 2^-29 of the power of two
// at or below the curve's largest coordinate, so that every coordinate of
// the curve and of its subcurves (a split's points lie between their ends,
// each coordinate) takes 31 bits with the sign.
__host__ __device__ __forceinline__ Tol make_tol(double tol, const Knots &k) {
    Tol t = make_tol(tol);
    uint32_t m = 0;
    const double c[8] = {k.ax, k.ay, k.bx, k.by, k.cx, k.cy, k.dx, k.dy};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t h = (uint32_t)(f64_bits(c[i]) >> 32) & 0x7FFFFFFFu;
        m = m > h ? m : h;
    }
    const uint32_t e = m >> 20;
    t.shift0 = e + 2;
    if (t.f_ok && e >= 1023 - 40 && e <= 1023 + 40) {
        const float unit = f32_from((127u + 1052u - e) << 23);  // units per 1
        const float u2 = (t.f * unit) * unit;
        if (u2 > 1e-18f && u2 < 1e18f) {
            t.lo = u2 * (1.0f - 3.814697265625e-6f);  // -+ 2^-18
            t.hi = u2 * (1.0f + 3.814697265625e-6f);
        }
    }
    return t;
}

// floor-like fixed point of one coordinate: within one unit below x (the
// magnitude truncated, its bits inverted where x is negative).
__host__ __device__ __forceinline__ int32_t to_fixed(double x, uint32_t shift0) {
    const uint64_t b = f64_bits(x);
    const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
    const uint32_t sh = shift0 - ((hi >> 20) & 0x7FFu);
#ifdef __CUDA_ARCH__
    const uint32_t m = __funnelshift_l(lo, hi, 11) | 0x80000000u;
    const uint32_t q = __funnelshift_rc(m, 0u, sh);
#else
    const uint32_t m = (hi << 11) | (lo >> 21) | 0x80000000u;
    const uint32_t q = sh >= 32u ? 0u : m >> sh;
#endif
    return (int32_t)q ^ ((int32_t)hi >> 31);
}

// errorSq(k) < tol2 from fixed-point coordinates: 1 / 0 where the error
// bounds allow the decision, -1 otherwise.  The differences are exact integers
// within one unit of the true ones; f32 takes over from there.  With d the
// chord, a control point p (from a) that projects before d's end is at
// squared distance cross(p, d)^2 / |d|^2, and the comparison with tol2 needs
// no division; past the end it is |p - d|^2.
//
// Bounds: an input (a difference, at most L in size) is off by at most
// 1 + uL, u = 2^-24; K = 1 + 4uL covers it and, by K times the other
// factor, the roundings of a product.  A sum of two products of p and d is
// then within K (P + 2 S) + 2 K^2 of its true value, with P = |px| + |py|
// and S = |dx| + |dy|; the bounds below have 6 % on top of that for their own
// roundings, and the tolerance's bracket (2^-18) covers the relative
// roundings of the squares and products that are compared.
//
// f32 copies of the coordinates, subtracted, left 1.8 % of the tests on a
// 4096-pixel canvas to the f64 differences, which one warp in two then
// waited for; a unit is 64 times finer than their last place, and leaves
// 0.03 %.
__host__ __device__ __forceinline__ int chord_test(const Knots &k, const Tol &t) {
    const uint32_t s0 = t.shift0;
    const int32_t ax = to_fixed(k.ax, s0), ay = to_fixed(k.ay, s0);
    const float dx = (float)(to_fixed(k.dx, s0) - ax), dy = (float)(to_fixed(k.dy, s0) - ay);
    const float p[2][2] = {{(float)(to_fixed(k.bx, s0) - ax), (float)(to_fixed(k.by, s0) - ay)},
                           {(float)(to_fixed(k.cx, s0) - ax), (float)(to_fixed(k.cy, s0) - ay)}};
    const float L = fmaxf(fmaxf(fmaxf(fabsf(p[0][0]), fabsf(p[0][1])), fmaxf(fabsf(p[1][0]), fabsf(p[1][1]))),
                          fmaxf(fabsf(dx), fabsf(dy)));
    const float K = 1.0f + 2.384185791015625e-7f * L;  // 1 + 4 u L
    const float S = fabsf(dx) + fabsf(dy);
    const float dd = dx * dx + dy * dy, m_dd = 2.125f * K * (S + K);
    const float dd_lo = dd - m_dd, dd_hi = dd + m_dd;
    if (!(dd_lo > 0.0f)) return -1;
    bool below = true, above = false;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float px = p[i][0], py = p[i][1];
        const float P = fabsf(px) + fabsf(py);
        const float m = 1.0625f * K * (P + 2.0f * S + 2.0f * K);
        const float diff = (px * dx + py * dy) - dd;
        if (diff < -(m + m_dd)) {
            const float c = fabsf(px * dy - py * dx);
            const float lo = fmaxf(c - m, 0.0f), hi = c + m;
            below = below && hi * hi < t.lo * dd_lo;
            above = above || lo * lo > t.hi * dd_hi;
        } else if (diff > m + m_dd) {
            const float vx = px - dx, vy = py - dy;
            const float n = vx * vx + vy * vy, mn = 4.25f * K * (fabsf(vx) + fabsf(vy) + 2.125f * K);
            below = below && n + mn < t.lo;
            above = above || n - mn > t.hi;
        } else {
            return -1;
        }
    }
    return above ? 0 : below ? 1 : -1;
}

// errorSq(k) < t.d, exactly as the f64 comparison decides it.
// The rarely needed tests, out of line so that the subdivision loops stay
// small in the instruction cache.
static __device__ __noinline__ bool below_tol_slow(Knots k, Tol t) {
    if (t.f_ok) {
        const bool proj = !pt_eq(k.ax, k.ay, k.dx, k.dy);
        int r = -1;
        if (t.lo < 0.0f) r = error_sq_lt_f32_pts(k.ax, k.ay, k.bx, k.by, k.cx, k.cy, k.dx, k.dy, proj, t.f, t.e);
        if (r < 0)
            r = error_sq_lt_f32(k.bx - k.ax, k.by - k.ay, k.cx - k.ax, k.cy - k.ay, proj, k.dx - k.ax, k.dy - k.ay, t.f,
                                t.e);
        if (r >= 0) return r != 0;
    }
    return error_sq(k) < t.d;
}

// Out of line, like the split: the subdivision loops stay small in the
// instruction cache and the curve kernels need 96 registers instead of
// 118-124 (flatten of the 2,000-path batch 0.68 -> 0.59 ms).  The
// fixed-point test took the count of that batch from 285 to 185 us.
static __device__ __noinline__ bool below_tol(const Knots &k, const Tol &t) {
    const int r = chord_test(k, t);
    if (r >= 0) return r != 0;
    return below_tol_slow(k, t);
}

// x / 2.  For normal x whose half is normal this only lowers the exponent,
// which integer operations do exactly (an f64 multiply is an expensive
// instruction on GB300); zeros, subnormals and non-finite values divide.
__device__ __forceinline__ double half_of(double x) {
    const long long b = __double_as_longlong(x);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7FFu;
    if (e > 1u && e < 0x7FFu) return __longlong_as_double(b - (1ll << 52));
    return x / 2;
}
// The f64 form, out of line so that it runs only on the lanes that need it.
static __device__ __noinline__ double lerp_half_f64(double a, double b) { return a + half_of(b - a); }
__device__ __forceinline__ double lerp_half(double a, double b) {
    bool done;
    const double r = lerp_half_int(a, b, done);
    if (done) return r;
    return lerp_half_f64(a, b);
}

// Knots.deCasteljau (Spline.zig:128-152): k becomes the first half, the
// second half is returned.  Out of line: one copy serves the descent to a
// lane's subtree and the depth-first walks (flatten of the 2,000-path batch
// 0.72 -> 0.68 ms against the inlined copies).
static __device__ __noinline__ Knots de_casteljau(Knots &k) {
    const double abx = lerp_half(k.ax, k.bx), aby = lerp_half(k.ay, k.by);
    const double bcx = lerp_half(k.bx, k.cx), bcy = lerp_half(k.by, k.cy);
    const double cdx = lerp_half(k.cx, k.dx), cdy = lerp_half(k.cy, k.dy);
    const double abbcx = lerp_half(abx, bcx), abbcy = lerp_half(aby, bcy);
    const double bccdx = lerp_half(bcx, cdx), bccdy = lerp_half(bcy, cdy);
    const double fx = lerp_half(abbcx, bccdx), fy = lerp_half(abbcy, bccdy);
    const Knots r{fx, fy, bccdx, bccdy, cdx, cdy, k.dx, k.dy};
    k.bx = abx; k.by = aby;
    k.cx = abbcx; k.cy = abbcy;
    k.dx = fx; k.dy = fy;
    return r;
}

// Depth-first walk of a subtree (Spline.decomposeInto, Spline.zig:56-71)
// with an explicit stack: leaf(k) for every subcurve that decomposeInto stops
// at, in order.  `open` counts the pending second halves above the subtree,
// so the stack bound is the whole curve's.  False if the stack would overflow
// (coordinates are bounded, so this does not happen for valid input) or the
// subtree does not end within kSplineMaxSplits tests.
template <class L>
__device__ __forceinline__ bool walk_leaves(const Knots &k0, bool is_leaf, int open, const Tol &tol, L &&leaf) {
    if (is_leaf) {
        leaf(k0);
        return true;
    }
    Knots stack[kSplineStack];
    int sp = 0;
    int32_t budget = kSplineMaxSplits;  // bounds the walk even for pathological input
    Knots k = k0;
    while (true) {
        if (--budget < 0) return false;
        if (below_tol(k, tol)) {
            leaf(k);
            if (sp == 0) return true;
            k = stack[--sp];
            continue;
        }
        if (sp + open >= kSplineStack) return false;  // cannot recurse deeper
        stack[sp++] = de_casteljau(k);                 // processed after the first half
    }
}

// A curve's subdivision tree shared by 2^g neighbouring lanes: lane j
// walks the subtree that the bits of j lead to (first level in the highest
// bit, 0 for the first half), so the lanes' leaves, lane after lane, are the
// curve's in order.  A leaf above level g belongs to the lane whose
// remaining bits are 0.  Each lane goes down from the root by itself (g tests
// and splits, without shared memory or exchange), which costs less than
// one leaf per level.
__device__ __forceinline__ bool lane_subtree(Knots &k, int g, int j, const Tol &tol, bool &is_leaf, int &open) {
    is_leaf = false;
    open = 0;
    for (int l = g - 1; l >= 0; l--) {
        if (below_tol(k, tol)) {
            is_leaf = true;
            return (j & ((2 << l) - 1)) == 0;
        }
        const Knots second = de_casteljau(k);
        if ((j >> l) & 1) k = second;
        else open++;
    }
    return true;
}

// A curve's length class, from a rough count of its leaves: halving divides
// the second differences a - 2b + c and b - 2c + d by 4, so about
// 2^k = (|second difference| / tolerance)^(1/2) leaves are left.  Class 0 is
// k <= 3, then one class per k, class 5 k >= 8.
constexpr int kCurveClasses = 6;
__device__ __forceinline__ int curve_class(double ax, double ay, const double *p, double tol) {
    float x[4], y[4], t;
    bool ok = f32_trunc(ax, x[0]) && f32_trunc(ay, y[0]) && f32_trunc(tol, t);
#pragma unroll
    for (int i = 0; i < 3; i++) ok = ok && f32_trunc(p[2 * i], x[i + 1]) && f32_trunc(p[2 * i + 1], y[i + 1]);
    if (!ok) return kCurveClasses - 1;
    const float x1 = x[0] - 2.0f * x[1] + x[2], y1 = y[0] - 2.0f * y[1] + y[2];
    const float x2 = x[1] - 2.0f * x[2] + x[3], y2 = y[1] - 2.0f * y[2] + y[3];
    const float d = fmaxf(x1 * x1 + y1 * y1, x2 * x2 + y2 * y2);
    float bound = 4096.0f * (t * t);  // 16^3 t^2
    int c = 0;
    for (; c < kCurveClasses - 1 && !(d <= bound); c++) bound *= 16.0f;
    return c;
}

// Depth-first subdivision of one curve by one thread.  Calls emit(x, y) for
// every lineTo the reference issues, including the final lineTo(d).
template <class F>
__device__ __forceinline__ bool spline_walk(double ax, double ay, const double *p, double tol, F &&emit) {
    const double bx = p[0], by = p[1], cx = p[2], cy = p[3], dx = p[4], dy = p[5];
    if (pt_eq(ax, ay, bx, by) && pt_eq(cx, cy, dx, dy)) {  // Spline.zig:39-42
        emit(dx, dy);
        return true;
    }
    const Knots k0{ax, ay, bx, by, cx, cy, dx, dy};
    const bool ok = walk_leaves(k0, false, 0, make_tol(tol, k0), [&](const Knots &k) {
        if (!pt_eq(k.ax, k.ay, ax, ay)) emit(k.ax, k.ay);
    });
    emit(dx, dy);
    return ok;
}

}  // namespace z2dg
