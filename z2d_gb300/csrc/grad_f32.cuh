// grad_f32.cuh -- a gradient pixel's integer colour lanes in plain f32,
// exact where it says so.
//
// The lanes are bytes: round(255 c) of every channel of the interpolated
// colour c (enc_ch), then integer premultiplication.  The offset, the
// interpolation, the sRGB gamma and the dither are evaluated in f32 here,
// together with a bound on the distance of every channel from the value of
// the reference's evaluation (f64 offset rounded to f32, then f32
// operations, std.math.pow for the gamma).  A channel whose 255 c stays
// farther than its bound from every half-integer rounds to the same byte, so
// the lanes are the reference's; a pixel with another channel, and what is
// not covered (stop tables beyond the descriptor, an offset within its bound of
// a stop, alpha near 0), takes the double-word offset and the
// exact colour code.  That is 0.1 % of the pixels (linear RGB) to 1.4 % (HSL
// with a dither) of 3840x2160 gradients of every kind.
// Every bound is the first-order rounding analysis with slack: u = 2^-24,
// each input's own bound, each operation u.
//
// What it saves: the double-word offset of a radial gradient is about 500
// instructions and std.math.pow about 200 per channel, against about 60 and
// 10 here.
#pragma once

namespace z2dg {

constexpr float kU = 0x1p-24f;

// An offset t within e of the reference's; `ok` 0: not decided, 1: t,
// 2: the invalid offset -1.
struct OffsetF32 {
    float t, e;
    int ok;
};

// The pixel centre after the inverse transformation, relative to the
// gradient's first point, with its bounds.
__device__ __forceinline__ void point_f32(const GradFast &F, bool has_tf, float fx, float fy, float &dx, float &dy,
                                          float &ex, float &ey) {
    if (has_tf) {
        const float px = __fmaf_rn(F.tf[0].h, fx, __fmaf_rn(F.tf[1].h, fy, F.tf[4].h));
        const float py = __fmaf_rn(F.tf[2].h, fx, __fmaf_rn(F.tf[3].h, fy, F.tf[5].h));
        dx = px - F.g0.h;
        dy = py - F.g1.h;
        ex = 6.0f * kU * (fabsf(F.tf[0].h * fx) + fabsf(F.tf[1].h * fy) + fabsf(F.tf[4].h) + fabsf(F.g0.h));
        ey = 6.0f * kU * (fabsf(F.tf[2].h * fx) + fabsf(F.tf[3].h * fy) + fabsf(F.tf[5].h) + fabsf(F.g1.h));
    } else {
        // the centre is exact, and so is the difference's rounding error:
        // what is left is the last sum's
        const DW d = two_sum(fx, -F.g0.h), e = two_sum(fy, -F.g1.h);
        dx = d.h + (d.l - F.g0.l);
        dy = e.h + (e.l - F.g1.l);
        ex = kU * fabsf(dx) + 0x1p-46f * fabsf(F.g0.h);
        ey = kU * fabsf(dy) + 0x1p-46f * fabsf(F.g1.h);
    }
}

__device__ __forceinline__ OffsetF32 offset_f32(int kind, const GradFast &F, bool has_tf, float fx, float fy) {
    float dx, dy, ex, ey;
    point_f32(F, has_tf, fx, fy, dx, dy, ex, ey);
    if (kind == Z2D_GRADIENT_LINEAR) {
        // k0, k1: split and product round once each; the sum is one fused step
        const float k0 = F.k[0].h, k1 = F.k[1].h, k2 = F.k[2].h;
        const float b = k1 * dy, q = __fmaf_rn(k0, dx, b) * k2;
        const float es = fabsf(k0) * ex + fabsf(k1) * ey + kU * (fabsf(k0 * dx) + 2.0f * fabsf(b));
        return OffsetF32{fminf(fmaxf(q, 0.0f), 1.0f), es * fabsf(k2) + 3.5f * kU * fabsf(q), 1};
    }
    if (kind == Z2D_GRADIENT_RADIAL) {
        const float cdx = F.k[0].h, cdy = F.k[1].h, ir_dr = F.k[2].h, nir2 = F.k[3].h, a = F.k[4].h, inv_a = F.k[5].h;
        const float dr = F.k[6].h, min_dr = F.k[7].h;
        const float b1 = __fmaf_rn(dy, cdy, ir_dr), b = __fmaf_rn(dx, cdx, b1);
        const float eb = fabsf(cdx) * ex + fabsf(cdy) * ey +
                         kU * (fabsf(dx * cdx) + fabsf(dy * cdy) + fabsf(ir_dr) + fabsf(b1) + fabsf(b));
        const float c1 = __fmaf_rn(dy, dy, nir2), c = __fmaf_rn(dx, dx, c1);
        const float ec = 2.0f * (fabsf(dx) * ex + fabsf(dy) * ey) + kU * (fabsf(nir2) + fabsf(c1) + fabsf(c));
        const float ac = a * c, disc = __fmaf_rn(b, b, -ac);
        const float ed = 2.0f * fabsf(b) * eb + eb * eb + fabsf(a) * ec + kU * (2.0f * fabsf(ac) + fabsf(disc)) + 1e-30f;
        if (!(disc > 4.0f * ed)) return OffsetF32{0.0f, 0.0f, disc < -4.0f * ed ? 2 : 0};
        // one Newton step on disc * rsqrt(disc); for disc' within ed the
        // root moves by at most ed / (2 sqrt(3 disc / 4)) < 0.6 ed / sqrt(disc)
        const float r = rsqrtf(disc), s0 = disc * r, sq = __fmaf_rn(__fmaf_rn(-s0, s0, disc), 0.5f * r, s0);
        const float e_lin = (eb + 0.6f * ed * r + kU * (2.0f * sq + 3.5f * (fabsf(b) + sq))) * fabsf(inv_a);
        const float t0 = (b + sq) * inv_a;
        const float d0 = t0 * dr - min_dr, m = 4.0f * kU * fabsf(min_dr);
        if (!(fabsf(d0) > e_lin * fabsf(dr) + 4.0f * kU * fabsf(t0 * dr) + m)) return OffsetF32{0.0f, 0.0f, 0};
        if (d0 > 0.0f) return OffsetF32{fminf(fmaxf(t0, 0.0f), 1.0f), e_lin, 1};
        const float t1 = (b - sq) * inv_a, d1 = t1 * dr - min_dr;
        if (!(fabsf(d1) > e_lin * fabsf(dr) + 4.0f * kU * fabsf(t1 * dr) + m)) return OffsetF32{0.0f, 0.0f, 0};
        return OffsetF32{fminf(fmaxf(t1, 0.0f), 1.0f), e_lin, d1 > 0.0f ? 1 : 2};
    }
    // conic: atan2f is within 3 ulp (of at most pi: 2^-20.4); the inputs'
    // relative errors move the angle by at most (ex |dy| + ey |dx|) / r^2
    const float r2 = dx * dx + dy * dy;
    if (!(r2 > 1e-20f) || !(r2 < 1e20f) || !(ex + ey < 0.01f * fmaxf(fabsf(dx), fabsf(dy))))
        return OffsetF32{0.0f, 0.0f, 0};
    const float th = atan2f(dy, dx);
    const float ea = 1.01f * __fdividef(ex * fabsf(dy) + ey * fabsf(dx), r2) + 0x1p-20f;
    // off the branch cut, where the angle jumps by 2 pi
    if (dx < 0.0f && !(fabsf(dy) > 2.0f * ey)) return OffsetF32{0.0f, 0.0f, 0};
    const float v = th - F.k[0].h, inv = kDwInvTwoPi.h;
    const float ev = ea + 3.0f * kU * (fabsf(th) + fabsf(F.k[0].h));
    float t = v * inv;
    t -= floorf(t);
    const float e = ev * inv + 2.0f * kU * (1.0f + fabsf(v * inv));
    // off the wrap, where the offset jumps between 0 and 1
    if (!(t > 2.0f * e && t < 1.0f - 2.0f * e)) return OffsetF32{0.0f, 0.0f, 0};
    return OffsetF32{t, e, 1};
}

// x^2.2 within kGammaErr of std.math.pow(x, 2.2) on [0, 1.001]: every float
// of the range compared, the largest difference is 3.6e-7
// (tests/gamma_device_check.cu).
constexpr float kGammaErr = 4.5e-7f;
__device__ __forceinline__ float gamma_f32(float x) { return exp2f(kGamma * __log2f(x)); }

// round(255 c) for a c known within e, as enc_ch rounds it; `ok` is cleared
// where e does not decide it (and for NaN).
__device__ __forceinline__ uint32_t enc_f32(float c, float e, bool &ok) {
    const float v = 255.0f * c, m = v + 12582912.0f;  // 1.5 * 2^23: rounds to an integer
    ok = ok && fabsf(v - (m - 12582912.0f)) < 0.5f - (255.0f * e + 512.0f * kU);
    return (uint32_t)(__float_as_int(m) - 0x4B400000);
}

// Dither.getPixel's amplitude for a target of `scale` bits.
__device__ __forceinline__ float dither_step_of(int scale) { return 1.0f / (float)((1 << scale) - 1); }

// The colour lanes for the offset o; false where f32 does not decide them.
__device__ __forceinline__ bool color_f32(int method, int dither, float dither_step, const DevGradient &g, OffsetF32 o,
                                          int32_t x, int32_t y, I16 &out) {
    const int n = g.n_stops;
    if (o.ok != 1 || n == 0 || n > kMaxStops) {
        out = I16{0u, 0u, 0u, 0u};
        return o.ok == 2 && dither == Z2D_DITHER_NONE;  // transparent
    }
    const float e = o.e + 2.0f * kU;  // with the reference's rounding to f32
    int i = 0;                        // stops at or below t
    while (i < n && o.t >= g.offsets[i]) i++;
    // The colour is constant before the first stop and beyond the last one
    // and continuous at both, so within e of them the first or the last
    // segment's bound holds; at an inner stop the side must be known.
    const bool flat = n == 1 || (i == 0 && g.offsets[0] - o.t > e) || (i == n && o.t - g.offsets[n - 1] > e);
    const int i0 = flat ? (i == 0 ? 0 : n - 1) : min(max(i - 1, 0), n - 2), i1 = flat ? i0 : i0 + 1;
    const float lo = g.offsets[i0], hi = g.offsets[i1];
    bool ok = flat || ((i0 == 0 || o.t - lo > e) && (i1 == n - 1 || hi - o.t > e));
    const RGBf a = g.prep[i0], b = g.prep[i1];
    float w = 0.0f, ew = 0.0f;
    if (!flat) {
        // the reference rounds the two differences and the quotient; here
        // the reciprocal is within 2 ulp (equal stops make it infinite and
        // every bound with it)
        const float inv = __fdividef(1.0f, hi - lo);
        w = fminf(fmaxf((o.t - lo) * inv, 0.0f), 1.0f);
        ew = e * inv * 1.01f + 9.0f * kU;
    }
    // a + (b - a) w: the difference, the product and the sum round once each
    // there, the difference and the fused step here
    auto lerp = [w](float p, float d) { return __fmaf_rn(d, w, p); };
    auto elerp = [ew](float d, float v) { return fabsf(d) * (ew + 4.0f * kU) + 2.0f * kU * fabsf(v); };
    const float da = b.a - a.a, al = lerp(a.a, da);
    float ea = elerp(da, al);
    float d0 = b.r - a.r;
    const float d1 = b.g - a.g, d2 = b.b - a.b;
    float r, gg = lerp(a.g, d1), bl = lerp(a.b, d2), er, eg = elerp(d1, gg), eb = elerp(d2, bl);
    if (method <= Z2D_INTERP_SRGB) {
        r = lerp(a.r, d0);
        er = elerp(d0, r);
        if (method == Z2D_INTERP_LINEAR_RGB && dither == Z2D_DITHER_NONE) {
            out = I16{enc_f32(r, er, ok), enc_f32(gg, eg, ok), enc_f32(bl, eb, ok), enc_f32(al, ea, ok)};
            return ok;
        }
    }
    // demultiplied; the quotient of values within their bounds
    ok = ok && al > 0.02f && ea < 0.005f * al;
    const float inv = __fdividef(1.0f, al), einv = 1.01f * inv;
    gg *= inv;
    bl *= inv;
    eg = (eg + fabsf(gg) * ea) * einv + 5.0f * kU * fabsf(gg);
    eb = (eb + fabsf(bl) * ea) * einv + 5.0f * kU * fabsf(bl);
    if (method <= Z2D_INTERP_SRGB) {
        r *= inv;
        er = (er + fabsf(r) * ea) * einv + 5.0f * kU * fabsf(r);
        if (method == Z2D_INTERP_SRGB) {
            // the slope of x^2.2 is below 2.21 x up to 1.002
            ok = ok && r < 1.001f && gg < 1.001f && bl < 1.001f && er < 1e-3f && eg < 1e-3f && eb < 1e-3f;
            er = 2.25f * (r + er) * er + kGammaErr;
            eg = 2.25f * (gg + eg) * eg + kGammaErr;
            eb = 2.25f * (bl + eb) * eb + kGammaErr;
            r = gamma_f32(r);
            gg = gamma_f32(gg);
            bl = gamma_f32(bl);
        }
    } else {
        // HSL: the hues the way the polar rule takes them (exact stops), then
        // toLinearRGB's channels l - s min(l, 1 - l) max(-1, min(k - 3, 9 - k, 1))
        // with k = (n + hue / 30) mod 12, continuous in all three
        float ah = a.r, bh = b.r;
        if (method == Z2D_INTERP_HSL_SHORTER) {
            if (bh - a.r > 180.0f) ah += 360.0f;
            if (b.r - a.r < -180.0f) bh += 360.0f;
        } else if (method == Z2D_INTERP_HSL_LONGER) {
            const float d = b.r - a.r;
            if (0.0f < d && d < 180.0f) ah += 360.0f;
            if (-180.0f < d && d <= 0.0f) bh += 360.0f;
        } else if (method == Z2D_INTERP_HSL_INCREASING) {
            if (b.r < a.r) bh += 360.0f;
        } else {
            if (a.r < b.r) ah += 360.0f;
        }
        d0 = bh - ah;
        const float h = __fmaf_rn(d0, w, a.r);  // (from the stop's own hue, as the reference has it)
        // the reference rounds the hues' difference, its product with w and
        // the sum, here the sum; k = (hue mod 360) / 30 + n rounds by 12 u and
        // 20 u on both sides, the mod here by 12 u more
        const float eh = fabsf(d0) * (ew + 2.0f * kU) + 2.0f * kU * fabsf(h);
        const float turns = floorf(h * (1.0f / 360.0f));
        float k0 = __fmaf_rn(turns, -360.0f, h) * (1.0f / 30.0f);
        k0 = k0 < 0.0f ? k0 + 12.0f : k0 >= 12.0f ? k0 - 12.0f : k0;  // (the quotient may round over a turn)
        const float sat = gg, light = bl, es = eg, el = eb;
        const float room = fminf(light, 1.0f - light), amp = sat * room;
        // |f| <= 1, slope 1 / 30 per degree; amp moves by at most
        // es |room| + |sat| el
        const float ech = fabsf(amp) * (eh * (1.0f / 30.0f) + 80.0f * kU) + es * fabsf(room) + (fabsf(sat) + es + 1.0f) * el +
                          6.0f * kU * (fabsf(light) + fabsf(amp));
        auto channel = [k0, amp, light](float n) {
            float k = k0 + n;
            if (k >= 12.0f) k -= 12.0f;
            return __fmaf_rn(-amp, fmaxf(-1.0f, fminf(fminf(k - 3.0f, 9.0f - k), 1.0f)), light);
        };
        r = channel(0.0f);
        gg = channel(8.0f);
        bl = channel(4.0f);
        er = eg = eb = ech;
    }
    float av = al;
    if (dither != Z2D_DITHER_NONE) {
        const float m = dither == Z2D_DITHER_BAYER ? bayer(x, y) : blue_noise(x, y);
        const float add = m * dither_step;
        auto dithered = [add](float c) { return fmaxf(0.0f, fminf(c + add, 1.0f)); };
        // NaNs must not be clamped away
        ok = ok && r >= 0.0f && gg >= 0.0f && bl >= 0.0f;
        r = dithered(r);
        gg = dithered(gg);
        bl = dithered(bl);
        av = dithered(al);
        er += 3.0f * kU, eg += 3.0f * kU, eb += 3.0f * kU, ea += 3.0f * kU;
    }
    out = premul16(I16{enc_f32(r, er, ok), enc_f32(gg, eg, ok), enc_f32(bl, eb, ok), enc_f32(av, ea, ok)});
    return ok;
}

// The gradient's lanes at (x, y); false where f32 does not decide them.
__device__ __forceinline__ bool grad_lanes_f32(int kind, int method, int dither, float dither_step, const DevGradient &g,
                                               int32_t x, int32_t y, I16 &out) {
    const int32_t mode = g.fz.mode;
    if (mode == kFastNone || mode == kFastVoid || mode == kFastRadialA0 ||
        (uint32_t)(x + (1 << 22)) >= (1u << 23) || (uint32_t)(y + (1 << 22)) >= (1u << 23))
        return false;
    const OffsetF32 o = offset_f32(kind, g.fz, g.has_tf != 0, (float)x + 0.5f, (float)y + 0.5f);
    return color_f32(method, dither, dither_step, g, o, x, y, out);
}

}  // namespace z2dg
