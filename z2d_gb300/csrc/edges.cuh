// edges.cuh -- Polygon.addEdge on the device and the ordered keys of the
// per-fill extents, shared by the fill flattener and the stroker.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "f64_int.cuh"
#include "fill.cuh"

namespace z2dg {

// Order-preserving map of finite doubles to u64 (for atomic min/max).
__device__ __forceinline__ unsigned long long dkey(double v) {
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__host__ __device__ __forceinline__ double dkey_inv(unsigned long long k) {
    unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double d;
    memcpy(&d, &b, 8);
    return d;
#endif
}

// The f64 operations of addEdge that have exact integer forms
// (f64_int.cuh), with the f64 instruction for the operands they decline.
__device__ __forceinline__ double scale_coord(double v, double s) {
    bool ok;
    const double r = f64_scale_pow2(v, s, ok);
    if (ok) return r;
    return f64_mul_hw(v, s);
}
__device__ __forceinline__ int32_t round_i32(double v) {
    bool ok;
    const int32_t r = f64_round_i32(v, ok);
    if (ok) return r;
    return f64_round_i32_hw(v);
}
__device__ __forceinline__ void add_edge(const FillCmd &F, DEdge *out, double x0, double y0, double x1, double y1,
                                         double &et, double &eb, double &el, double &er, bool &any) {
    // Polygon.addEdge (Polygon.zig:61-109)
    const double ax = scale_coord(x0, F.edge_scale), ay = scale_coord(y0, F.edge_scale);
    const double bx = scale_coord(x1, F.edge_scale), by = scale_coord(y1, F.edge_scale);
    DEdge e;
    const bool down = f64_lt(ay, by);
    if (!down && !f64_lt(by, ay)) {
        e.top = 0;
        e.x_start = 0;
        e.x_inc = 0;
        e.xi = 0;
        e.fx = e.fxi = e.fdt = 0.0f;
        e.rt = 1;
        e.rb = 0;  // horizontal: never active
        *out = e;
        return;
    }
    // from the upper to the lower end: the division, most of the work, is one
    // call for a warp's edges of both directions (with a call for each, and
    // the extents reduced by 64-bit shuffles, the curve edges of 2,000 paths
    // took 119 us, now 96; of 1,024 glyphs 82, now 66)
    const double bot = down ? by : ay, x_end = down ? bx : ax;
    e.top = down ? ay : by;
    e.x_start = down ? ax : bx;
    e.x_inc = f64_div_dev(x_end - e.x_start, bot - e.top);
    e.rb = round_i32(bot);
    if (!edge_fields(e, down)) e.rt = f64_round_i32_hw(e.top);
    const bool lr = f64_lt(ax, bx);
    const double l = lr ? ax : bx, r = lr ? bx : ax;
    if (!any) {
        et = e.top; eb = bot; el = l; er = r;
        any = true;
    } else {
        if (f64_lt(e.top, et)) et = e.top;
        if (f64_lt(eb, bot)) eb = bot;
        if (f64_lt(l, el)) el = l;
        if (f64_lt(er, r)) er = r;
    }
    *out = e;
}

// The smallest of the warp's 64-bit keys, from two 32-bit reductions: of the
// high words, then of the low words of those that have the smallest.
__device__ __forceinline__ unsigned long long warp_min(unsigned long long k) {
    const uint32_t hi = (uint32_t)(k >> 32), h = __reduce_min_sync(0xffffffffu, hi);
    const uint32_t l = __reduce_min_sync(0xffffffffu, hi == h ? (uint32_t)k : 0xffffffffu);
    return ((unsigned long long)h << 32) | l;
}

// Merges the lanes' edge extents into their fills' FillState: one set of
// atomics per warp when every lane that has edges draws the same fill, one
// per lane otherwise.  All 32 lanes must call it.
__device__ __forceinline__ void merge_extents(FillState *st, int32_t f, bool any, double et, double eb, double el,
                                              double er) {
    const unsigned all = 0xffffffffu;
    const unsigned am = __ballot_sync(all, any);
    if (!am) return;
    const int lead = __ffs(am) - 1;
    const int32_t f0 = __shfl_sync(all, f, lead);
    if (__all_sync(all, !any || f == f0)) {
        // reduced as ordered keys: integer minima (f64 min/max instructions
        // run on GB300's narrow f64 pipe), maxima as those of the complement
        const unsigned long long mt = warp_min(any ? dkey(et) : ~0ull), mb = ~warp_min(any ? ~dkey(eb) : ~0ull);
        const unsigned long long ml = warp_min(any ? dkey(el) : ~0ull), mr = ~warp_min(any ? ~dkey(er) : ~0ull);
        if ((int)(threadIdx.x & 31) == lead) {
            FillState &S = st[f0];
            atomicMin(&S.ext[0], mt);
            atomicMax(&S.ext[1], mb);
            atomicMin(&S.ext[2], ml);
            atomicMax(&S.ext[3], mr);
            atomicOr(&S.has_edges, 1);
        }
    } else if (any) {
        FillState &S = st[f];
        atomicMin(&S.ext[0], dkey(et));
        atomicMax(&S.ext[1], dkey(eb));
        atomicMin(&S.ext[2], dkey(el));
        atomicMax(&S.ext[3], dkey(er));
        atomicOr(&S.has_edges, 1);
    }
}

}  // namespace z2dg
