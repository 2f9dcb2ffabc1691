// fill.cuh -- device structures of the fill pipeline (fill.cu).
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "z2d_internal.h"

namespace z2dg {

constexpr int kSplineStack = 48;  // subdivision depth bound (coordinates are bounded)
constexpr int32_t kSplineMaxSplits = 1 << 22;  // subdivisions per curve before giving up
constexpr int kTileRows = 4;      // pixel rows per band / tile
constexpr int kTileCols = 256;    // pixels per tile row
constexpr int kRasterThreads = 32 * kTileRows;  // one warp per tile row
constexpr int32_t kMaxBandEdges = 32000;  // edges of one fill in one band (16-bit winding counters)

// One fill command, prepared on the host.
struct FillCmd {
    int32_t node_off, n_nodes;
    int32_t aa;         // Z2D_AA_NONE, Z2D_AA_MULTISAMPLE_4X or Z2D_AA_SUPERSAMPLE_4X
    int32_t rule, op;
    int32_t precision;  // after the float upgrade of multisample.zig:36 / direct.zig:25
    int32_t pattern_kind;
    int32_t reduces;    // pixel pattern whose operator reduces to the source (shared.zig:111-117)
    int32_t fast_kind;  // FAST_* specialisation the rasteriser may use
    int32_t job;        // index of the surface (job) the fill draws on
    int32_t stroke;     // device-stroked command whose polygon this fill draws, or -1
    int32_t poly;       // host-built polygon this fill draws, or -1
    double tol;         // max(tolerance, 0.001) (painter.zig:103)
    double scale;       // 4 for multisample / supersample, 1 for none (painter.zig:93-97)
    double edge_scale;  // multiplier of node coordinates in Polygon.addEdge: scale, or 1 for
                        // stroke contours whose points are already scaled
    DevSrc src;         // the pattern as a compositor source
    Px px_paint;        // pattern pixel converted to the surface format (paintStride)
    I16 px_rgba;        // RGBA.fromPixel lanes of the pattern pixel (compositeStride)
};

// Per-node results of the flatten passes.
struct NodeInfo {
    double sx, sy;  // start point (the buffer's last point before the node)
    double ex, ey;  // close_path: the subpath's first point
    int32_t n_emit; // edges emitted (one per lineTo the reference issues)
    int32_t n_added;
    int32_t edge_off;
    int32_t pool;   // first of its polyline's points in the curve pool, or -1 (see k_curve_count_w)
};

// Polygon.Edge plus its rounded active range: the edge is active on sample
// row y exactly when rt <= y < rb (top < y+0.5 <= bottom, Polygon.zig:284-285;
// a horizontal edge has rt = 1, rb = 0 and is never active).  The first 16
// bytes hold what crossing_f32 needs, as one vector: x_start split
// into a whole part xi and a rest fx, the slope, and fdt = rt + 0.5 - top,
// whose sign bit is the direction (set: -1 down, clear: +1 up).
struct DEdge {
    int32_t xi;
    float fx, fxi, fdt;
    int32_t rt, rb;
    double x_start, x_inc, top;
};

static_assert(sizeof(DEdge) == 48, "DEdge layout: 16-byte f32 block, ranges, f64 fields");

// A thread's warp among all of its grid's, for grids of one warp per item: with
// 2^27 items and more the thread's own number does not fit 32 bits.
Z2D_HD long long warp_number(uint32_t block, uint32_t threads, uint32_t thread) {
    return ((long long)block * threads + thread) >> 5;
}

Z2D_HD float f32_of_bits(uint32_t b) {
    float f;
    memcpy(&f, &b, 4);
    return f;
}

// |v| as 32.32 fixed point (truncated), from the bits of v: no f64
// instruction.  False for |v| >= 2^26 and for what is not finite.
Z2D_HD bool fixed_coord(double v, uint32_t &whole, uint32_t &frac, bool &neg) {
    uint64_t b;
    memcpy(&b, &v, 8);
    const int32_t sh = 31 + 1023 - (int32_t)((b >> 52) & 0x7FFu);  // 31 - exponent
    neg = (b >> 63) != 0;
    const uint64_t q = ((b << 11) | (1ull << 63)) >> (sh < 0 ? 0 : sh > 63 ? 63 : sh);
    whole = (uint32_t)(q >> 32);
    frac = (uint32_t)q;
    return sh >= 6;
}
// A 32-bit fraction as an f32 in [0, 1), truncated to 23 bits.
Z2D_HD float frac_f32(uint32_t f) { return f32_of_bits(0x3F800000u | (f >> 9)) - 1.0f; }

// The f32 fields and rt of an edge whose x_start, x_inc and top are set.
// rt is round(top), half away from zero.  Every field is truncated, not
// rounded: fx is within 2^-23 of x_start - xi, fdt within 2^-23 of
// rt + 0.5 - top (in [0, 1]), fxi within 2^-23 of x_inc relatively.  What
// does not fit (coordinates of 2^26 and more, slopes outside f32's normal
// range) leaves a NaN in fx: every crossing of the edge is then evaluated
// in f64.  False when top does not fit: rt is then the caller's to set.
Z2D_HD bool edge_fields(DEdge &e, bool down) {
    uint32_t w, f;
    bool neg;
    bool ok = fixed_coord(e.x_start, w, f, neg);
    const float fx = frac_f32(f);
    e.xi = (int32_t)(neg ? 0u - w : w);
    e.fx = neg ? -fx : fx;
    uint64_t b;
    memcpy(&b, &e.x_inc, 8);
    const int32_t se = (int32_t)((b >> 52) & 0x7FFu) - 1023 + 127;
    const bool zero = (b << 1) == 0;
    ok &= zero || (se > 0 && se < 255);
    e.fxi = zero ? 0.0f
                 : f32_of_bits(((uint32_t)(b >> 32) & 0x80000000u) | ((uint32_t)se << 23) |
                               ((uint32_t)(b >> 29) & 0x7FFFFFu));
    const bool top_ok = fixed_coord(e.top, w, f, neg);
    // away from zero by one where the fraction is 1/2 or more
    const uint32_t up = f >> 31;
    const float r = frac_f32(f), m = (float)up;
    const float d = neg ? (0.5f - m) + r : (0.5f + m) - r;
    e.rt = (int32_t)(neg ? 0u - (w + up) : w + up);
    e.fdt = down ? -d : d;
    if (!(ok && top_ok)) e.fx = f32_of_bits(0x7FC00000u);
    return top_ok;
}

// The direction of a (not horizontal) edge.
Z2D_HD int32_t edge_dir(const DEdge &e) {
    uint32_t b;
    memcpy(&b, &e.fdt, 4);
    return (b >> 31) ? -1 : 1;
}

// The crossing of an edge with sample row sr is
//   X = round(x_start + x_inc * ((sr + 0.5) - top))      (Polygon.zig:272-276)
// in f64, rounded half away from zero.  With the edge's split fields,
// X = xi + round(fx + fxi * t), t = (sr - rt) + fdt >= 0: the f32 value
// carries the distance along the edge only, not the coordinates.  With
// u = 2^-24, T the largest t asked of the edge and p = |fxi| T, to first
// order its error is at most
//   u (2 p (slope) + 3 p (t: two sums and the conversion)
//      + 3 |fxi| (fdt) + 2 (fx) + (1 + p) (the fused multiply-add's rounding))
// and the f64 evaluation's own error is below u / 4 for |x_start| < 2^26 (a
// larger one has fx = NaN), p < 2^21.  The bound used is 1.25 times
// u (7 p + 3 |fxi| + 5).  A value farther than the bound from every
// half-integer rounds as the f64 value does; the others, and those
// whose bound is 1/2 or more (so p stays below 2^21 where rounding by adding
// 1.5 * 2^23 is exact), have to be evaluated in f64.
constexpr float kRoundMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int32_t kRoundMagicBits = 0x4B400000;
// The largest distance from the rounded value that decides it.
Z2D_HD float crossing_limit(float fxi, float t_max) {
    const float s = fabsf(fxi), p = s * t_max;
    return 0.5f - 7.450580596923828e-8f * (7.0f * p + 3.0f * s + 5.0f);
}
// round(fx + fxi * t) + kRoundMagicBits; false when f32 does not decide it.
Z2D_HD bool crossing_f32(float fx, float fxi, float t, float limit, int32_t &n) {
#ifdef __CUDA_ARCH__
    const float v = __fmaf_rn(fxi, t, fx);
#else
    const float v = fmaf(fxi, t, fx);
#endif
    const float m = v + kRoundMagic;
    memcpy(&n, &m, 4);
    return fabsf(v - (m - kRoundMagic)) <= limit;  // NaN fails
}

enum : int32_t {
    FAST_NONE = 0,
    FAST_PIXEL_SRC_OVER = 1,   // pixel pattern, integer precision, src_over
    FAST_SOURCE_SRC_OVER = 2,  // gradient or dither pattern, integer precision, src_over
};

enum : int32_t {
    FILL_OPEN_CHAIN = 1,  // an open 2-point subpath: rows may be unbalanced
    FILL_EXACT = 2,       // rasterised by k_exact
    FILL_SS_ZERO = 4,     // supersample mask too small to downsample: all zero
};

struct FillState {
    int32_t edge_base, n_edges, flags, has_edges;
    unsigned long long ext[4];  // top(min), bottom(max), left(min), right(max) as ordered keys
    int32_t active;             // inBox passed
    int32_t start_y, end_y;     // draw rows [start_y, end_y] (supersample: the composite region)
    int32_t start_x, end_x;     // draw columns [start_x, end_x)
    int32_t band0, band1;       // bands the fill touches
    int32_t fb_base;            // first (fill, band) slot
    int32_t mask_w, mask_x0;
    long long mask_base;        // exact-path action mask offset (bytes)
    int32_t cull_x0, cull_x1;   // columns a tile must overlap to be affected
};

// What k_raster reads of a fill on its common path
// (written by k_fill_setup from the FillCmd and FillState).
struct RasterFill {
    int32_t start_x, end_x, start_y, end_y;  // FillState's draw box
    uint32_t meta;  // RF_* fields below
    int32_t _pad[3];
};
static_assert(sizeof(RasterFill) == 32, "RasterFill: the box is one 16-byte load");
enum : uint32_t {
    RF_OP_MASK = 0x1F,        // operator
    RF_AA_SHIFT = 5,          // anti-aliasing mode, 2 bits
    RF_EVEN_ODD = 1u << 7,    // fill rule
    RF_FAST_SHIFT = 8,        // FillCmd.fast_kind, 2 bits
    RF_EXACT = 1u << 10,      // FILL_EXACT
    RF_SS_ZERO = 1u << 11,    // FILL_SS_ZERO
    RF_BOUNDED = 1u << 12,    // the operator is bounded
    RF_IN_ROWS = 1u << 31,    // set by k_raster: the row is one of the draw box
};

// counters (int32 slots; the mask byte count is a 64-bit pair)
enum : int32_t {
    CNT_EDGES = 0,
    CNT_FILL_BANDS = 1,
    CNT_MASK_LO = 2,  // + CNT_MASK_HI = 3
    CNT_EXACT = 4,
    CNT_STATUS = 5,
    CNT_CURVES = 6,       // curves queued by k_node_count_w, per class (6 slots)
    CNT_CURVES_EMIT = 12, // curves queued by k_node_emit_w
    CNT_POOL = 14,        // points asked of the curve pool (64-bit pair, + 15)
    CNT_QUEUE = 16,       // k_raster's work-queue counter (64-bit pair, + 17)
    CNT_COUNT = 18
};

// action-mask byte of the exact path: bit 7 = clear first, bits 0-4 = coverage
constexpr uint8_t kMaskClear = 0x80;

// One surface of a batch with the contiguous range of its fills.  The host
// sets sfc and fill0/fill1; k_fill_setup widens the touched band and tile
// column ranges; the host then lays out global bands, tiles and band-list
// storage job after job.
struct DevJob {
    DevSurface sfc;
    int32_t fill0, fill1;      // fills [fill0, fill1), in call order
    int32_t band_lo, band_hi;  // 4-row bands touched (band_hi < band_lo: none)
    int32_t tcol_lo, tcol_hi;  // 256-pixel tile columns touched
    int32_t gband_base;        // first global band of the job
    int32_t tile_base;         // first CTA of the job in k_raster's grid
    long long list_base;       // first band-list entry (one slot per fill and band)
};

// Runs ordered lists of fills on device surfaces (one list per job; jobs are
// independent).  `fills` hold the prepared commands grouped by job (node
// offsets into `nodes`, host memory; the fills' node ranges are disjoint);
// grad_of_fill[i] >= 0 names the gradient of fill i in `grads`.
// Nodes that no fill owns are skipped; device-stroked
// commands (`strokes`, fills with stroke >= 0) read their nodes from the
// same array; fills with poly >= 0 draw a host-built polygon of `strokes`.
// A call with few short fills, on one surface or many, in a single launch,
// with its tables as parameters or in one copy before it: the host flattens the paths (fill_plotter.plot,
// Spline.decompose, Polygon.addEdge), sets the fills up (inBox,
// multisample.run's draw box), bins their edges and lays out the band
// lists; the rasteriser draws the tiles.  Sets `done` = false without
// touching the device when the call is not one it takes (another
// anti-aliasing mode, strokes, an open two-point chain, more nodes, edges or
// bands than its limits, a packed surface, a gradient with a stop table),
// and the caller runs the full pipeline.
int run_small_jobs(Ctx &c, std::vector<DevJob> &jobs, const z2d_node *nodes, const std::vector<FillCmd> &fills,
                   const std::vector<DevGradient> &grads, const std::vector<int32_t> &grad_of_fill, bool &done);

struct StrokeSet;
int run_jobs(Ctx &c, std::vector<DevJob> &jobs, const z2d_node *nodes, int32_t n_nodes, std::vector<FillCmd> &fills,
             const std::vector<DevGradient> &grads,
             const std::vector<int32_t> &grad_of_fill, const StrokeSet *strokes = nullptr);

}  // namespace z2dg
