// raster.cuh -- the tile rasteriser (raster.cu) as the fill pipeline
// (fill.cu) launches it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "fill.cuh"

namespace z2dg {

// The supersample mask value of a pixel whose 4x4 sample block has n covered
// samples, as 8-bit alpha: the mask is alpha8, or the surface's own format
// for alpha4/2/1 surfaces (supersample.zig:69-83), each covered sample is
// opaque, and downsampleBuffer averages the 16 (surface.zig:447-469).
Z2D_HD uint32_t ss_mask8(int n, int fmt) {
    if (fmt >= Z2D_FORMAT_ALPHA4) return scale_alpha(((uint32_t)n * fmt_max(fmt)) / 16u, fmt_bits(fmt), 8);
    return ((uint32_t)n * 255u) / 16u;
}

// An edge in the bin of one (fill, band), as a pixel row of the band needs
// it: the crossing with the band's sample row s is
//   xi + round(fx + fxi (t + s)),  c = xi - kRoundMagicBits,
// if bit s of `rows` is set and f32 decides it (limit); bit 31 is set for a
// downward edge.  `id` is the edge's index, for f64.
struct BinEdge {
    int32_t c;
    float fx, fxi, t;
    uint32_t rows;
    float limit;
    int32_t id, _pad;
};
// The record of an edge (its DEdge fields) for the n sample rows from `row`
// (>= 0).
// A pixel row evaluates fma(fxi, r, fma(fxi, t + w, fx)) with s = w + r.
// With T >= |t|, |t + w| and the largest t + s, p = |fxi| T and u = 2^-24, the
// error is at most u (2 p (slope) + 3 p (t: the conversion and two sums)
// + 3 |fxi| (fdt) + 2 (fx) + 2 (1 + p) (the multiply-adds)), within the bound
// of crossing_limit.
Z2D_HD BinEdge bin_edge(int32_t xi, float fx, float fxi, float fdt, int32_t rt, int32_t rb, int32_t id, int32_t row,
                        int32_t n) {
    BinEdge B;
    // rt and rb are the ends of an edge of any length, saturated at the ends of
    // the int32 range: they are compared with the band before they are
    // subtracted from it
    const int32_t lo = rt <= row ? 0 : rt - row < n ? rt - row : n;
    const int32_t hi = rb <= row ? 0 : rb - row < n ? rb - row : n;
    const uint32_t away = rt <= row ? (uint32_t)row - (uint32_t)rt : (uint32_t)rt - (uint32_t)row;
    const float rel = rt <= row ? (float)away : -(float)away;
    B.c = (int32_t)((uint32_t)xi - (uint32_t)kRoundMagicBits);
    B.fx = fx;
    B.fxi = fxi;
    B.t = rel + fabsf(fdt);
    B.rows = lo < hi ? ((1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
    uint32_t dir;
    memcpy(&dir, &fdt, 4);
    B.rows |= dir & 0x80000000u;
    B.limit = crossing_limit(fxi, fmaxf(rel + (float)hi, 1.0f - rel));
    B.id = id;
    B._pad = 0;
    return B;
}
static_assert(sizeof(BinEdge) == 32, "BinEdge: two 16-byte accesses");

// An edge as the one-upload path's host writes it: what its f32 fields are
// made from, in 32 bytes (the upload of a call of 1,500 edges is most of what
// its tables weigh).
struct SmallEdge {
    double x_start, x_inc, top;
    int32_t rt, rb2;  // rb2: 2 rb, + 1 for a downward edge
};
static_assert(sizeof(SmallEdge) == 32, "SmallEdge: two 16-byte accesses");

// A tile of a batch of several surfaces: its surface, its band counted
// from the surface's first touched one, and its tile column.
struct TileRec {
    int32_t job, band, col, _pad;
};

struct RasterArgs {
    DevJob job0;                // the job of a one-surface batch, by value
    const DevJob *jobs;
    const FillCmd *fills;
    const FillState *st;
    const void *edges;          // DEdge, or (kBinSmall) SmallEdge
    const void *bins;           // BinEdge records, or int32 indices of `edges` (BinKind)
    const int32_t *bin_off;
    const int32_t *band_count;  // per global band
    const int4 *band_fills;     // {fill, cull_x0, cull_x1, (fill, band) slot} per band, in call order
    const RasterFill *rfills;
    const uint32_t *luts;       // 32 source words per fill (coverage_word)
    const TileRec *tiles;       // per tile (several surfaces only)
    const uint8_t *masks;
    unsigned long long *queue;  // work-queue counter, zero at launch
    unsigned long long n_items; // tiles (CTA items) or tiles x rows (warp items)
    const int32_t *order;       // tile order of the queue, or null (tile index order)
    int32_t one_per_tile;       // not persistent: CTA i draws the i-th tile of the queue
};

// What the fills of a batch have in common: pixel src_over fills
// (FAST_PIXEL_SRC_OVER) none of which takes the exact path, all with 4x4
// samples or all without anti-aliasing, or anything.  (2,000 paths without
// anti-aliasing: the general kernel 2.00 ms, kPlainDirect 1.20.)
enum : int { kGeneral = 0, kPlain4x = 1, kPlainDirect = 2 };
inline int raster_mode(const FillCmd *fills, size_t n, bool any_exact) {
    bool plain = !any_exact, direct = true, sampled = true;
    for (size_t i = 0; i < n; i++) {
        plain &= fills[i].fast_kind == FAST_PIXEL_SRC_OVER;
        direct &= fills[i].aa == Z2D_AA_NONE;
        sampled &= fills[i].aa != Z2D_AA_NONE;
    }
    return !plain ? kGeneral : sampled ? kPlain4x : direct ? kPlainDirect : kGeneral;
}

// The source word of a FAST_PIXEL_SRC_OVER fill for coverage k of a pixel:
// the pixel at full coverage, dst_in(pixel, opacity(k)) below it; on the
// alpha formats its alpha alone.  0 beyond full coverage.
Z2D_HD uint32_t coverage_word(const FillCmd &F, int fmt, int k) {
    const int full = F.aa == Z2D_AA_NONE ? 1 : 16;
    if (k > full) return 0u;
    I16 s = I16{F.src.pix.r & 0xFFu, F.src.pix.g & 0xFFu, F.src.pix.b & 0xFFu, F.src.pix.a & 0xFFu};
    if (k < full) {
        const uint32_t o = F.aa == Z2D_AA_SUPERSAMPLE_4X ? ss_mask8(k, fmt) : k == 0 ? 0u : (uint32_t)(k * 16 - 1);
        s = I16{(s.r * o) / 255u, (s.g * o) / 255u, (s.b * o) / 255u, (s.a * o) / 255u};
    }
    return fmt <= Z2D_FORMAT_RGBA ? i16_to_word(s, word_order(fmt)) : s.a;
}

// What the bins of (fill, band) hold: the edges' records, or indices of edges
// whose records every pixel row works out, either of the one-upload path's
// SmallEdge (with records from the host a call of 1,500 edges took 67 us
// instead of 56) or of DEdge, where the device has no room for the records.
// kBinShared is kBinSmall with all of a call's tables in shared memory.
enum BinKind : int { kBinRecords = 0, kBinSmall = 1, kBinIndex = 2, kBinShared = 3 };

// How k_raster runs: `multi` for several surfaces, `cta_items` for a whole
// tile per work item, the mode, and what the bins hold.  kBinSmall and
// kBinShared come with a tile per item and 4x4 samples, kBinIndex with a row
// per item and in the general mode only.
struct RasterVariant {
    bool multi, cta_items;
    BinKind bins;
    int mode;
};

// A small call's tables, as a parameter of its one launch.
constexpr size_t kParamBytes = 8192;
struct ParamBlob {
    uint4 v[kParamBytes / sizeof(uint4)];
};
int raster_occupancy(Ctx &c, RasterVariant v, int &ctas_per_sm);
int raster_launch(Ctx &c, RasterVariant v, const RasterArgs &A, unsigned grid);
// A CTA per tile of a call whose tables are the first n words of P: A's
// pointers, and those of its fills' gradients, are offsets into them.
int raster_launch_small(Ctx &c, bool multi, int mode, const RasterArgs &A, const ParamBlob &P, int32_t n, int32_t n_fills,
                        unsigned grid);

}  // namespace z2dg
