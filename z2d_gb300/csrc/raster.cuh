// raster.cuh -- the tile rasteriser (raster.cu) as the fill pipeline
// (fill.cu) launches it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fill.cuh"

namespace z2dg {

// An edge in the bin of one (fill, band): the f32 half of its DEdge and its
// index, for the crossings that are evaluated in f64.
struct BinEdge {
    int32_t xi;
    float fx, fxi, fdt;
    int32_t rt, rb;
    int32_t id, _pad;
};
static_assert(sizeof(BinEdge) == 32, "BinEdge: two 16-byte accesses");

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
    const DEdge *edges;
    const void *bins;           // BinEdge records, or (gather) int32 indices of `edges`
    const int32_t *bin_off;
    const int32_t *band_count;  // per global band
    const int4 *band_fills;     // {fill, cull_x0, cull_x1, (fill, band) slot} per band, in call order
    const RasterFill *rfills;
    const TileRec *tiles;       // per tile (several surfaces only)
    const uint8_t *masks;
    int32_t n_jobs;
    unsigned long long *queue;  // work-queue counter, zero at launch
    unsigned long long n_items; // tiles (CTA items) or tiles x rows (warp items)
    const int32_t *order;       // tile order of the queue, or null (tile index order)
    int32_t one_per_tile;       // not persistent: CTA i draws the i-th tile of the queue
};

// How k_raster runs: `multi` for several surfaces, `cta_items` for a whole
// tile per work item, `plain` when every fill of the batch is a pixel src_over
// fill (FAST_PIXEL_SRC_OVER) and none takes the exact path; `gather` for bins
// of edge indices and edges without their f32 fields, as the one-upload path's
// host writes them (with records and fields from the host a call of 1,500
// edges took 67 us instead of 56).
struct RasterVariant {
    bool multi, cta_items, plain, gather;
};
int raster_occupancy(Ctx &c, RasterVariant v, int &ctas_per_sm);
int raster_launch(Ctx &c, RasterVariant v, const RasterArgs &A, unsigned grid);

}  // namespace z2dg
