// raster.cu -- the tile rasteriser: coverage of the binned edges of a batch's
// fills, composited in call order (WorkingEdgeSet, multisample.run,
// raster/shared.zig, Surface.paintStride/compositeStride).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "raster.cuh"
#include "raster_px.cuh"
#include "z2d_internal.h"

namespace z2dg {

// --------------------------------------------------------- compositing
// One pixel of the supersample batch [dst_in(dst = pattern, src = mask), op]
// (supersample.zig:171-184) as StrideCompositor.runPrecision evaluates it
// (compositor.zig:540-621): the mask reads as alpha-only lanes.
static __device__ __noinline__ I16 apply_ssaa(const FillCmd &F, int32_t x, int32_t y, uint32_t m8, I16 d) {
    if (F.precision == Z2D_PRECISION_INTEGER) {
        const I16 r = int_op(Z2D_OP_DST_IN, src_i16_fast(F.src, x, y, 0), I16{0, 0, 0, m8});
        return int_op_any(F.op, d, r);
    }
    const F4 r = float_op(Z2D_OP_DST_IN, src_f4_fast(F.src, x, y, 0), decode_raw(I16{0, 0, 0, m8}));
    return encode_raw(float_op_any(F.op, decode_raw(d), r));
}

// The source word (word_order) of a pixel of a FAST_SOURCE_SRC_OVER fill with
// `opacity`: dst_in(pattern, opacity), the pattern itself at 255 (where
// dst_in changes nothing).
__device__ __forceinline__ uint32_t source_word(I16 s, uint32_t opacity, int fmt) {
    const uint32_t L = i16_to_word(s, word_order(fmt));
    return div255x2((L & 0x00FF00FFu) * opacity) | (div255x2(((L >> 8) & 0x00FF00FFu) * opacity) << 8);
}

// multisample.run's clears for unbounded operators (multisample.zig:96-110),
// including its quirks: the rows below the draw box are cleared up to the
// surface WIDTH, and the right-hand clear starts at x = 0.
__device__ __forceinline__ bool msaa_unbounded_clear(const FillState &S, int32_t x, int32_t y, int32_t sw) {
    if (y < S.start_y) return true;
    if (y > S.end_y) return y < sw;
    return (S.start_x > 0 && x < S.start_x) || (S.end_x < sw && x < sw - S.end_x);
}

// Crossings of one warp's pixel row: up to 4 sample rows of 1024 sample
// columns, one 32-bit word of columns per lane.  Sample column c belongs to
// lane c / per (per = sample columns per lane: 32 with 4x sampling, 8
// without) and is bit c % per of the lane's word.
//   even-odd: one plane per sample row; a crossing toggles its bit.
//   non-zero: planes U0 D0 U1 D1 U2 D2 per sample row; the first upward
//     crossing of a column sets its bit of U0, the second one that of U1, the
//     third one that of U2 (D for downward).  A fourth crossing of one
//     column, row and direction sends the (fill, row) to winding_bits.
// Against 16-bit counters per column this is one atomic per crossing instead
// of three, and the even-odd rule needs no walk over the crossings at all:
// the inside bits are the prefix XOR of the toggles.  Issue bound, on the
// ALU pipe: a fill costs a row and tile of the 2,000-path 4096x4096 batch
// (2.9 M of them, 28 edges each on average) about 690 warp instructions
// instead of 1,250, and the kernel takes 1.95 ms instead of 4.30.
constexpr int kPlanes = 6;
constexpr int kSubWords = kPlanes * 32;         // one sample row
constexpr int kDenseWords = 2 * 16 * 32 + 2 * 32;  // or winding_bits' counters
constexpr int kCovOff = kDenseWords > 4 * kSubWords ? kDenseWords : 4 * kSubWords;  // then 256 coverage bytes
constexpr int kWarpWords = kCovOff + kTileCols / 4;

// An edge as a pixel row's sample rows see it (bin_edge): its crossing with
// sample row r of the pixel row is c0 + round(v0 + fxi r).
struct RowEdge {
    float v0, fxi, lim;
    int32_t c0;        // xi - (tile's first sample column) - the bits of 1.5 * 2^23
    int32_t id;
    uint32_t rows;     // sample rows on which the edge is active
    bool down;
};
// Bin entry `bin` for the pixel row whose sc sample rows begin at row `off` of
// the band's.  What does not depend on the pixel row is in the record: a
// record is read by every row and tile column of its band (2,000 paths: with
// rows, t and limit worked out here 2.07 ms, with the record 1.97).
// (Tables in global memory are read through the read-only path.)
template <int BINS, class T>
__device__ __forceinline__ T table(const T *p) {
    if constexpr (BINS == kBinShared) return *p;
    else return __ldg(p);
}
template <int BINS>
constexpr bool kSmallEdges = BINS == kBinSmall || BINS == kBinShared;
template <int BINS>
__device__ __forceinline__ RowEdge row_edge(const void *__restrict__ bins, const void *__restrict__ edges,
                                            int32_t bin, bool valid, int32_t sub0, int32_t off, int32_t sc,
                                            int32_t col0) {
    RowEdge R{};
    if (!valid) return R;
    BinEdge B;
    if constexpr (kSmallEdges<BINS>) {
        const int32_t id = table<BINS>(reinterpret_cast<const int32_t *>(bins) + bin);
        const int4 a = table<BINS>(reinterpret_cast<const int4 *>(edges) + 2 * (size_t)id);
        const int4 b = table<BINS>(reinterpret_cast<const int4 *>(edges) + 2 * (size_t)id + 1);
        DEdge e;
        e.x_start = __hiloint2double(a.y, a.x);
        e.x_inc = __hiloint2double(a.w, a.z);
        e.top = __hiloint2double(b.y, b.x);
        edge_fields(e, (b.w & 1) != 0);
        B = bin_edge(e.xi, e.fx, e.fxi, e.fdt, b.z, b.w >> 1, id, sub0 - off, kTileRows * sc);
    } else if constexpr (BINS == kBinIndex) {
        const int32_t id = __ldg(reinterpret_cast<const int32_t *>(bins) + bin);
        const DEdge *e = reinterpret_cast<const DEdge *>(edges) + id;
        const int4 a = __ldg(reinterpret_cast<const int4 *>(e));
        const int2 b = __ldg(reinterpret_cast<const int2 *>(&e->rt));
        B = bin_edge(a.x, __int_as_float(a.y), __int_as_float(a.z), __int_as_float(a.w), b.x, b.y, id, sub0 - off,
                     kTileRows * sc);
    } else {
        const int4 a = __ldg(reinterpret_cast<const int4 *>(bins) + 2 * (size_t)bin);
        const int4 b = __ldg(reinterpret_cast<const int4 *>(bins) + 2 * (size_t)bin + 1);
        B = BinEdge{a.x, __int_as_float(a.y), __int_as_float(a.z), __int_as_float(a.w), (uint32_t)b.x,
                    __int_as_float(b.y), b.z, 0};
    }
    R.id = B.id;
    R.rows = (B.rows >> off) & ((1u << sc) - 1u);
    R.down = (int32_t)B.rows < 0;
    R.fxi = B.fxi;
    R.v0 = __fmaf_rn(B.fxi, B.t + (float)off, B.fx);
    R.lim = B.limit;
    R.c0 = B.c - col0;
    return R;
}

// The reference's evaluation, out of line: needed for one crossing in
// thousands, and four copies of it in the crossing loop would be most of the
// loop's code.
static __device__ __noinline__ int32_t crossing_f64(double x_start, double x_inc, double top, int32_t sr) {
    return (int32_t)round(x_start + (x_inc * (((double)sr + 0.5) - top)));
}

// Sample column, relative to the tile's first, where edge R crosses sample
// row sub0 + r (r one of R.rows).
template <int BINS>
__device__ __forceinline__ int32_t edge_crossing(const void *__restrict__ edges, const RowEdge &R, int32_t r,
                                                 int32_t sub0, int32_t col0) {
    int32_t n;
    if (crossing_f32(R.v0, R.fxi, (float)r, R.lim, n)) return n + R.c0;
    using E = std::conditional_t<kSmallEdges<BINS>, SmallEdge, DEdge>;
    const E *e = reinterpret_cast<const E *>(edges) + R.id;
    return crossing_f64(e->x_start, e->x_inc, e->top, sub0 + r) - col0;
}

// Inside bits of the lane's columns on the row's sample rows by the non-zero
// rule, for any number of crossings per column: two sample rows at a time,
// with biased 16-bit counters per column (two a word; at most
// kMaxBandEdges < 2^15 crossings, so no half carries) in `words`, which is
// clear before and after.  For rows where four crossings of one direction
// share a sample column, and without trying the planes first for
// kDenseEdges edges and more: of 320 surfaces with fills and strokes, 12 % of
// the non-zero rows with 128-256 edges in their band run over the planes,
// 56 % of those with 256-512 and 90 % of those with more (strokes drawn over
// themselves, paths much smaller than their detail).  Out of line, for the
// registers of the common path.
constexpr int32_t kDenseEdges = 256;
template <int BINS>
static __device__ __noinline__ uint4 winding_bits(const void *bins, const void *edges, int32_t e0, int32_t ne,
                                                  int32_t sub0, int32_t off, int32_t sc, int32_t col0, uint32_t *words,
                                                  int lane) {
    constexpr uint32_t kBias2 = 0x80008000u;
    constexpr int kRow = 16 * 32;              // a sample row's counters
    uint32_t *touch = words + 2 * kRow;        // column pairs touched, per sample row and lane
    const int32_t lg_per = sc == 1 ? 3 : 5, per = 1 << lg_per;
    uint32_t out[4] = {0u, 0u, 0u, 0u};
    __syncwarp();
    for (int i = lane; i < 2 * kRow; i += 32) words[i] = kBias2;
    __syncwarp();
#pragma unroll
    for (int s0 = 0; s0 < 4; s0 += 2) {
        if (s0 >= sc) break;
        int32_t left = 0;  // rows s0 and s0 + 1 as lo + 65536 hi
        for (int32_t base = 0; base < ne; base += 32) {
            const RowEdge R = row_edge<BINS>(bins, edges, e0 + base + lane, base + lane < ne, sub0, off, sc, col0);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (!((R.rows >> (s0 + h)) & 1u)) continue;
                const int32_t c = edge_crossing<BINS>(edges, R, s0 + h, sub0, col0);
                if (c <= 0) {
                    left += R.down ? (h ? -65536 : -1) : (h ? 65536 : 1);
                } else if (c < 32 * per) {
                    // a lane's pairs of columns lie 32 words apart: every
                    // lane reads its own bank
                    const int32_t pair = (c & (per - 1)) >> 1, own = c >> lg_per;
                    const uint32_t d = R.down ? 0xFFFFFFFFu : 1u;
                    atomicAdd(&words[h * kRow + ((pair << 5) | own)], (c & 1) ? d << 16 : d);
                    atomicOr(&touch[h * 32 + own], 1u << pair);
                }
            }
        }
        left = __reduce_add_sync(0xffffffffu, left);
        __syncwarp();
        int32_t tot[2];
        uint32_t pairs[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            pairs[h] = touch[h * 32 + lane];
            touch[h * 32 + lane] = 0u;
            tot[h] = 0;
            for (uint32_t m = pairs[h]; m; m &= m - 1) {
                const uint32_t v = words[h * kRow + (__ffs(m) - 1) * 32 + lane];
                tot[h] += (int32_t)(v & 0xFFFFu) + (int32_t)(v >> 16) - 0x10000;
            }
        }
        const int32_t t = tot[0] + tot[1] * 65536;
        int32_t incl = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        incl += left - t;
        const int32_t lo = (int32_t)(int16_t)(incl & 0xFFFF);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            int32_t wnd = h ? (incl - lo) >> 16 : lo;
            uint32_t bits = wnd != 0 ? 0xFFFFFFFFu : 0u;
            for (uint32_t m = pairs[h]; m; m &= m - 1) {
                const int k = __ffs(m) - 1;
                uint32_t *w = words + h * kRow + k * 32 + lane;
                const uint32_t v = *w;
                *w = kBias2;
                bool was = wnd != 0;
                wnd += (int32_t)(v & 0xFFFFu) - 0x8000;
                if ((wnd != 0) != was) bits ^= 0xFFFFFFFFu << (2 * k);
                was = wnd != 0;
                wnd += (int32_t)(v >> 16) - 0x8000;
                if ((wnd != 0) != was) bits ^= 0xFFFFFFFEu << (2 * k);
            }
            out[s0 + h] = bits;
        }
        __syncwarp();
    }
    for (int i = lane; i < 2 * kRow; i += 32) words[i] = 0u;
    __syncwarp();
    return make_uint4(out[0], out[1], out[2], out[3]);
}

// The alpha formats' pixel access and src_over, out of line: the 4-byte
// formats' loops stay small.
static __device__ __noinline__ uint32_t load_alpha(uint8_t *data, int fmt, size_t i) {
    return load_raw(DevSurface{data, fmt, 0, 0}, i);
}
static __device__ __noinline__ void store_alpha(uint8_t *data, int fmt, size_t i, uint32_t v) {
    store_raw(DevSurface{data, fmt, 0, 0}, i, v);
}
static __device__ __noinline__ uint32_t alpha_src_over(uint32_t raw, uint32_t sa, int fmt) {
    const uint32_t da = raw_to_i16(raw, fmt).a;
    return i16_to_raw(I16{0, 0, 0, sa + da - (sa * da) / 255u}, fmt);
}

// One work item is one pixel row of a tile of 4 rows x 256 pixels.  The warp
// walks the band's fills in call order: the fill's crossings with the row's
// 4 (or 1) sample rows go to the planes, where lane l owns the 32 (or 8)
// sample columns of pixels [8l, 8l+8); it turns them into inside bits and
// coverage, which pass through shared memory to the lanes that composite:
// lane l holds pixels l, l + 32, ..., l + 224 of the row in registers from
// the first fill to the last.  A block of 32 consecutive pixels that the fill
// leaves uncovered is skipped by the whole warp, and loads and stores are
// coalesced.  `words` is the warp's own shared-memory scratch.
// MULTI = false draws a one-surface batch from A.job0, whose fields are
// kernel parameters (warp-uniform values that need no registers);
// MULTI = true finds the tile's job in the job table.
template <bool MULTI, int MODE, int BINS>
__device__ __forceinline__ void raster_row(const RasterArgs &A, const int32_t tile, const int warp, const int lane,
                                           uint32_t *words) {
    // tile -> (job, band, tile column)
    int32_t jb = 0, lb, col;
    if constexpr (MULTI) {
        const int4 t = table<BINS>(reinterpret_cast<const int4 *>(A.tiles + tile));
        jb = t.x;
        lb = t.y;
        col = t.z;
    } else {
        const int32_t ncols = A.job0.tcol_hi - A.job0.tcol_lo + 1;
        lb = tile / ncols;
        col = tile - lb * ncols;
    }
    const DevJob &JB = MULTI ? A.jobs[jb] : A.job0;
    const int32_t b = JB.band_lo + lb;
    const int32_t cnt = A.band_count[JB.gband_base + lb];
    if (cnt == 0) return;
    const int32_t x0 = (JB.tcol_lo + col) * kTileCols, y = b * kTileRows + warp;
    const int32_t W = JB.sfc.w, H = JB.sfc.h, fmt = JB.sfc.fmt;
    if (y >= H) return;
    const int4 *list = A.band_fills + JB.list_base + (long long)lb * (JB.fill1 - JB.fill0);
    const int32_t px0 = x0 + lane;  // this lane's first pixel; the others follow 32 apart
    constexpr uint32_t kAll = 0xffffffffu;
    constexpr bool PLAIN = MODE != kGeneral;
    // The loops over sample rows are unrolled in the plain variant, where they
    // are the kernel's work (2,000 paths then 2.41 ms, not unrolled 2.70), not in
    // the general one, where every warp is at another place of a large
    // program and waits for instructions (240 gradient fills 0.78 ms, unrolled
    // 1.05).  What a loop needs rarely is out of line for the same
    // reason: with it inline the plain kernel had 86 KB of code instead of 61
    // and 320 surfaces with strokes took 5.1 ms instead of 3.9.
    const uint32_t below = (1u << lane) - 1u;  // the lanes before this one

    for (int i = lane; i < kCovOff; i += 32) words[i] = 0u;
    uint32_t raw[8];
    // This lane's pixels that some fill has drawn, a bit per block: only those
    // are stored.  (Their neighbours may be another stream's to draw: a block
    // stored whole would put back what it held when this row began.)
    uint32_t touched = 0;
    {
        const DevSurface dst = JB.sfc;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            raw[q] = 0u;
            if (px0 + 32 * q >= W) continue;
            const size_t at = (size_t)W * y + px0 + 32 * q;
            raw[q] = fmt <= Z2D_FORMAT_RGBA ? reinterpret_cast<const uint32_t *>(dst.data)[at] : load_alpha(dst.data, fmt, at);
        }
    }
    __syncwarp();

    // The band's fill list is read 32 entries at a time, one per lane.  Each
    // lane also loads its fill's record and edge range and tests them, so
    // that the fills that matter to this row are known, with their
    // records in registers, before the first of them is drawn.
    for (int32_t k0 = 0; k0 < cnt; k0 += 32) {
        int32_t my_f = 0, my_e0 = 0, my_ne = 0;
        uint32_t my_meta = 0, my_box = 0;
        bool hit = false;
        if (k0 + lane < cnt) {
            const int4 ent = list[k0 + lane];
            if (ent.z > x0 && ent.y < x0 + kTileCols) {
                const int4 ra = table<BINS>(reinterpret_cast<const int4 *>(A.rfills + ent.x));
                const uint32_t rb = table<BINS>(&A.rfills[ent.x].meta);
                my_e0 = table<BINS>(A.bin_off + ent.w);
                my_ne = table<BINS>(A.bin_off + ent.w + 1) - my_e0;
                my_f = ent.x;
                my_meta = rb;
                const int32_t aa = (int32_t)((my_meta >> RF_AA_SHIFT) & 3u);
                const bool bounded = (my_meta & RF_BOUNDED) != 0;
                const bool boxed = bounded || aa == Z2D_AA_SUPERSAMPLE_4X;  // touches only its box
                const bool in_rows = y >= ra.z && y <= ra.w;
                hit = !boxed || (in_rows && ra.y > x0 && ra.x < x0 + kTileCols);
                // no edge in the band: nothing is covered, and a bounded
                // operator draws nothing (see the same test below)
                if (PLAIN ? my_ne == 0 || (my_meta & RF_SS_ZERO)
                          : bounded && my_ne == 0 && !(my_meta & (RF_EXACT | RF_SS_ZERO)))
                    hit = false;
                if (in_rows) my_meta |= RF_IN_ROWS;
                // the box's columns within the tile
                const int32_t xhi = aa == Z2D_AA_NONE ? W : min(ra.y, W);
                my_box = (uint32_t)max(0, min(ra.x - x0, kTileCols)) |
                         ((uint32_t)max(0, min(xhi - x0, kTileCols)) << 16);
            }
        }
        for (uint32_t hits = __ballot_sync(kAll, hit); hits; hits &= hits - 1) {
            const int src = __ffs(hits) - 1;
            const uint32_t meta = __shfl_sync(kAll, my_meta, src);
            const int32_t e0 = __shfl_sync(kAll, my_e0, src), ne = __shfl_sync(kAll, my_ne, src);
            const int32_t aa = (int32_t)((meta >> RF_AA_SHIFT) & 3u);
            const bool bounded = PLAIN || (meta & RF_BOUNDED) != 0;
            const bool ssaa = aa == Z2D_AA_SUPERSAMPLE_4X;
            const bool direct = MODE == kPlainDirect || (MODE == kGeneral && aa == Z2D_AA_NONE);
            const bool exact = !PLAIN && (meta & RF_EXACT) != 0;
            const bool in_rows = PLAIN || (meta & RF_IN_ROWS) != 0;
            const int32_t sc = direct ? 1 : 4, per = 8 * sc, lg_per = direct ? 3 : 5;
            uint32_t cov_any = 0;  // lanes with a covered pixel among [8l, 8l+8)
            if (PLAIN || (!exact && in_rows && !(meta & RF_SS_ZERO))) {
                const int32_t sub0 = y * sc, off = warp * sc, col0 = x0 * sc, ncol = kTileCols * sc;
                const bool eo = (meta & RF_EVEN_ODD) != 0;
                // One edge per lane.  Crossings at or left of the tile's
                // first sample column all count from column 0: they are
                // summed per sample row (rows 0, 1 and 2, 3 packed as
                // lo + 65536 hi: every sum is at most kMaxBandEdges < 2^15
                // in magnitude, so the halves stay apart).
                int32_t l01 = 0, l23 = 0;
                uint32_t flags = 0;  // 1: a crossing in the tile, 2: a second of its column, 4: a fourth
                const bool dense = !eo && ne >= kDenseEdges;
                if (dense) flags = 4u;
                for (int32_t base = dense ? ne : 0; base < ne; base += 32) {
                    const RowEdge R = row_edge<BINS>(A.bins, A.edges, e0 + base + lane, base + lane < ne, sub0, off, sc, col0);
                    auto cross = [&](int r) {
                        if (!((R.rows >> r) & 1u)) return;
                        const int32_t c = edge_crossing<BINS>(A.edges, R, r, sub0, col0);
                        if (c <= 0) {
                            const int32_t d = R.down ? -1 : 1;
                            if (r < 2) l01 += r == 0 ? d : d * 65536;
                            else l23 += r == 2 ? d : d * 65536;
                        } else if (c < ncol) {
                            uint32_t *w = words + r * kSubWords + (c >> lg_per);
                            const uint32_t bit = 1u << (c & (per - 1));
                            flags |= 1u;
                            if (eo) {
                                atomicXor(w, bit);
                            } else {
                                if (R.down) w += 32;
                                if (atomicOr(w, bit) & bit) {
                                    flags |= 2u;
                                    if ((atomicOr(w + 64, bit) & bit) && (atomicOr(w + 128, bit) & bit)) flags |= 4u;
                                }
                            }
                        }
                    };
                    if constexpr (PLAIN) {
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            if (r >= sc) break;
                            cross(r);
                        }
                    } else {
#pragma unroll 1
                        for (int r = 0; r < sc; r++) cross(r);
                    }
                }
                __syncwarp();
                flags = __reduce_or_sync(kAll, flags);
                l01 = __reduce_add_sync(kAll, l01);
                l23 = __reduce_add_sync(kAll, l23);
                // no crossing in the tile and none left of it in balance: the
                // winding is 0 across the tile, nothing is covered
                if (flags == 0 && l01 == 0 && l23 == 0) {
                    if (bounded) continue;  // zero coverage draws nothing
                    goto composite;         // unbounded operators still clear
                }
                {
                // coverage of pixel q (0..16) of the lane's [8l, 8l+8) is byte
                // q / 2 of cov_ev (q even) or cov_od (q odd)
                uint32_t cov_ev = 0, cov_od = 0;
                if constexpr (PLAIN) {
                int32_t wl[4];  // winding left of the lane's columns (even-odd: its parity)
                wl[0] = (int32_t)(int16_t)(l01 & 0xFFFF);
                wl[1] = (l01 - wl[0]) >> 16;
                wl[2] = (int32_t)(int16_t)(l23 & 0xFFFF);
                wl[3] = (l23 - wl[2]) >> 16;
                uint32_t in[4] = {0u, 0u, 0u, 0u};  // inside bits of the lane's columns per sample row
                if (eo) {
#pragma unroll
                    for (int s = 0; s < 4; s++) {
                        if (s >= sc) break;
                        uint32_t *w = words + s * kSubWords + lane;
                        uint32_t t = *w;
                        *w = 0u;
                        // the crossings of the lanes before this one, and of
                        // the columns left of the tile
                        const uint32_t odd = __ballot_sync(kAll, __popc(t) & 1);
                        const uint32_t first = (uint32_t)(__popc(odd & below) + wl[s]) & 1u;
                        t ^= t << 1;
                        t ^= t << 2;
                        t ^= t << 4;
                        t ^= t << 8;
                        t ^= t << 16;
                        in[s] = t ^ (0u - first);
                    }
                } else if (flags & 4u) {
                    if (!dense) {  // clear the planes
                        for (int i = lane; i < 4 * kSubWords; i += 32) words[i] = 0u;
                    }
                    const uint4 v = winding_bits<BINS>(A.bins, A.edges, e0, ne, sub0, off, sc, col0, words, lane);
                    in[0] = v.x;
                    in[1] = v.y;
                    in[2] = v.z;
                    in[3] = v.w;
                } else {
                    uint32_t up[4], dn[4];
                    int32_t tot[4] = {0, 0, 0, 0};  // the lane's winding change
#pragma unroll
                    for (int s = 0; s < 4; s++) {
                        if (s >= sc) break;
                        uint32_t *w = words + s * kSubWords + lane;
                        up[s] = w[0];
                        dn[s] = w[32];
                        w[0] = 0u;
                        w[32] = 0u;
                        tot[s] = __popc(up[s]) - __popc(dn[s]);
                        if (flags & 2u) tot[s] += __popc(w[64]) + __popc(w[128]) - __popc(w[96]) - __popc(w[160]);
                    }
                    const int32_t t01 = tot[0] + tot[1] * 65536, t23 = tot[2] + tot[3] * 65536;
                    int32_t i01 = t01, i23 = t23;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int32_t u01 = __shfl_up_sync(kAll, i01, o);
                        const int32_t u23 = __shfl_up_sync(kAll, i23, o);
                        if (lane >= o) {
                            i01 += u01;
                            i23 += u23;
                        }
                    }
                    i01 += l01 - t01;
                    i23 += l23 - t23;
                    wl[0] = (int32_t)(int16_t)(i01 & 0xFFFF);
                    wl[1] = (i01 - wl[0]) >> 16;
                    wl[2] = (int32_t)(int16_t)(i23 & 0xFFFF);
                    wl[3] = (i23 - wl[2]) >> 16;
#pragma unroll
                    for (int s = 0; s < 4; s++) {
                        if (s >= sc) break;
                        // the inside state changes where the winding leaves
                        // or reaches zero
                        int32_t wnd = wl[s];
                        uint32_t bits = wnd != 0 ? 0xFFFFFFFFu : 0u;
                        if (flags & 2u) {
                            uint32_t *w = words + s * kSubWords + lane;
                            const uint32_t u1 = w[64], d1 = w[96], u2 = w[128], d2 = w[160];
                            w[64] = w[96] = w[128] = w[160] = 0u;
                            for (uint32_t m = up[s] | dn[s]; m; m &= m - 1) {
                                const uint32_t k = m & (0u - m);  // the next column's bit
                                const uint32_t was = wnd != 0 ? 0xFFFFFFFFu : 0u;
                                wnd += (up[s] & k ? 1 : 0) + (u1 & k ? 1 : 0) + (u2 & k ? 1 : 0) - (dn[s] & k ? 1 : 0) -
                                       (d1 & k ? 1 : 0) - (d2 & k ? 1 : 0);
                                bits ^= (was ^ (wnd != 0 ? 0xFFFFFFFFu : 0u)) & (0u - k);
                            }
                        } else {
                            for (uint32_t m = up[s] | dn[s]; m; m &= m - 1) {
                                const uint32_t k = m & (0u - m);
                                const uint32_t was = wnd != 0 ? 0xFFFFFFFFu : 0u;
                                wnd += (up[s] & k ? 1 : 0) - (dn[s] & k ? 1 : 0);
                                bits ^= (was ^ (wnd != 0 ? 0xFFFFFFFFu : 0u)) & (0u - k);
                            }
                        }
                        in[s] = bits;
                    }
                }
                if (direct) {  // one sample row: bit q is pixel q's sample
#pragma unroll
                    for (int q = 0; q < 8; q += 2) {
                        cov_ev |= ((in[0] >> q) & 1u) << (4 * q);
                        cov_od |= ((in[0] >> (q + 1)) & 1u) << (4 * q);
                    }
                } else {
#pragma unroll
                    for (int s = 0; s < 4; s++) {  // nibble q holds pixel q's 4 samples of a row
                        uint32_t n = in[s] - ((in[s] >> 1) & 0x55555555u);
                        n = (n & 0x33333333u) + ((n >> 2) & 0x33333333u);
                        cov_ev += n & 0x0F0F0F0Fu;
                        cov_od += (n >> 4) & 0x0F0F0F0Fu;
                    }
                }
                } else {
                auto cover = [&](uint32_t bits) {
                    if (direct) {  // one sample row: bit q is pixel q's sample
                        cov_ev = (bits & 1u) | ((bits & 4u) << 6) | ((bits & 16u) << 12) | ((bits & 64u) << 18);
                        bits >>= 1;
                        cov_od = (bits & 1u) | ((bits & 4u) << 6) | ((bits & 16u) << 12) | ((bits & 64u) << 18);
                    } else {  // nibble q holds pixel q's 4 samples of this row
                        uint32_t n = bits - ((bits >> 1) & 0x55555555u);
                        n = (n & 0x33333333u) + ((n >> 2) & 0x33333333u);
                        cov_ev += n & 0x0F0F0F0Fu;
                        cov_od += (n >> 4) & 0x0F0F0F0Fu;
                    }
                };
                // winding (even-odd: its parity) left of the lane's columns,
                // rows 0, 1 and 2, 3 packed
                int32_t i01 = l01, i23 = l23;
                uint4 counted = make_uint4(0u, 0u, 0u, 0u);
                if (flags & 4u) {
                    if (!dense) {  // clear the planes
                        for (int i = lane; i < 4 * kSubWords; i += 32) words[i] = 0u;
                    }
                    counted = winding_bits<BINS>(A.bins, A.edges, e0, ne, sub0, off, sc, col0, words, lane);
                } else if (!eo) {
                    int32_t tot[4] = {0, 0, 0, 0};  // the lane's winding change
#pragma unroll
                    for (int s = 0; s < 4; s++) {
                        if (s >= sc) break;
                        const uint32_t *w = words + s * kSubWords + lane;
                        tot[s] = __popc(w[0]) - __popc(w[32]);
                        if (flags & 2u) tot[s] += __popc(w[64]) + __popc(w[128]) - __popc(w[96]) - __popc(w[160]);
                    }
                    const int32_t t01 = tot[0] + tot[1] * 65536, t23 = tot[2] + tot[3] * 65536;
                    i01 = t01;
                    i23 = t23;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int32_t u01 = __shfl_up_sync(kAll, i01, o);
                        const int32_t u23 = __shfl_up_sync(kAll, i23, o);
                        if (lane >= o) {
                            i01 += u01;
                            i23 += u23;
                        }
                    }
                    i01 += l01 - t01;
                    i23 += l23 - t23;
                }
                auto left_of = [&](int s) -> int32_t {
                    const int32_t pair = s < 2 ? i01 : i23, low = (int32_t)(int16_t)(pair & 0xFFFF);
                    return (s & 1) ? (pair - low) >> 16 : low;
                };
                if (eo) {
#pragma unroll 1
                    for (int s = 0; s < 4; s++) {
                        if (s >= sc) break;
                        uint32_t *w = words + s * kSubWords + lane;
                        uint32_t t = *w;
                        *w = 0u;
                        // the crossings of the lanes before this one, and of
                        // the columns left of the tile
                        const uint32_t odd = __ballot_sync(kAll, __popc(t) & 1);
                        const uint32_t first = (uint32_t)(__popc(odd & below) + left_of(s)) & 1u;
                        t ^= t << 1;
                        t ^= t << 2;
                        t ^= t << 4;
                        t ^= t << 8;
                        t ^= t << 16;
                        cover(t ^ (0u - first));
                    }
                } else if (flags & 4u) {
                    cover(counted.x);
                    if (!direct) {
                        cover(counted.y);
                        cover(counted.z);
                        cover(counted.w);
                    }
                } else {
#pragma unroll 1
                    for (int s = 0; s < 4; s++) {
                        if (s >= sc) break;
                        // the inside state changes where the winding leaves
                        // or reaches zero
                        uint32_t *w = words + s * kSubWords + lane;
                        const uint32_t up = w[0], dn = w[32];
                        w[0] = w[32] = 0u;
                        int32_t wnd = left_of(s);
                        uint32_t bits = wnd != 0 ? 0xFFFFFFFFu : 0u;
                        if (flags & 2u) {
                            const uint32_t u1 = w[64], d1 = w[96], u2 = w[128], d2 = w[160];
                            w[64] = w[96] = w[128] = w[160] = 0u;
                            for (uint32_t m = up | dn; m; m &= m - 1) {
                                const int k = __ffs(m) - 1;
                                const bool was = wnd != 0;
                                wnd += (int32_t)(((up >> k) & 1u) + ((u1 >> k) & 1u) + ((u2 >> k) & 1u)) -
                                       (int32_t)(((dn >> k) & 1u) + ((d1 >> k) & 1u) + ((d2 >> k) & 1u));
                                if ((wnd != 0) != was) bits ^= 0xFFFFFFFFu << k;
                            }
                        } else {
                            for (uint32_t m = up | dn; m; m &= m - 1) {
                                const int k = __ffs(m) - 1;
                                const bool was = wnd != 0;
                                wnd += (int32_t)((up >> k) & 1u) - (int32_t)((dn >> k) & 1u);
                                if ((wnd != 0) != was) bits ^= 0xFFFFFFFFu << k;
                            }
                        }
                        cover(bits);
                    }
                }
                }
                // only the box's columns are drawn
                const uint32_t box = __shfl_sync(kAll, my_box, src);
                if (box != ((uint32_t)kTileCols << 16)) {
                    const int lo = (int)(box & 0xFFFFu) - 8 * lane, hi = (int)(box >> 16) - 8 * lane;
                    uint32_t m = hi >= 8 ? 0xFFu : hi <= 0 ? 0u : (1u << hi) - 1u;
                    if (lo > 0) m &= lo >= 8 ? 0u : 0xFFu << lo;
                    if (m != 0xFFu) {
                        // bit q of m -> byte q / 2 of the even or odd bytes
                        const uint32_t ev = m & 0x55u, od = (m >> 1) & 0x55u;
                        cov_ev &= (((ev & 1u) | ((ev & 4u) << 6) | ((ev & 16u) << 12) | ((ev & 64u) << 18))) * 0xFFu;
                        cov_od &= (((od & 1u) | ((od & 4u) << 6) | ((od & 16u) << 12) | ((od & 64u) << 18))) * 0xFFu;
                    }
                }
                cov_any = __ballot_sync(kAll, (cov_ev | cov_od) != 0u);
                reinterpret_cast<uint2 *>(words + kCovOff)[lane] =
                    make_uint2(__byte_perm(cov_ev, cov_od, 0x5140), __byte_perm(cov_ev, cov_od, 0x7362));
                // the planes are clear again and the coverage is written
                __syncwarp();
                }
            }
        composite:
            // coverage of this lane's pixel of block q; blocks whose bit of
            // `blocks` is clear are uncovered (the coverage bytes are written
            // only where some lane has coverage)
            uint32_t blocks = 0;
            if (cov_any) {
#pragma unroll
                for (int q = 0; q < 8; q++) blocks |= ((cov_any >> (4 * q)) & 0xFu ? 1u : 0u) << q;
            }
            const uint8_t *cov = reinterpret_cast<const uint8_t *>(words + kCovOff) + lane;
            if (PLAIN || (((meta >> RF_FAST_SHIFT) & 3u) == FAST_PIXEL_SRC_OVER && !exact && bounded)) {
                // Pixel source, integer src_over: the compositeOpaque /
                // compositeOpacity paths reduce to src_over(d, pixel) at full
                // coverage and src_over(d, dst_in(pixel, opacity)) otherwise.
                // The supersample batch [dst_in(pixel, mask), src_over] is the
                // same with the downsampled mask value as opacity; at zero
                // coverage both leave the pixel as it is.
                // (A bounded fill outside its rows was skipped above.)
                if (!blocks) continue;
                // Lane k holds the source word for coverage k (k_edge_fill).
                const uint32_t lut_w = table<BINS>(A.luts + 32 * (size_t)__shfl_sync(kAll, my_f, src) + lane);
                if (fmt <= Z2D_FORMAT_RGBA) {
                    const bool has_alpha = fmt == Z2D_FORMAT_RGBA || fmt == Z2D_FORMAT_ARGB;
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        if (!((blocks >> q) & 1u)) continue;
                        const int c = cov[32 * q];
                        const uint32_t L = __shfl_sync(kAll, lut_w, c);
                        const uint32_t nv = word_src_over_fma(raw[q], L, has_alpha);
                        raw[q] = c != 0 ? nv : raw[q];
                        touched |= c != 0 ? 1u << q : 0u;
                    }
                } else {  // alpha formats: the alpha lane of src_over alone
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        if (!((blocks >> q) & 1u)) continue;
                        const int c = cov[32 * q];
                        const uint32_t sa = __shfl_sync(kAll, lut_w, c);
                        if (c == 0) continue;
                        raw[q] = alpha_src_over(raw[q], sa, fmt);
                        touched |= 1u << q;
                    }
                }
                continue;
            }
            if constexpr (!PLAIN) {
            const int32_t f = __shfl_sync(kAll, my_f, src);
            const FillState &S = A.st[f];
            const FillCmd &F = A.fills[f];
            const bool has_alpha = fmt == Z2D_FORMAT_RGBA || fmt == Z2D_FORMAT_ARGB;
            if (((meta >> RF_FAST_SHIFT) & 3u) == FAST_SOURCE_SRC_OVER && !exact && fmt <= Z2D_FORMAT_RGBA &&
                (!ssaa || has_alpha)) {
                // A gradient or dither drawn by integer src_over.  A source
                // pixel costs hundreds of instructions, so the covered
                // pixels of the whole row are listed first and evaluated 32 at
                // a time, whatever block they lie in.  (Supersampled, a
                // pixel without coverage composites a clear source: without
                // an alpha channel that would still rewrite its padding byte.)
                if (!blocks) continue;
                // the planes, clear at this point, hold the colours and the
                // list
                uint8_t *at = reinterpret_cast<uint8_t *>(words + kTileCols);
                int n = 0;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    if (!((blocks >> q) & 1u)) continue;
                    const bool on = cov[32 * q] != 0;
                    const uint32_t m = __ballot_sync(kAll, on);
                    if (on) at[n + __popc(m & below)] = (uint8_t)(32 * q + lane);
                    touched |= on ? 1u << q : 0u;
                    n += __popc(m);
                }
                __syncwarp();
                auto word_at = [&](int p, I16 s) {
                    const int c = reinterpret_cast<const uint8_t *>(words + kCovOff)[p];
                    const uint32_t op8 = ssaa ? ss_mask8(c, fmt) : c >= (direct ? 1 : 16) ? 255u : (uint32_t)(c * 16 - 1);
                    words[p] = source_word(s, op8, fmt);
                };
                // in f32 first; what that does not decide goes to the front
                // of the list (behind the reads) and is evaluated exactly
                int late = 0;
                for (int i0 = 0; i0 < n; i0 += 32) {
                    const bool live = i0 + lane < n;
                    const int p = live ? at[i0 + lane] : 0;
                    I16 s;
                    const bool ok = live && src_i16_f32(F.src, x0 + p, y, s);
                    if (ok) word_at(p, s);
                    const uint32_t m = __ballot_sync(kAll, live && !ok);
                    if (live && !ok) at[late + __popc(m & below)] = (uint8_t)p;
                    late += __popc(m);
                    __syncwarp();
                }
                for (int i = lane; i < late; i += 32) {
                    const int p = at[i];
                    word_at(p, src_i16_slow(F.src, x0 + p, y, 0));
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    if (!((blocks >> q) & 1u)) continue;
                    if (cov[32 * q] != 0) raw[q] = word_src_over_fma(raw[q], words[32 * q + lane], has_alpha);
                }
                __syncwarp();
                for (int i = lane; i < kTileCols + kTileCols / 4; i += 32) words[i] = 0u;
                __syncwarp();
                continue;
            }
            // with a bounded operator only covered pixels are drawn
            const bool sparse = bounded && !ssaa && !exact;
#pragma unroll 1
            for (int q = 0; q < 8; q++) {
                const bool some = (blocks >> q) & 1u;
                if (sparse && !some) continue;
                const int32_t x = px0 + 32 * q;
                // raw[] is read and written with constant indices only, so it
                // stays in registers
                uint32_t rq = raw[0];
#pragma unroll
                for (int j = 1; j < 8; j++)
                    if (q == j) rq = raw[j];
                int c = some ? cov[32 * q] : 0;
                bool on;
                if (ssaa) {
                    // every pixel of the composite region runs the batch
                    // [dst_in(pattern, mask), op] (supersample.zig:171-184)
                    on = x < W && x >= S.start_x && x < S.end_x;
                    if (on) {
                        if (exact && x >= S.mask_x0 && x < S.mask_x0 + S.mask_w)
                            c = A.masks[S.mask_base + (long long)(y - S.start_y) * S.mask_w + (x - S.mask_x0)] & 0x1F;
                        rq = i16_to_raw(apply_ssaa(F, x, y, ss_mask8(c, fmt), raw_to_i16(rq, fmt)), fmt);
                    }
                } else {
                    bool clear = false;
                    if (exact && in_rows && x >= S.mask_x0 && x < S.mask_x0 + S.mask_w) {
                        const uint8_t m = A.masks[S.mask_base + (long long)(y - S.start_y) * S.mask_w + (x - S.mask_x0)];
                        c = m & 0x1F;
                        if (direct) clear = (m & kMaskClear) != 0;
                    }
                    if (!direct && !bounded) clear = msaa_unbounded_clear(S, x, y, W);
                    const bool in_box = in_rows && (direct ? true : (x >= S.start_x && x < S.end_x));
                    on = x < W && (clear || (in_box && c > 0));
                    if (on) {
                        I16 d = clear ? normalize(I16{0, 0, 0, 0}, fmt) : raw_to_i16(rq, fmt);
                        if (in_box && c > 0) d = apply_fill(F, fmt, x, y, c, direct ? 1 : 16, d);
                        rq = i16_to_raw(d, fmt);
                    }
                }
                if (!__any_sync(kAll, on)) continue;
                touched |= on ? 1u << q : 0u;
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (q == j) raw[j] = rq;
            }
            }
        }
    }
    // the surface pointer is read again here rather than kept in registers
    // through the fill loop
    uint8_t *data = MULTI ? *reinterpret_cast<uint8_t *const volatile *>(&A.jobs[jb].sfc.data) : A.job0.sfc.data;
#pragma unroll
    for (int q = 0; q < 8; q++)
        if (((touched >> q) & 1u) && px0 + 32 * q < W) {
            const size_t at = (size_t)W * y + px0 + 32 * q;
            if (fmt <= Z2D_FORMAT_RGBA) reinterpret_cast<uint32_t *>(data)[at] = raw[q];
            else store_alpha(data, fmt, at, raw[q]);
        }
}

// Persistent rasteriser: a grid of resident CTAs that take items from a
// device work queue (one 64-bit counter) until it is empty; tiles are
// queued job after job, or in the order of A.order when given.
//  * CTA_ITEMS: an item is a whole tile; the CTA's four warps draw its four
//    rows and meet at a barrier before the next tile, so the rows share the
//    band's fill list and edges in the SM's L1.
//  * otherwise an item is one (tile, row) pair, numbered tile * 4 + row,
//    taken by a single warp: a warp that finishes a cheap row takes the
//    next item at once instead of holding its CTA until the slowest warp of
//    the tile is done.
// CTAs per SM: nine of the plain variants for one surface (56 registers;
// 2,000 paths with 7, 8, 9, 10 and 11: 2.08, 1.97, 1.93, 1.95 and 2.09 ms, when
// whole blocks were stored),
// eight for several surfaces (320 surfaces with 7, 8 and 9: 3.14, 3.06 and
// 3.15 ms: the job's fields take registers), six of the general ones (240
// gradient fills with 4, 6 and 8: 0.82, 0.75 and 0.77 ms).
constexpr int raster_ctas(bool multi, int mode, int bins) {
    return mode == kGeneral ? 6 : multi || bins != kBinRecords ? 8 : 9;
}
template <bool MULTI, bool CTA_ITEMS, int MODE, int BINS = kBinRecords>
__global__ void __launch_bounds__(kRasterThreads, raster_ctas(MULTI, MODE, BINS)) k_raster(const RasterArgs A) {
    extern __shared__ uint32_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *words = smem + warp * kWarpWords;
    if constexpr (CTA_ITEMS) {
        __shared__ unsigned long long next_tile;
        for (;;) {
            unsigned long long t = blockIdx.x;  // one_per_tile: a grid of one CTA per tile, dispatched in queue order
            if (!A.one_per_tile) {
                if (threadIdx.x == 0) next_tile = atomicAdd(A.queue, 1ull);
                __syncthreads();
                t = next_tile;
                __syncthreads();  // every thread has read it before it is replaced
                if (t >= A.n_items) break;
            }
            const int32_t tile = A.order ? A.order[t] : (int32_t)t;
            raster_row<MULTI, MODE, BINS>(A, tile, warp, lane, words);
            if (A.one_per_tile) break;
        }
    } else {
        for (;;) {
            unsigned long long item = 0;
            if (lane == 0) item = atomicAdd(A.queue, 1ull);
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= A.n_items) break;
            const long long t = (long long)(item / kTileRows);
            const int32_t tile = A.order ? A.order[t] : (int32_t)t;
            __syncwarp();  // the previous item's reads of `words` are done before it is reset
            raster_row<MULTI, MODE, BINS>(A, tile, (int)(item % kTileRows), lane, words);
        }
    }
}

// A CTA per tile of a small call, whose tables are the launch's parameters: no
// copy, event or staging slot is between the call and its one launch.  Each CTA
// takes them to shared memory first.  Such calls are bound by their CUDA calls
// and by the wait for the tables (the 300x300 star from Python: copied 16.4 us,
// written by a launch of their own in front 13.8, now 11.6).
// Larger tables stay with the copy: a launch's parameters are written by the
// host a second time, read by every CTA, and end at 32 KB.  A call alone and
// waited for: a polygon of 90 segments, just below 8 KB, 27.8 us and copied
// 28.8; of 130, above it, 30.2 and 29.3; of 280 36.3 and 33.5 (among others
// parameters are the faster way for all of them: 13, 14 and 17 us against 17,
// 17.5 and 21).
template <bool MULTI, int MODE>
__global__ void __launch_bounds__(kRasterThreads, raster_ctas(MULTI, MODE, kBinShared))
    k_raster_small(const __grid_constant__ RasterArgs A, const __grid_constant__ ParamBlob P, int32_t n, int32_t n_fills) {
    extern __shared__ uint32_t smem[];
    __shared__ uint4 tables[kParamBytes / sizeof(uint4)];
    for (int32_t i = threadIdx.x; i < n; i += kRasterThreads) tables[i] = P.v[i];
    __syncthreads();
    RasterArgs B = A;
    auto place = [&](auto *&p) {
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(reinterpret_cast<uintptr_t>(tables) +
                                                                  reinterpret_cast<uintptr_t>(p));
    };
    place(B.jobs);
    place(B.fills);
    place(B.st);
    place(B.edges);
    place(B.bins);
    place(B.bin_off);
    place(B.band_count);
    place(B.band_fills);
    place(B.rfills);
    place(B.luts);
    place(B.tiles);
    if constexpr (MODE == kGeneral) {
        for (int32_t f = threadIdx.x; f < n_fills; f += kRasterThreads) {
            FillCmd &F = const_cast<FillCmd &>(B.fills[f]);
            if (F.src.grad) place(F.src.grad);
        }
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    raster_row<MULTI, MODE, kBinShared>(B, (int32_t)blockIdx.x, warp, lane, smem + warp * kWarpWords);
}

static size_t raster_smem() { return sizeof(uint32_t) * kWarpWords * kTileRows; }

template <int MODE, class F>
static int of_mode(RasterVariant v, int k, F &&f) {
    if constexpr (MODE != kPlainDirect)
        if (v.bins == kBinSmall)
            return v.multi ? f(k_raster<true, true, MODE, kBinSmall>, k) : f(k_raster<false, true, MODE, kBinSmall>, k);
    if (v.multi) return v.cta_items ? f(k_raster<true, true, MODE>, k) : f(k_raster<true, false, MODE>, k);
    return v.cta_items ? f(k_raster<false, true, MODE>, k) : f(k_raster<false, false, MODE>, k);
}
template <class F>
static int with_variant(RasterVariant v, F &&f) {
    const int k = (v.mode * 3 + v.bins) * 4 + ((v.multi ? 2 : 0) | (v.cta_items ? 1 : 0));
    if (v.bins == kBinIndex)
        return v.multi ? f(k_raster<true, false, kGeneral, kBinIndex>, k)
                       : f(k_raster<false, false, kGeneral, kBinIndex>, k);
    switch (v.mode) {
        case kPlain4x: return of_mode<kPlain4x>(v, k, f);
        case kPlainDirect: return of_mode<kPlainDirect>(v, k, f);
        default: return of_mode<kGeneral>(v, k, f);
    }
}

// A variant's resident CTAs per SM, asked once per variant.
int raster_occupancy(Ctx &, RasterVariant v, int &ctas_per_sm) {
    static std::atomic<int> cache[36];
    return with_variant(v, [&](auto kernel, int k) -> int {
        int occ = cache[k].load(std::memory_order_relaxed);
        if (occ <= 0) {
            Z2D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kRasterThreads, raster_smem()));
            occ = std::max(occ, 1);
            cache[k].store(occ, std::memory_order_relaxed);
        }
        ctas_per_sm = occ;
        return Z2D_OK;
    });
}

int raster_launch(Ctx &c, RasterVariant v, const RasterArgs &A, unsigned grid) {
    return with_variant(v, [&](auto kernel, int) -> int {
        kernel<<<grid, kRasterThreads, raster_smem(), c.stream>>>(A);
        c.launches++;
        Z2D_CUDA(cudaGetLastError());
        return Z2D_OK;
    });
}

int raster_launch_small(Ctx &c, bool multi, int mode, const RasterArgs &A, const ParamBlob &P, int32_t n, int32_t n_fills,
                        unsigned grid) {
    const auto kernel = mode == kPlain4x ? (multi ? k_raster_small<true, kPlain4x> : k_raster_small<false, kPlain4x>)
                                         : (multi ? k_raster_small<true, kGeneral> : k_raster_small<false, kGeneral>);
    kernel<<<grid, kRasterThreads, raster_smem(), c.stream>>>(A, P, n, n_fills);
    c.launches++;
    Z2D_CUDA(cudaGetLastError());
    return Z2D_OK;
}

}  // namespace z2dg
