// fill.cu -- painter.fill on the GPU, for one fill or an ordered batch of
// fills on one surface.
//
// Pipeline (one launch each, all on the context stream):
//   k_node_count_w  32 nodes per warp: how many edges each line/curve
//                 emits; k_curve_count_w subdivides the curves among them
//                 (Spline.zig:37-165), 1 to 32 lanes a curve
//   stroke_count  device-stroked commands (stroke_gpu.cu): their polygons'
//                 edge counts
//   k_fill_scan   warp per fill: the sequential part of fill_plotter.plot
//                 (fill_plotter.zig:21-97) -- start points, close_path edges,
//                 per-node edge offsets, open-chain detection
//   k_node_emit_w 32 nodes per warp: emits Polygon edges (Polygon.zig:61-109)
//                 and per-fill extents; stroke_emit does the same for the
//                 stroke polygons
//   k_fill_setup  thread per fill: Polygon.inBox and the draw box of
//                 multisample.run / direct.run
//   k_bin_count / k_bin_fill   (edge, 4-row band) lists per fill
//   k_band_lists  CTA or warp per band: the fills touching the band, in call
//                 order
//   k_exact       thread per degenerate fill: literal restatement of the
//                 sorted-span rasteriser, writing a per-pixel action mask
//   k_raster      (raster.cu) per pixel row of a 4x256 tile: for each fill in
//                 order, crossings as bit planes in shared memory, inside
//                 bits, coverage, then z2d's span compositing rules
//                 (raster/shared.zig) on pixels held in registers.
//
// Why the winding scan equals z2d's sorted spans: on every sub-scanline
// z2d sorts the active edges' rounded crossings, keeps the 0<->non-zero
// transitions (non-zero) or all of them (even-odd) and fills [x_{2k},
// x_{2k+1}).  A sample column c is then covered exactly when the crossings
// at x <= c have non-zero (odd) winding, provided the row's crossings are
// balanced.  Closed subpaths always give balanced rows; fills with an open
// 2-point subpath are routed to k_exact.
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#include "fill.cuh"
#include "host_pool.h"
#include "edges.cuh"
#include "spline.cuh"
#include "raster.cuh"
#include "raster_px.cuh"
#include "stroke_gpu.cuh"

namespace z2dg {

// ------------------------------------------------------------ kernels
// The sequential walk of fill_plotter.plot over one fill's nodes, one warp
// per fill: the warp stages 32 nodes at a time in shared memory, takes runs of
// segments together, lane 0 walks the rest, and the warp writes their
// NodeInfo back.  Bound by the latency of the walk (1,024 glyphs of 113
// nodes: node by node 45 us, now 13).
constexpr int kScanWarps = 4;
struct ScanStage {
    double x[32], y[32];    // node end point (curve: p[4], p[5])
    double sx[32], sy[32];  // NodeInfo fields the walk sets
    double ex[32], ey[32];
    int32_t tag[32], n_emit[32], n_added[32], off[32];
};

__global__ void __launch_bounds__(32 * kScanWarps) k_fill_scan(const z2d_node *__restrict__ nodes,
                                                               const FillCmd *__restrict__ fills,
                                                               NodeInfo *__restrict__ info, FillState *__restrict__ st,
                                                               int32_t n_fills, int32_t *__restrict__ counters,
                                                               int32_t *__restrict__ status,
                                                               const int32_t *__restrict__ stroke_edges,
                                                               const int32_t *__restrict__ poly_edges) {
    __shared__ ScanStage stages[kScanWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t f = blockIdx.x * kScanWarps + w;
    if (f >= n_fills) return;  // uniform across the warp
    ScanStage &S = stages[w];
    const int32_t node_off = fills[f].node_off, n_nodes = fills[f].n_nodes;
    const double tol = fills[f].tol;
    double fx = 0, fy = 0, lx = 0, ly = 0;
    int32_t count = 0;  // PointBuffer.len, saturating at 3
    int32_t off = 0;
    if (fills[f].stroke >= 0) {  // a device-stroked polygon: its edge count is known
        off = stroke_edges[fills[f].stroke];
        if (off < 0) {
            if (lane == 0) atomicExch(status, Z2D_ERR_INVALID_ARGUMENT);
            off = 0;
        }
    } else if (fills[f].poly >= 0) {  // a host-built polygon: one edge per point
        off = poly_edges[fills[f].poly];
    }
    int32_t flags = 0;
    for (int32_t base = 0; base < n_nodes; base += 32) {
        const int32_t j = base + lane;
        const bool valid = j < n_nodes;
        NodeInfo inf{};
        if (valid) {
            const z2d_node nd = nodes[node_off + j];
            inf = info[node_off + j];
            S.tag[lane] = nd.tag;
            S.x[lane] = nd.tag == Z2D_CURVE_TO ? nd.p[4] : nd.p[0];
            S.y[lane] = nd.tag == Z2D_CURVE_TO ? nd.p[5] : nd.p[1];
            S.n_emit[lane] = inf.n_emit;
            S.n_added[lane] = inf.n_added;
            S.sx[lane] = inf.sx;
            S.sy[lane] = inf.sy;
            S.ex[lane] = inf.ex;
            S.ey[lane] = inf.ey;
        }
        __syncwarp();
        // Runs of line_to and curve_to nodes whose start is the node before
        // (all but the first after a close_path) need no walk: their starts,
        // counts and edge offsets are a scan over the lanes.  Lane 0 walks the
        // others one at a time.
        const int32_t m = min(32, n_nodes - base);
        const uint32_t plain = __ballot_sync(0xffffffffu, valid && base + lane > 0 &&
                                                              (S.tag[lane] == Z2D_LINE_TO || S.tag[lane] == Z2D_CURVE_TO) &&
                                                              S.n_emit[lane] >= 0);
        for (int32_t k = 0; k < m;) {
            const uint32_t rest = plain >> k;
            const int32_t run = (rest & 1u) ? min(m - k, __ffs(~rest) == 0 ? 32 : __ffs(~rest) - 1) : 0;
            if (run >= 2) {
                const bool in = lane >= k && lane < k + run;
                int32_t incl = in ? S.n_emit[lane] : 0, add = in ? S.n_added[lane] : 0;
                const int32_t mine = incl;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                add = __reduce_add_sync(0xffffffffu, min(add, 3));
                if (in) {
                    S.off[lane] = off + incl - mine;
                    S.sx[lane] = lane == k ? lx : S.x[lane - 1];
                    S.sy[lane] = lane == k ? ly : S.y[lane - 1];
                }
                off += __shfl_sync(0xffffffffu, incl, 31);
                count = min(count + add, 3);
                lx = S.x[k + run - 1];
                ly = S.y[k + run - 1];
                k += run;
                continue;
            }
            if (lane == 0) {
                S.off[k] = off;
                int32_t ne;
                const double px = S.x[k], py = S.y[k];
                switch (S.tag[k]) {
                    case Z2D_MOVE_TO:
                        ne = 0;
                        if (base + k == n_nodes - 1) break;  // trailing move_to (fill_plotter.zig:38-40)
                        fx = lx = px;
                        fy = ly = py;
                        count = 1;
                        break;
                    case Z2D_LINE_TO:
                        S.sx[k] = lx;
                        S.sy[k] = ly;
                        ne = 1;
                        if (!pt_eq(lx, ly, px, py)) count = min(count + 1, 3);
                        lx = px;
                        ly = py;
                        break;
                    case Z2D_CURVE_TO: {
                        S.sx[k] = lx;
                        S.sy[k] = ly;
                        ne = S.n_emit[k];
                        if (ne < 0) {  // start depends on a preceding close_path
                            int32_t cne = 0, cna = 0;
                            double qx = lx, qy = ly;
                            auto cnt = [&](double x, double y) {
                                cne++;
                                if (!pt_eq(x, y, qx, qy)) cna++;
                                qx = x;
                                qy = y;
                            };
                            if (!spline_walk(lx, ly, nodes[node_off + base + k].p, tol, cnt))
                                atomicExch(status, Z2D_ERR_INVALID_STATE);
                            ne = cne;
                            S.n_added[k] = cna;
                        }
                        count = min(count + S.n_added[k], 3);
                        lx = px;
                        ly = py;
                        break;
                    }
                    default:  // close_path (fill_plotter.zig:72-92)
                        ne = 0;
                        S.sx[k] = lx;
                        S.sy[k] = ly;
                        S.ex[k] = fx;
                        S.ey[k] = fy;
                        if (count >= 3) {
                            if (!pt_eq(lx, ly, fx, fy)) {
                                ne = 1;
                                lx = fx;
                                ly = fy;
                            }
                        } else if (!pt_eq(lx, ly, fx, fy)) {
                            flags |= FILL_OPEN_CHAIN;  // a lone edge stays unmatched
                        }
                        break;
                }
                S.n_emit[k] = ne;
                off += ne;
            }
            // lane 0's state for the runs
            off = __shfl_sync(0xffffffffu, off, 0);
            count = __shfl_sync(0xffffffffu, count, 0);
            lx = __shfl_sync(0xffffffffu, lx, 0);
            ly = __shfl_sync(0xffffffffu, ly, 0);
            k++;
        }
        __syncwarp();
        if (valid) {
            inf.edge_off = S.off[lane];
            inf.n_emit = S.n_emit[lane];
            inf.n_added = S.n_added[lane];
            inf.sx = S.sx[lane];
            inf.sy = S.sy[lane];
            inf.ex = S.ex[lane];
            inf.ey = S.ey[lane];
            info[node_off + j] = inf;
        }
        __syncwarp();
    }
    if (lane == 0) {
        st[f].n_edges = off;
        st[f].edge_base = atomicAdd(&counters[CNT_EDGES], off);
        st[f].flags = flags;
        st[f].ext[0] = ~0ull;  // min slots start at the largest key
        st[f].ext[1] = 0ull;
        st[f].ext[2] = ~0ull;
        st[f].ext[3] = 0ull;
    }
}


// ------------------------------------------------------- curve flattening
constexpr int kFlattenWarps = 4;
constexpr int kScratch = 64;  // leaf points a lane keeps

// "Last valid value before this lane" within groups of G lanes, seeded with
// the group's carry.
__device__ __forceinline__ void prev_point_scan(bool has, double lx, double ly, double cx, double cy, int j, int G,
                                                double &px, double &py) {
    // inclusive "most recent valid" scan, then shift by one lane
    int v = has ? 1 : 0;
    double x = lx, y = ly;
    for (int o = 1; o < G; o <<= 1) {
        const int tv = __shfl_up_sync(0xffffffffu, v, o, G);
        const double tx = __shfl_up_sync(0xffffffffu, x, o, G);
        const double ty = __shfl_up_sync(0xffffffffu, y, o, G);
        if (j >= o && !v) {
            v = tv;
            x = tx;
            y = ty;
        }
    }
    px = cx;
    py = cy;
    if (G == 1) return;
    const int pv = __shfl_up_sync(0xffffffffu, v, 1, G);
    const double qx = __shfl_up_sync(0xffffffffu, x, 1, G);
    const double qy = __shfl_up_sync(0xffffffffu, y, 1, G);
    if (j > 0 && pv) {
        px = qx;
        py = qy;
    }
}

// Exclusive sum over the lanes of a group of G, and the group's total.
__device__ __forceinline__ int group_excl_sum(int v, int j, int G, int &total) {
    int incl = v;
    for (int o = 1; o < G; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o, G);
        if (j >= o) incl += t;
    }
    total = __shfl_sync(0xffffffffu, incl, G - 1, G);
    return incl - v;
}

// What a lane's share of a curve gives the curve: the lineTo calls its
// leaves issue (those whose start is not the curve's start: decomposeInto
// plots no such point), the points among them that differ from the one
// before, the first and the last point.
struct LaneCurve {
    int32_t cnt = 0, internal = 0, leaves = 0;
    double fx = 0, fy = 0, lx = 0, ly = 0;
    bool ok = true;
};
template <class P>
__device__ __forceinline__ LaneCurve walk_lane(double sx, double sy, const double *p, double tolerance, int g, int j,
                                               P &&leaf_start) {
    LaneCurve r;
    Knots k{sx, sy, p[0], p[1], p[2], p[3], p[4], p[5]};
    const Tol tol = make_tol(tolerance, k);
    bool is_leaf;
    int open;
    if (!lane_subtree(k, g, j, tol, is_leaf, open)) return r;
    r.ok = walk_leaves(k, is_leaf, open, tol, [&](const Knots &q) {
        leaf_start(r.leaves, q);
        r.leaves++;
        if (pt_eq(q.ax, q.ay, sx, sy)) return;
        if (r.cnt == 0) {
            r.fx = q.ax;
            r.fy = q.ay;
        } else if (!pt_eq(q.ax, q.ay, r.lx, r.ly)) {
            r.internal++;
        }
        r.lx = q.ax;
        r.ly = q.ay;
        r.cnt++;
    });
    return r;
}

// Appends idx to a device list (one atomic per warp); all lanes call it.
__device__ __forceinline__ void queue_push(bool push, int32_t idx, int32_t *list, int32_t *count, int lane) {
    const unsigned all = 0xffffffffu;
    const unsigned m = __ballot_sync(all, push);
    if (!m) return;
    int32_t base = 0;
    if (lane == 0) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(all, base, 0);
    if (push) list[base + __popc(m & ((1u << lane) - 1u))] = idx;
}

// The node kernels take 32 consecutive nodes per warp: every lane handles
// its own line, move and close_path node and queues its curve, if it has
// one, with the curves of its class (curve_class).
__global__ void __launch_bounds__(32 * kFlattenWarps) k_node_count_w(const z2d_node *__restrict__ nodes,
                                                                     const int32_t *__restrict__ node_fill,
                                                                     const FillCmd *__restrict__ fills,
                                                                     NodeInfo *__restrict__ info, int32_t n_nodes,
                                                                     int32_t *__restrict__ curves,
                                                                     int32_t *__restrict__ counters) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int32_t base = (blockIdx.x * kFlattenWarps + w) * 32; base < n_nodes;
         base += gridDim.x * kFlattenWarps * 32) {
        const int32_t i = base + lane;
        NodeInfo inf{};
        int curve = -1;  // its length class
        if (i < n_nodes) {
            const int32_t f = node_fill[i];
            if (f >= 0) {  // else no fill owns the node
                const z2d_node nd = nodes[i];
                const bool first_of_fill = (i == fills[f].node_off);
                if (nd.tag == Z2D_LINE_TO || nd.tag == Z2D_CURVE_TO) {
                    const z2d_node pv = first_of_fill ? nd : nodes[i - 1];
                    const bool static_start = !first_of_fill && (pv.tag == Z2D_MOVE_TO || pv.tag == Z2D_LINE_TO ||
                                                                 pv.tag == Z2D_CURVE_TO);
                    if (!static_start) {
                        inf.n_emit = -1;  // resolved by k_fill_scan
                    } else {
                        const double sx = pv.tag == Z2D_CURVE_TO ? pv.p[4] : pv.p[0];
                        const double sy = pv.tag == Z2D_CURVE_TO ? pv.p[5] : pv.p[1];
                        if (nd.tag == Z2D_LINE_TO) {
                            inf.n_emit = 1;
                            inf.n_added = pt_eq(sx, sy, nd.p[0], nd.p[1]) ? 0 : 1;
                        } else if (pt_eq(sx, sy, nd.p[0], nd.p[1]) && pt_eq(nd.p[2], nd.p[3], nd.p[4], nd.p[5])) {
                            inf.n_emit = 1;  // a straight one: lineTo(d) (Spline.zig:39-42)
                            inf.n_added = pt_eq(sx, sy, nd.p[4], nd.p[5]) ? 0 : 1;
                        } else {  // k_curve_count_w fills in its info
                            curve = curve_class(sx, sy, nd.p, fills[f].tol);
                        }
                    }
                }
            }
        }
        inf.pool = -1;
        if (i < n_nodes && curve < 0) info[i] = inf;
        for (int k = 0; k < kCurveClasses; k++)
            queue_push(curve == k, i, curves + k * (size_t)n_nodes, counters + CNT_CURVES + k, lane);
    }
}

// Counts every queued curve's lineTo calls (n_emit) and the points
// PointBuffer keeps of them (n_added).  2^g neighbouring lanes walk a curve:
// about 8 leaves each (g = 0 for class 0, g = k - 3 for a curve of about 2^k
// leaves), fewer while the grid has lanes to spare.  The lanes of a warp then
// have walks of like length, and the splits that every lane of a curve
// repeats stay few against the leaves.  (A warp per curve left most lanes
// idle on short curves: 1,024 glyphs of 110 curves 655 us, in classes 157; 320
// surfaces with 16 k fills 2.1 ms, then 0.76; 2,000 paths of long curves 396
// us, then 285.  Three classes of 1, 8 and 32 lanes: 222, 925 and 309 us.)
// A curve's edges are its leaves' chords when every leaf start but the first
// differs from the curve's start (consecutive leaves share their end points,
// so the lineTo sequence start, a1, a2, ..., d is the chord sequence): such a
// curve, if its leaves fit the lanes' scratch, leaves its polyline (leaf
// starts, then d) in the curve pool, and the emit pass reads points instead
// of subdividing again.  Bound by the issue of the subdivision (below_tol,
// de_casteljau).
__global__ void __launch_bounds__(32 * kFlattenWarps) k_curve_count_w(const z2d_node *__restrict__ nodes,
                                                                      const int32_t *__restrict__ node_fill,
                                                                      const FillCmd *__restrict__ fills,
                                                                      NodeInfo *__restrict__ info, int32_t n_nodes,
                                                                      const int32_t *__restrict__ curves,
                                                                      int32_t *__restrict__ counters,
                                                                      int32_t *__restrict__ status,
                                                                      double2 *__restrict__ scratch,
                                                                      double2 *__restrict__ pool, int32_t pool_cap) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double2 *scr = scratch + (size_t)(blockIdx.x * kFlattenWarps + w) * (32 * kScratch);
    const int32_t warps = gridDim.x * kFlattenWarps;
    int32_t n[kCurveClasses];
    long long lanes = 0;
    for (int k = 0; k < kCurveClasses; k++) {
        n[k] = counters[CNT_CURVES + k];
        lanes += (long long)n[k] << k;
    }
    int spare = 0;
    while (spare < kCurveClasses - 1 && (lanes << (spare + 1)) <= 32ll * warps) spare++;
    // chunks of 32 >> g curves, the longest class first
    int32_t chunks = 0;
    for (int k = 0; k < kCurveClasses; k++)
        chunks += (int32_t)((((long long)n[k] << min(k + spare, 5)) + 31) >> 5);
    for (int32_t c0 = blockIdx.x * kFlattenWarps + w; c0 < chunks; c0 += warps) {
        int32_t c = c0;
        int k = kCurveClasses - 1;
        for (; k > 0; k--) {
            const int32_t m = (int32_t)((((long long)n[k] << min(k + spare, 5)) + 31) >> 5);
            if (c < m) break;
            c -= m;
        }
        const int g = min(k + spare, 5), G = 1 << g;
        const int j = lane & (G - 1);
        const int32_t q = c * (32 >> g) + (lane >> g);
        int32_t nk = n[0];
#pragma unroll
        for (int i = 1; i < kCurveClasses; i++)
            if (k == i) nk = n[i];
        const bool live = q < nk;
        int32_t i = 0;
        double sx = 0, sy = 0, dx = 0, dy = 0;
        LaneCurve r;
        if (live) {
            i = curves[k * (size_t)n_nodes + q];
            const z2d_node nd = nodes[i];
            const z2d_node pv = nodes[i - 1];
            sx = pv.tag == Z2D_CURVE_TO ? pv.p[4] : pv.p[0];
            sy = pv.tag == Z2D_CURVE_TO ? pv.p[5] : pv.p[1];
            dx = nd.p[4];
            dy = nd.p[5];
            r = walk_lane(sx, sy, nd.p, fills[node_fill[i]].tol, g, j, [&](int32_t m, const Knots &q) {
                if (m < kScratch) scr[m * 32 + lane] = make_double2(q.ax, q.ay);
            });
            if (!r.ok) atomicExch(status, Z2D_ERR_INVALID_STATE);
        }
        __syncwarp();
        double px, py;
        prev_point_scan(r.cnt > 0, r.lx, r.ly, sx, sy, j, G, px, py);
        const int32_t first_add = (r.cnt > 0 && !pt_eq(r.fx, r.fy, px, py)) ? 1 : 0;
        int32_t emit = 0, added = 0, leaves = 0, unfit = 0;
        group_excl_sum(r.cnt, j, G, emit);
        group_excl_sum(r.internal + first_add, j, G, added);
        const int32_t at = group_excl_sum(r.leaves, j, G, leaves);
        group_excl_sum(r.leaves > kScratch || !r.ok ? 1 : 0, j, G, unfit);
        const bool chords = leaves == emit + 1;
        // the group's last lane sees the last point before d
        const bool last = live && j == G - 1;
        const double ex = r.cnt > 0 ? r.lx : px, ey = r.cnt > 0 ? r.ly : py;
        // room for the polylines of the warp's curves: one reservation
        const bool keep = live && chords && unfit == 0;
        int32_t room = 0;
        const int32_t mine = group_excl_sum(last && keep ? leaves + 1 : 0, lane, 32, room);
        int32_t base = -1;
        if (room > 0) {
            if (lane == 0) {
                const unsigned long long b = atomicAdd(reinterpret_cast<unsigned long long *>(&counters[CNT_POOL]),
                                                       (unsigned long long)room);
                base = (b + (unsigned long long)room <= (unsigned long long)pool_cap) ? (int32_t)b : -1;
            }
            base = __shfl_sync(0xffffffffu, base, 0);
        }
        // (the last lane's own sum is that of the curves before)
        const int32_t first = __shfl_sync(0xffffffffu, mine, G - 1, G) + base;
        const bool pooled = keep && base >= 0;
        if (pooled) {
            double2 *out = pool + first + at;
            for (int32_t m = 0; m < r.leaves; m++) out[m] = scr[m * 32 + lane];
            if (last) pool[first + leaves] = make_double2(dx, dy);
        }
        if (last) {
            NodeInfo inf{};
            inf.n_emit = emit + 1;  // with the final lineTo(d)
            inf.n_added = added + (pt_eq(dx, dy, ex, ey) ? 0 : 1);
            inf.pool = pooled ? first : -1;
            info[i] = inf;
        }
        __syncwarp();
    }
}

// Emits the edges of one curve with the whole warp: its leaves counted by
// one walk, emitted by another.
__device__ __forceinline__ void curve_emit_warp(const FillCmd &F, DEdge *out, const NodeInfo &inf, const double *p,
                                                int lane, double &et, double &eb, double &el, double &er, bool &any) {
    const LaneCurve r = walk_lane(inf.sx, inf.sy, p, F.tol, 5, lane, [](int32_t, const Knots &) {});
    __syncwarp();
    double px, py;
    prev_point_scan(r.cnt > 0, r.lx, r.ly, inf.sx, inf.sy, lane, 32, px, py);
    int tot = 0;
    const int off = group_excl_sum(r.cnt, lane, 32, tot);
    const double ex = r.cnt > 0 ? r.lx : px, ey = r.cnt > 0 ? r.ly : py;
    if (r.cnt > 0) {
        int32_t k = off;
        walk_lane(inf.sx, inf.sy, p, F.tol, 5, lane, [&](int32_t, const Knots &q) {
            if (pt_eq(q.ax, q.ay, inf.sx, inf.sy)) return;
            if (k < inf.n_emit) add_edge(F, out + k, px, py, q.ax, q.ay, et, eb, el, er, any);
            k++;
            px = q.ax;
            py = q.ay;
        });
    }
    if (lane == 31 && tot < inf.n_emit)  // final lineTo(d)
        add_edge(F, out + tot, ex, ey, p[4], p[5], et, eb, el, er, any);
}

__global__ void __launch_bounds__(32 * kFlattenWarps) k_node_emit_w(const z2d_node *__restrict__ nodes,
                                                                    const int32_t *__restrict__ node_fill,
                                                                    const FillCmd *__restrict__ fills,
                                                                    const NodeInfo *__restrict__ info,
                                                                    FillState *__restrict__ st, DEdge *__restrict__ edges,
                                                                    int32_t n_nodes, int32_t *__restrict__ curves,
                                                                    int32_t *__restrict__ counters) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int32_t base = (blockIdx.x * kFlattenWarps + w) * 32; base < n_nodes;
         base += gridDim.x * kFlattenWarps * 32) {
        const int32_t i = base + lane;
        int32_t f = -1;
        bool curve = false;
        double et = 0, eb = 0, el = 0, er = 0;
        bool any = false;
        if (i < n_nodes) {
            const NodeInfo inf = info[i];
            if (inf.n_emit > 0) {
                const z2d_node nd = nodes[i];
                f = node_fill[i];
                const FillCmd &F = fills[f];
                DEdge *out = edges + st[f].edge_base + inf.edge_off;
                const bool straight = nd.tag == Z2D_CURVE_TO && pt_eq(inf.sx, inf.sy, nd.p[0], nd.p[1]) &&
                                      pt_eq(nd.p[2], nd.p[3], nd.p[4], nd.p[5]);
                // one add_edge for lanes of every kind
                const int last = nd.tag == Z2D_CURVE_TO ? 4 : 0;
                const bool close = nd.tag == Z2D_CLOSE_PATH;
                if (nd.tag == Z2D_LINE_TO || close || straight)
                    add_edge(F, out, inf.sx, inf.sy, close ? inf.ex : nd.p[last], close ? inf.ey : nd.p[last + 1], et,
                             eb, el, er, any);
                else curve = true;  // k_curve_emit_w emits it
            }
        }
        queue_push(curve, i, curves, counters + CNT_CURVES_EMIT, lane);
        merge_extents(st, f, any, et, eb, el, er);
    }
}

// Emits the queued curves' edges.  A warp takes up to 32 curves (as many as
// give every warp of the grid some) and goes through the edges of those with
// a polyline 32 at a time, whichever curve they belong to: a curve of a few
// edges does not idle the other lanes.  Edge k of a curve joins points k and
// k + 1.
__global__ void __launch_bounds__(32 * kFlattenWarps) k_curve_emit_w(const z2d_node *__restrict__ nodes,
                                                                     const int32_t *__restrict__ node_fill,
                                                                     const FillCmd *__restrict__ fills,
                                                                     const NodeInfo *__restrict__ info,
                                                                     FillState *__restrict__ st,
                                                                     DEdge *__restrict__ edges,
                                                                     const int32_t *__restrict__ curves,
                                                                     const int32_t *__restrict__ counters,
                                                                     const double2 *__restrict__ pool) {
    constexpr uint32_t all = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t n = counters[CNT_CURVES_EMIT], warps = gridDim.x * kFlattenWarps;
    const int32_t per = max(1, min(32, (n + warps - 1) / warps));
    for (int32_t q0 = (blockIdx.x * kFlattenWarps + w) * per; q0 < n; q0 += warps * per) {
        int32_t i = -1, f = -1, cnt = 0, src = 0;
        long long dst = 0;
        if (lane < per && q0 + lane < n) {
            i = curves[q0 + lane];
            f = node_fill[i];
            const NodeInfo &inf = info[i];
            if (inf.pool >= 0) {
                cnt = inf.n_emit;
                src = inf.pool;
                dst = (long long)st[f].edge_base + inf.edge_off;
                i = -1;
            }
        }
        int32_t total;
        const int32_t excl = group_excl_sum(cnt, lane, 32, total);
        for (int32_t k0 = 0; k0 < total; k0 += 32) {
            const int32_t k = k0 + lane;
            // the last lane whose first edge is <= k owns edge k
            int own = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int32_t e = __shfl_sync(all, excl, own + step);
                if (e <= k) own += step;
            }
            const int32_t at = k - __shfl_sync(all, excl, own), of = __shfl_sync(all, f, own);
            const double2 *P = pool + __shfl_sync(all, src, own) + at;
            DEdge *out = edges + __shfl_sync(all, dst, own) + at;
            double et = 0, eb = 0, el = 0, er = 0;
            bool any = false;
            if (k < total) {
                const double2 a = P[0], b = P[1];
                add_edge(fills[of], out, a.x, a.y, b.x, b.y, et, eb, el, er, any);
            }
            merge_extents(st, of, any, et, eb, el, er);
        }
        // curves without a polyline, one after the other
        for (uint32_t m = __ballot_sync(all, i >= 0); m; m &= m - 1) {
            const int own = __ffs(m) - 1;
            const int32_t ci = __shfl_sync(all, i, own), cf = __shfl_sync(all, f, own);
            const NodeInfo inf = info[ci];
            const z2d_node nd = nodes[ci];
            double et = 0, eb = 0, el = 0, er = 0;
            bool any = false;
            curve_emit_warp(fills[cf], edges + st[cf].edge_base + inf.edge_off, inf, nd.p, lane, et, eb, el, er, any);
            __syncwarp();
            merge_extents(st, cf, any, et, eb, el, er);
        }
    }
}

__device__ __forceinline__ int32_t clampi(int32_t v, int32_t lo, int32_t hi) { return max(lo, min(v, hi)); }

__global__ void k_fill_setup(const FillCmd *__restrict__ fills, FillState *__restrict__ st, int32_t n_fills,
                             DevJob *__restrict__ jobs, int32_t *__restrict__ counters, RasterFill *__restrict__ rf) {
    const int32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_fills) return;
    const FillCmd F = fills[f];
    DevJob &J = jobs[F.job];
    const int32_t sw = J.sfc.w, sh = J.sfc.h;
    FillState S = st[f];
    S.active = 0;
    if (!S.has_edges) {  // inBox of the empty polygon is false
        st[f] = S;
        return;
    }
    const double et = dkey_inv(S.ext[0]), eb = dkey_inv(S.ext[1]), el = dkey_inv(S.ext[2]), er = dkey_inv(S.ext[3]);
    const double sc = F.scale;
    // Polygon.inBox (Polygon.zig:142-201)
    if (er < 0.0 || eb < 0.0) {
        st[f] = S;
        return;
    }
    const int32_t psx = (int32_t)floor(el / sc), psy = (int32_t)floor(et / sc);
    const int32_t pex = (int32_t)ceil(er / sc), pey = (int32_t)ceil(eb / sc);
    const int32_t pw = pex - psx, ph = pey - psy;
    if (pw == 0 || ph == 0 || psx + pw < 0 || psy + ph < 0 || psx >= sw || psy >= sh) {
        st[f] = S;
        return;
    }
    S.active = 1;
    const bool bounded = is_bounded(F.op);
    if (F.aa == Z2D_AA_NONE) {  // direct.run (direct.zig:36-49)
        const int32_t y0 = bounded ? (int32_t)floor(et) : 0;
        const int32_t y1 = bounded ? (int32_t)ceil(eb) : sh - 1;
        S.start_y = clampi(y0, 0, sh - 1);
        S.end_y = clampi(y1, S.start_y, sh - 1);
        // spans are clamped to the surface, not to the extents; crossings
        // lie within one pixel of the x extents
        S.start_x = clampi((int32_t)floor(el) - 1, 0, sw);
        S.end_x = clampi((int32_t)ceil(er) + 2, S.start_x, sw);
        if (!bounded) S.flags |= FILL_EXACT;
    } else if (F.aa == Z2D_AA_SUPERSAMPLE_4X) {
        // supersample.run (supersample.zig:41-84, 172-184): a 4x mask over
        // [bx0, bx1] x [by0, by1] in sample units, downsampled 4x4 -> 1
        // unless it is narrower or lower than 4 samples, then composited at
        // (max(0, x0), max(0, y0)) and clipped to the surface by
        // SurfaceCompositor.run (compositor.zig:313-374).  Downsampled mask
        // pixel (i, j) averages the samples of surface pixel (cx + i, cy + j).
        const int32_t x0 = bounded ? (int32_t)floor(el / 4.0) : 0;
        const int32_t y0 = bounded ? (int32_t)floor(et / 4.0) : 0;
        const int32_t x1 = bounded ? (int32_t)ceil(er / 4.0) : sw;
        const int32_t y1 = bounded ? (int32_t)ceil(eb / 4.0) : sh;
        const int32_t tw = sw * 4, th = sh * 4;
        const int32_t bx0 = clampi(x0 * 4, 0, tw - 1), by0 = clampi(y0 * 4, 0, th - 1);
        const int32_t bx1 = clampi(x1 * 4, bx0, tw - 1), by1 = clampi(y1 * 4, by0, th - 1);
        const int32_t mw = bx1 + 1 - bx0, mh = by1 + 1 - by0;
        const bool down = mw >= 4 && mh >= 4;
        const int32_t rw = down ? mw / 4 : mw, rh = down ? mh / 4 : mh;
        const int32_t cx = max(0, x0), cy = max(0, y0);
        const int32_t w = (rw + cx > sw) ? sw - cx : rw, h = (rh + cy > sh) ? sh - cy : rh;
        if (w <= 0 || h <= 0) {
            S.active = 0;
            st[f] = S;
            return;
        }
        S.start_x = cx;
        S.end_x = cx + w;
        S.start_y = cy;
        S.end_y = cy + h - 1;
        // Without the downsample, nothing is ever painted into the mask: it
        // is 1 sample wide (or high) only when extent_right (or _bottom) is
        // 0 and the polygon lies left of (or above) the surface.
        if (!down) S.flags |= FILL_SS_ZERO;
    } else {  // multisample.run (multisample.zig:46-78)
        S.start_y = clampi((int32_t)floor(et / 4.0), 0, sh - 1);
        S.end_y = clampi((int32_t)ceil(eb / 4.0), S.start_y, sh - 1);
        S.start_x = clampi((int32_t)floor(el / 4.0), 0, sw - 1);
        S.end_x = clampi((int32_t)ceil(er / 4.0), S.start_x, sw);
    }
    if ((S.flags & FILL_OPEN_CHAIN) && !(S.flags & FILL_SS_ZERO)) S.flags |= FILL_EXACT;
    // rows the fill touches: the draw rows, or every row for unbounded
    // operators (their clears reach outside the draw box); a supersample
    // fill touches exactly its composite region
    const bool boxed = bounded || F.aa == Z2D_AA_SUPERSAMPLE_4X;
    const int32_t ty0 = boxed ? S.start_y : 0;
    const int32_t ty1 = boxed ? S.end_y : sh - 1;
    S.band0 = ty0 / kTileRows;
    S.band1 = ty1 / kTileRows;
    S.fb_base = atomicAdd(&counters[CNT_FILL_BANDS], S.band1 - S.band0 + 1);
    if (S.flags & FILL_EXACT) {
        // action mask over the rows the exact rasteriser visits
        S.mask_w = (F.aa == Z2D_AA_NONE) ? sw : (S.end_x - S.start_x);
        S.mask_x0 = (F.aa == Z2D_AA_NONE) ? 0 : S.start_x;
        // mask, then 8-byte aligned work arrays of 4 ints per edge
        // (permutation, crossings, and 2 breakpoints)
        const long long bytes = ((((long long)S.mask_w * (S.end_y - S.start_y + 1) + 7) & ~7ll) + 16ll * S.n_edges + 15) & ~7ll;
        S.mask_base = atomicAdd(reinterpret_cast<unsigned long long *>(&counters[CNT_MASK_LO]), (unsigned long long)bytes);
        atomicAdd(&counters[CNT_EXACT], 1);
    }
    atomicMin(&J.band_lo, S.band0);
    atomicMax(&J.band_hi, S.band1);
    const int32_t cx0 = boxed ? S.start_x : 0, cx1 = boxed ? S.end_x : sw;
    S.cull_x0 = cx0;
    S.cull_x1 = cx1;
    atomicMin(&J.tcol_lo, cx0 / kTileCols);
    atomicMax(&J.tcol_hi, (max(cx1, cx0 + 1) - 1) / kTileCols);
    st[f] = S;
    RasterFill R;
    R.start_x = S.start_x;
    R.end_x = S.end_x;
    R.start_y = S.start_y;
    R.end_y = S.end_y;
    R.meta = ((uint32_t)F.op & RF_OP_MASK) | ((uint32_t)F.aa << RF_AA_SHIFT) |
             (F.rule == Z2D_FILL_EVEN_ODD ? RF_EVEN_ODD : 0u) | ((uint32_t)F.fast_kind << RF_FAST_SHIFT) |
             ((S.flags & FILL_EXACT) ? RF_EXACT : 0u) | ((S.flags & FILL_SS_ZERO) ? RF_SS_ZERO : 0u) |
             (bounded ? RF_BOUNDED : 0u);
    R._pad[0] = R._pad[1] = R._pad[2] = 0;
    rf[f] = R;
}

// Band range of an edge's active sample rows within the fill's draw rows.
__device__ __forceinline__ bool edge_bands(const DEdge &e, const FillCmd &F, const FillState &S, int32_t &b0,
                                           int32_t &b1) {
    const int32_t S_ = (int32_t)F.scale;
    const int32_t lo = max(e.rt, S.start_y * S_), hi = min(e.rb, (S.end_y + 1) * S_);
    if (lo >= hi) return false;
    b0 = lo / (kTileRows * S_);
    b1 = (hi - 1) / (kTileRows * S_);
    return true;
}

// Binning visits every (edge, band) pair.  A long edge spans hundreds of
// bands, so a thread per edge would serialise its atomics; instead each warp
// takes 32 edges and walks their pairs 32 at a time, every lane finding the
// edge of its pair by a binary search over the warp's prefix sums.
template <class Visit>
__device__ __forceinline__ void for_edge_bands(const FillCmd *__restrict__ fills, const FillState *__restrict__ st,
                                               const DEdge *__restrict__ edges, const int32_t *__restrict__ edge_fill,
                                               int32_t n_edges, Visit &&visit) {
    const int lane = threadIdx.x & 31;
    const int32_t stride = gridDim.x * blockDim.x;
    for (int32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n_edges; base += stride) {
        const int32_t i = base + lane;
        int32_t nb = 0, fb0 = 0, row0 = 0;  // row0: the first band's first sample row, | 1 with 4 a pixel
        if (i < n_edges) {
            const int32_t f = edge_fill[i];
            if (f >= 0) {
                const FillState &S = st[f];
                int32_t b0, b1;
                if (S.active && !(S.flags & FILL_EXACT) && edge_bands(edges[i], fills[f], S, b0, b1)) {
                    nb = b1 - b0 + 1;
                    fb0 = S.fb_base + (b0 - S.band0);
                    const int32_t S_ = (int32_t)fills[f].scale;
                    row0 = b0 * kTileRows * S_ | (S_ == 4 ? 1 : 0);
                }
            }
        }
        int32_t incl = nb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int32_t excl = incl - nb;
        const int32_t total = __shfl_sync(0xffffffffu, incl, 31);
        for (int32_t k0 = 0; k0 < total; k0 += 32) {
            const int32_t k = k0 + lane;
            // the last lane whose first pair is <= k owns pair k
            int owner = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int32_t e = __shfl_sync(0xffffffffu, excl, owner + step);
                if (e <= k) owner += step;
            }
            const int32_t o_excl = __shfl_sync(0xffffffffu, excl, owner);
            const int32_t o_fb0 = __shfl_sync(0xffffffffu, fb0, owner);
            const int32_t o_row0 = __shfl_sync(0xffffffffu, row0, owner);
            const int32_t rows = (o_row0 & 1) ? 4 * kTileRows : kTileRows;
            if (k < total) visit(base + owner, o_fb0 + (k - o_excl), (o_row0 & ~1) + (k - o_excl) * rows, rows);
        }
    }
}

__global__ void k_bin_count(const FillCmd *__restrict__ fills, const FillState *__restrict__ st,
                            const DEdge *__restrict__ edges, const int32_t *__restrict__ edge_fill, int32_t n_edges,
                            int32_t *__restrict__ fb_count, int32_t *__restrict__ status) {
    for_edge_bands(fills, st, edges, edge_fill, n_edges, [&](int32_t, int32_t fb, int32_t, int32_t) {
        if (atomicAdd(&fb_count[fb], 1) >= kMaxBandEdges) atomicExch(status, Z2D_ERR_INVALID_ARGUMENT);
    });
}

// The rasteriser reads an edge once per tile column and row of a band: the
// bin holds what it reads, one coalesced 32-byte record per entry, instead of
// an index to gather it by (RECORDS; without, the index: BinKind).
template <bool RECORDS>
__global__ void k_bin_fill(const FillCmd *__restrict__ fills, const FillState *__restrict__ st,
                           const DEdge *__restrict__ edges, const int32_t *__restrict__ edge_fill, int32_t n_edges,
                           int32_t *__restrict__ fb_cursor, void *__restrict__ bins) {
    for_edge_bands(fills, st, edges, edge_fill, n_edges, [&](int32_t edge, int32_t fb, int32_t row, int32_t rows) {
        const int32_t at = atomicAdd(&fb_cursor[fb], 1);
        if constexpr (!RECORDS) {
            reinterpret_cast<int32_t *>(bins)[at] = edge;
            return;
        }
        const int4 a = __ldg(reinterpret_cast<const int4 *>(edges + edge));
        const int2 r = __ldg(reinterpret_cast<const int2 *>(&edges[edge].rt));
        const BinEdge B = bin_edge(a.x, __int_as_float(a.y), __int_as_float(a.z), __int_as_float(a.w), r.x, r.y, edge,
                                   row, rows);
        int4 *out = reinterpret_cast<int4 *>(reinterpret_cast<BinEdge *>(bins) + at);
        out[0] = make_int4(B.c, __float_as_int(B.fx), __float_as_int(B.fxi), __float_as_int(B.t));
        out[1] = make_int4((int32_t)B.rows, __float_as_int(B.limit), B.id, 0);
    });
}

// Edge -> fill map (edges of one fill are contiguous), and the fill's source
// word for every coverage: 17 words that a fill's every row and tile would
// otherwise compute again, with a division per channel.
__global__ void k_edge_fill(const FillState *__restrict__ st, const FillCmd *__restrict__ fills,
                            const DevJob *__restrict__ jobs, int32_t *__restrict__ edge_fill,
                            uint32_t *__restrict__ luts) {
    const int32_t f = blockIdx.x;
    const FillState &S = st[f];
    const int32_t e0 = S.edge_base, n = S.n_edges;
    for (int32_t k = threadIdx.x; k < n; k += blockDim.x) edge_fill[e0 + k] = f;
    if (threadIdx.x < 32) {
        const FillCmd &F = fills[f];
        luts[32 * (size_t)f + threadIdx.x] =
            F.fast_kind == FAST_PIXEL_SRC_OVER ? coverage_word(F, jobs[F.job].sfc.fmt, (int)threadIdx.x) : 0u;
    }
}

// Ordered list of the fills touching each band (call order preserved by a
// block-wide stream compaction).
// The job a global index belongs to: the last job whose base is <= i
// (bases ascending; jobs with nothing to draw repeat the next base).
template <class Base>
__device__ __forceinline__ int32_t job_of(const DevJob *__restrict__ jobs, int32_t n_jobs, long long i, Base base) {
    int32_t lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int32_t mid = (lo + hi + 1) >> 1;
        if (base(jobs[mid]) <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

constexpr int32_t kWarpFills = 512;
// With a warp per band, for the jobs of at most max_fills fills: a CTA per band
// spends its time starting and meeting at barriers (16,384 bands of one fill:
// 43 us, a warp each 11).
__global__ void __launch_bounds__(256) k_band_lists_w(const FillState *__restrict__ st, const DevJob *__restrict__ jobs,
                                                      int32_t n_jobs, int32_t n_gbands, int32_t max_fills,
                                                      int32_t *__restrict__ band_count, int4 *__restrict__ band_fills,
                                                      TileRec *__restrict__ tiles) {
    const long long at = warp_number(blockIdx.x, blockDim.x, threadIdx.x);
    if (at >= n_gbands) return;
    const int32_t gb = (int32_t)at, lane = threadIdx.x & 31;
    const int32_t j = job_of(jobs, n_jobs, gb, [](const DevJob &J) { return (long long)J.gband_base; });
    const DevJob &J = jobs[j];
    const int32_t lb = gb - J.gband_base, b = J.band_lo + lb, nf = J.fill1 - J.fill0;
    if (nf > max_fills) return;
    if (tiles) {
        const int32_t nc = J.tcol_hi - J.tcol_lo + 1;
        for (int32_t t = lane; t < nc; t += 32) tiles[J.tile_base + (long long)lb * nc + t] = TileRec{j, lb, t, 0};
    }
    int4 *out = band_fills + J.list_base + (long long)lb * nf;
    int32_t n = 0;
    for (int32_t f0 = J.fill0; f0 < J.fill1; f0 += 32) {
        const int32_t f = f0 + lane;
        bool hit = false;
        int4 ent = make_int4(f, 0, 0, 0);
        if (f < J.fill1) {
            const FillState &S = st[f];
            hit = S.active && b >= S.band0 && b <= S.band1;
            ent.y = S.cull_x0;
            ent.z = S.cull_x1;
            ent.w = S.fb_base + (b - S.band0);
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) out[n + __popc(m & ((1u << lane) - 1u))] = ent;
        n += __popc(m);
    }
    if (lane == 0) band_count[gb] = n;
}

// One CTA per global band from gb0 on, of the jobs of more than max_fills
// fills: the job's fills touching the band, in call order
// (ordered compaction), with the tile-column range each one can affect and
// the fill's (fill, band) slot of the band, and (several surfaces) the
// records of the band's tiles.
__global__ void __launch_bounds__(256) k_band_lists(const FillState *__restrict__ st, const DevJob *__restrict__ jobs,
                                                    int32_t n_jobs, int32_t gb0, int32_t max_fills,
                                                    int32_t *__restrict__ band_count,
                                                    int4 *__restrict__ band_fills, TileRec *__restrict__ tiles) {
    const int32_t gb = gb0 + (int32_t)blockIdx.x;
    const int32_t j = job_of(jobs, n_jobs, gb, [](const DevJob &J) { return (long long)J.gband_base; });
    const DevJob J = jobs[j];
    const int32_t lb = gb - J.gband_base;
    const int32_t b = J.band_lo + lb;
    const int32_t nf = J.fill1 - J.fill0;
    if (nf <= max_fills) return;
    if (tiles) {
        const int32_t nc = J.tcol_hi - J.tcol_lo + 1;
        for (int32_t t = threadIdx.x; t < nc; t += blockDim.x)
            tiles[J.tile_base + (long long)lb * nc + t] = TileRec{j, lb, t, 0};
    }
    __shared__ int32_t warp_tot[8];
    __shared__ int32_t base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    const int32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int4 *out = band_fills + J.list_base + (long long)lb * nf;
    for (int32_t f0 = J.fill0; f0 < J.fill1; f0 += blockDim.x) {
        const int32_t f = f0 + threadIdx.x;
        bool hit = false;
        int4 ent = make_int4(f, 0, 0, 0);
        if (f < J.fill1) {
            const FillState &S = st[f];
            hit = S.active && b >= S.band0 && b <= S.band1;
            ent.y = S.cull_x0;
            ent.z = S.cull_x1;
            ent.w = S.fb_base + (b - S.band0);
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) warp_tot[wid] = __popc(m);
        __syncthreads();
        int32_t before = 0, total = 0;
        for (int w = 0; w < 8; w++) {
            if (w < wid) before += warp_tot[w];
            total += warp_tot[w];
        }
        if (hit) out[base + before + __popc(m & ((1u << lane) - 1u))] = ent;
        __syncthreads();
        if (threadIdx.x == 0) base += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) band_count[gb] = base;
}

}  // namespace z2dg

namespace z2dg {

// ----------------------------------------------------------- exact path
// Literal restatement of multisample.run / direct.run's sorted-span loop
// (multisample.zig:115-188, direct.zig:51-126, Polygon.zig:232-353) for one
// fill, one thread, writing a per-pixel action mask.  Used for fills whose
// rows may be unbalanced (open 2-point subpaths) and for unbounded operators
// without anti-aliasing, where z2d's per-span clears depend on span order.
__device__ void sort_insertion(int32_t *perm, int32_t *xv, int32_t n) {
    // std.sort.insertionContext; stable, so it orders ties like the stable
    // sort the CPU oracle uses beyond 24 active edges
    for (int32_t i = 1; i < n; i++)
        for (int32_t j = i; j > 0 && xv[j] < xv[j - 1]; j--) {
            const int32_t te = perm[j]; perm[j] = perm[j - 1]; perm[j - 1] = te;
            const int32_t tx = xv[j]; xv[j] = xv[j - 1]; xv[j - 1] = tx;
        }
}

__device__ void shell_sort_unique(int32_t *a, int32_t &n) {
    for (int32_t gap = n / 2; gap > 0; gap /= 2)
        for (int32_t i = gap; i < n; i++) {
            const int32_t t = a[i];
            int32_t j = i;
            for (; j >= gap && a[j - gap] > t; j -= gap) a[j] = a[j - gap];
            a[j] = t;
        }
    int32_t m = 0;
    for (int32_t i = 0; i < n; i++)
        if (m == 0 || a[i] != a[m - 1]) a[m++] = a[i];
    n = m;
}

__global__ void k_exact(const FillCmd *__restrict__ fills, const FillState *__restrict__ st, const DEdge *__restrict__ edges,
                        int32_t n_fills, const DevJob *__restrict__ jobs, uint8_t *__restrict__ masks) {
    const int32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_fills) return;
    const FillState S = st[f];
    if (!S.active || !(S.flags & FILL_EXACT)) return;
    const FillCmd F = fills[f];
    const int32_t sw = jobs[F.job].sfc.w;
    const DEdge *E = edges + S.edge_base;
    uint8_t *mask = masks + S.mask_base;  // zeroed by the host
    const int32_t mh = S.end_y - S.start_y + 1;
    // work arrays live after the mask, 8-byte aligned
    int32_t *perm = reinterpret_cast<int32_t *>(masks + S.mask_base + (((long long)S.mask_w * mh + 7) & ~7ll));
    int32_t *xv = perm + S.n_edges;
    int32_t *bp = xv + S.n_edges;
    int32_t n = 0;
    for (int32_t i = 0; i < S.n_edges; i++)
        if (E[i].rt < E[i].rb) perm[n++] = i;
    int32_t nbp = 0;
    for (int32_t i = 0; i < n; i++) {
        bp[nbp++] = E[perm[i]].rt;
        bp[nbp++] = E[perm[i]].rb;
    }
    shell_sort_unique(bp, nbp);
    int32_t bpi = -1;
    for (int32_t i = 0; i < nbp; i++)
        if (bp[i] >= S.start_y) {
            bpi = i == 0 ? 0 : i - 1;
            break;
        }
    if (bpi < 0) return;
    const bool direct = F.aa == Z2D_AA_NONE;
    const bool bounded = is_bounded(F.op);
    const int32_t sc = direct ? 1 : 4;
    int32_t n_active = 0;
    const int32_t sxs = S.start_x * 4, dws = (S.end_x - S.start_x) * 4;
    for (int32_t y = S.start_y; y <= S.end_y; y++) {
        uint8_t *mrow = mask + (long long)(y - S.start_y) * S.mask_w;
        for (int32_t off = 0; off < sc; off++) {
            const int32_t ys = y * sc + off;
            if (ys >= bp[bpi]) {  // WorkingEdgeSet.rescan (Polygon.zig:275-300)
                int32_t to = 0;
                for (int32_t from = 0; from < n; from++) {
                    const DEdge &e = E[perm[from]];
                    if (e.rt <= ys && ys < e.rb) {
                        if (from != to) {
                            const int32_t t = perm[to]; perm[to] = perm[from]; perm[from] = t;
                        }
                        to++;
                    }
                }
                n_active = to;
                if (bpi < nbp - 1) bpi++;
            }
            const double ym = (double)ys + 0.5;
            for (int32_t k = 0; k < n_active; k++) {
                const DEdge &e = E[perm[k]];
                xv[k] = (int32_t)round(e.x_start + (e.x_inc * (ym - e.top)));
            }
            sort_insertion(perm, xv, n_active);
            int32_t fl = n_active;
            if (F.rule == Z2D_FILL_NON_ZERO) {  // WorkingEdgeSet.filter
                int32_t wn = 0, to = 0;
                for (int32_t from = 0; from < n_active; from++) {
                    xv[to] = xv[from];
                    if (wn == 0) {
                        wn += edge_dir(E[perm[from]]);
                        to++;
                    } else {
                        wn += edge_dir(E[perm[from]]);
                        if (wn == 0) to++;
                    }
                }
                fl = to;
            }
            if (direct) {
                if (!bounded && fl == 0) {
                    for (int32_t x = 0; x < sw; x++) mrow[x] = kMaskClear;
                    continue;
                }
                for (int32_t p = 0; p < fl / 2; p++) {
                    const int32_t sx = max(0, xv[2 * p]);
                    if (sx >= sw) break;
                    const int32_t ex = clampi(xv[2 * p + 1], sx, sw);
                    if (!bounded)
                        for (int32_t x = 0; x < sx; x++) mrow[x] = kMaskClear;
                    for (int32_t x = sx; x < ex; x++) mrow[x] = (uint8_t)((mrow[x] & kMaskClear) | 1);
                    if (!bounded)
                        for (int32_t x = ex; x < sw; x++) mrow[x] = kMaskClear;
                }
            } else {
                int32_t x_min = 0;
                for (int32_t p = 0; p < fl / 2; p++) {
                    const int32_t sx = max(x_min, xv[2 * p] - sxs);
                    if (sx >= dws) break;
                    const int32_t ex = clampi(xv[2 * p + 1] - sxs, sx, dws);
                    for (int32_t c = sx; c < ex; c++) mrow[c >> 2] = (uint8_t)(mrow[c >> 2] + 1);
                    x_min = ex;
                }
            }
        }
    }
}

// Work estimate of each raster tile for the cost-ordered queue: the number
// of fills in its band's list (every one is visited by the tile's rows).
__global__ void k_tile_cost(const DevJob *__restrict__ jobs, int32_t n_jobs, const int32_t *__restrict__ band_count,
                            int32_t n_tiles, int32_t *__restrict__ cost, int32_t *__restrict__ idx) {
    const int32_t t = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= n_tiles) return;
    const int32_t j = job_of(jobs, n_jobs, t, [](const DevJob &J) { return (long long)J.tile_base; });
    const DevJob J = jobs[j];
    const int32_t ncols = J.tcol_hi - J.tcol_lo + 1;
    cost[t] = band_count[J.gband_base + (t - J.tile_base) / ncols];
    idx[t] = t;
}

// The fill owning each node: warp f writes f over fill f's node range (the
// ranges are disjoint; fills drawing stroke polygons own no nodes).
__global__ void k_node_owner(const FillCmd *__restrict__ fills, int32_t n_fills, int32_t *__restrict__ node_fill) {
    const int32_t f = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (f >= n_fills) return;
    const int32_t o = fills[f].node_off, n = fills[f].n_nodes;
    for (int32_t k = lane; k < n; k += 32) node_fill[o + k] = f;
}

// ----------------------------------------------------------- host side
static inline unsigned grid_for(long long n, int threads) { return (unsigned)((n + threads - 1) / threads); }

int run_jobs(Ctx &c, std::vector<DevJob> &jobs, const z2d_node *nodes, int32_t n_nodes, std::vector<FillCmd> &fills,
             const std::vector<DevGradient> &grads,
             const std::vector<int32_t> &grad_of_fill, const StrokeSet *strokes) {
    if (n_nodes < 0) return Z2D_ERR_INVALID_ARGUMENT;
    const int32_t n_fills = (int32_t)fills.size();
    const int32_t n_jobs = (int32_t)jobs.size();
    if (n_fills == 0 || n_nodes == 0 || n_jobs == 0) return Z2D_OK;
    if (!strokes) {  // few short fills: one launch
        bool done = false;
        const int rc = run_small_jobs(c, jobs, nodes, fills, grads, grad_of_fill, done);
        if (rc || done) return rc;
    }
    for (DevJob &J : jobs) {
        J.band_lo = J.tcol_lo = 0x7FFFFFFF;
        J.band_hi = J.tcol_hi = -1;
        J.gband_base = J.tile_base = 0;
        J.list_base = 0;
    }
    // packed surfaces of an odd length are drawn on padded copies
    PackedPads pads;
    {
        const int rc = pads.begin(c, jobs.size(), [&](size_t j) -> DevSurface & { return jobs[j].sfc; });
        if (rc) return rc;
    }
    // ---- upload: gradients | fills | jobs | counters | strokes | polygons
    // through the pinned staging buffer, then the nodes straight from the
    // caller's memory
    auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t o_grads = 0;
    const size_t o_ext = al(o_grads + sizeof(DevGradient) * grads.size());  // stop tables of long gradients
    const size_t o_fills = al(o_ext + ext_stops_bytes(grads.data(), grads.size()));
    const size_t o_jobs = al(o_fills + sizeof(FillCmd) * (size_t)n_fills);
    const size_t o_cnt = al(o_jobs + sizeof(DevJob) * (size_t)n_jobs);
    const bool has_strokes = strokes && !strokes->empty();
    const size_t n_sk = has_strokes ? strokes->strokes.size() : 0, n_sb = has_strokes ? strokes->subs.size() : 0;
    const size_t n_tr = has_strokes ? strokes->trig.size() : 0;
    const size_t o_sk = al(o_cnt + sizeof(int32_t) * CNT_COUNT);
    const size_t o_sb = al(o_sk + sizeof(StrokeDev) * n_sk);
    const size_t o_tr = al(o_sb + sizeof(SubpathDev) * n_sb);
    // host-built polygons: per polygon its edge count, per contour its
    // start / size / fill / first edge, then the points
    const size_t n_poly = has_strokes ? strokes->polys.size() : 0;
    std::vector<int32_t> poly_fill(n_poly, -1);
    for (int32_t f = 0; f < n_fills; f++)
        if (fills[f].poly >= 0) poly_fill[(size_t)fills[f].poly] = f;
    long long n_pts = 0, n_ctr = 0;
    for (size_t k = 0; k < n_poly; k++) {
        const long long np = (long long)strokes->polys[k]->points();
        if (np > 0x7FFFFFFFll) {
            set_error("batch too large: more than 2^31 edges in one polygon");
            return Z2D_ERR_INVALID_ARGUMENT;
        }
        n_pts += np;
        n_ctr += (long long)strokes->polys[k]->ends.size();
    }
    if (n_ctr > 0x7FFFFFFFll) {
        set_error("batch too large: more than 2^31 contours");
        return Z2D_ERR_INVALID_ARGUMENT;
    }
    const size_t o_pe = al(o_tr + sizeof(double) * n_tr);
    const size_t o_cs = al(o_pe + sizeof(int32_t) * n_poly);
    const size_t o_cn = al(o_cs + sizeof(long long) * (size_t)n_ctr);
    const size_t o_cf = al(o_cn + sizeof(int32_t) * (size_t)n_ctr);
    const size_t o_ce = al(o_cf + sizeof(int32_t) * (size_t)n_ctr);
    const size_t o_pt = al(o_ce + sizeof(int32_t) * (size_t)n_ctr);
    const size_t total = al(o_pt + sizeof(double) * 2 * (size_t)n_pts);
    const size_t o_nodes = total;
    if (c.params.ensure(o_nodes + sizeof(z2d_node) * (size_t)n_nodes) || c.staging.ensure(total))
        return Z2D_ERR_OUT_OF_MEMORY;
    uint8_t *h = c.staging.as<uint8_t>();
    uint8_t *dv = c.params.as<uint8_t>();
    const DevGradient *dgrads = reinterpret_cast<const DevGradient *>(dv + o_grads);
    for (int32_t i = 0; i < n_fills; i++)
        if (grad_of_fill[i] >= 0) fills[i].src.grad = dgrads + grad_of_fill[i];
    // make sure the previous call's kernels no longer read the staging buffer
    Z2D_CUDA(cudaStreamSynchronize(c.stream));
    // (the flatten kernels are done with the nodes at the first readback
    // below, so the caller's array is free again when this call returns)
    Z2D_CUDA(cudaMemcpyAsync(dv + o_nodes, nodes, sizeof(z2d_node) * (size_t)n_nodes, cudaMemcpyHostToDevice, c.stream));
    if (!grads.empty()) {
        memcpy(h + o_grads, grads.data(), sizeof(DevGradient) * grads.size());
        put_ext_stops(reinterpret_cast<DevGradient *>(h + o_grads), grads.size(), h + o_ext, dv + o_ext);
    }
    memcpy(h + o_fills, fills.data(), sizeof(FillCmd) * (size_t)n_fills);
    memcpy(h + o_jobs, jobs.data(), sizeof(DevJob) * (size_t)n_jobs);
    int32_t *cnt_h = reinterpret_cast<int32_t *>(h + o_cnt);
    for (int i = 0; i < CNT_COUNT; i++) cnt_h[i] = 0;
    if (has_strokes) {
        memcpy(h + o_sk, strokes->strokes.data(), sizeof(StrokeDev) * n_sk);
        memcpy(h + o_sb, strokes->subs.data(), sizeof(SubpathDev) * n_sb);
        if (n_tr > 0) memcpy(h + o_tr, strokes->trig.data(), sizeof(double) * n_tr);
    }
    if (n_poly > 0) {
        int32_t *pe = reinterpret_cast<int32_t *>(h + o_pe);
        long long *cs = reinterpret_cast<long long *>(h + o_cs);
        int32_t *cn = reinterpret_cast<int32_t *>(h + o_cn), *cf = reinterpret_cast<int32_t *>(h + o_cf);
        int32_t *ce = reinterpret_cast<int32_t *>(h + o_ce);
        std::vector<long long> base(n_poly);
        long long pt = 0, ct = 0;
        for (size_t k = 0; k < n_poly; k++) {
            const stroke::Polygon &P = *strokes->polys[k];
            base[k] = pt;
            pe[k] = (int32_t)P.points();
            uint64_t prev = 0;
            for (uint64_t e : P.ends) {
                cs[ct] = pt + (long long)prev;
                cn[ct] = (int32_t)(e - prev);
                cf[ct] = poly_fill[k];
                ce[ct] = (int32_t)prev;
                prev = e;
                ct++;
            }
            pt += (long long)P.points();
        }
        // the points, polygon by polygon, over host threads
        double *hp = reinterpret_cast<double *>(h + o_pt);
        const size_t nt = std::min<size_t>(std::max(1u, std::thread::hardware_concurrency()),
                                           (size_t)(n_pts >> 20) + 1);
        std::atomic<size_t> next{0};
        auto work = [&] {
            for (size_t k; (k = next.fetch_add(1)) < n_poly;) {
                const stroke::Polygon &P = *strokes->polys[k];
                if (!P.xy.empty()) memcpy(hp + 2 * base[k], P.xy.data(), sizeof(double) * P.xy.size());
            }
        };
        std::vector<std::thread> pool;
        for (size_t t = 1; t < nt; t++) pool.emplace_back(work);
        work();
        for (auto &th : pool) th.join();
    }
    Z2D_CUDA(cudaMemcpyAsync(dv, h, total, cudaMemcpyHostToDevice, c.stream));
    const z2d_node *d_nodes = reinterpret_cast<const z2d_node *>(dv + o_nodes);
    const FillCmd *d_fills = reinterpret_cast<const FillCmd *>(dv + o_fills);
    DevJob *d_jobs = reinterpret_cast<DevJob *>(dv + o_jobs);
    int32_t *d_cnt = reinterpret_cast<int32_t *>(dv + o_cnt);

    // node info, then the curve queues and the nodes' fills
    const size_t info_bytes = (sizeof(NodeInfo) * (size_t)n_nodes + 255) & ~(size_t)255;
    const size_t st_bytes = (sizeof(FillState) * (size_t)n_fills + 255) & ~(size_t)255;
    if (c.node_info.ensure(info_bytes + (kCurveClasses + 2) * sizeof(int32_t) * (size_t)n_nodes) ||
        c.fill_state.ensure(st_bytes + (sizeof(RasterFill) + 32 * sizeof(uint32_t)) * (size_t)n_fills))
        return Z2D_ERR_OUT_OF_MEMORY;
    RasterFill *d_rf = reinterpret_cast<RasterFill *>(c.fill_state.as<uint8_t>() + st_bytes);
    uint32_t *d_luts = reinterpret_cast<uint32_t *>(d_rf + n_fills);  // per fill, its source word per coverage
    NodeInfo *d_info = c.node_info.as<NodeInfo>();
    // the curves to count, one queue per class, those to emit, then each
    // node's fill
    int32_t *d_curves = reinterpret_cast<int32_t *>(c.node_info.as<uint8_t>() + info_bytes);
    int32_t *d_curves_emit = d_curves + kCurveClasses * (size_t)n_nodes;
    int32_t *d_nfill = d_curves_emit + (size_t)n_nodes;
    FillState *d_st = c.fill_state.as<FillState>();
    Z2D_CUDA(cudaMemsetAsync(d_st, 0, sizeof(FillState) * (size_t)n_fills, c.stream));
    // each node's fill; nodes no fill owns (stroke commands' nodes, gaps) keep -1
    long long owned = 0;
    for (const FillCmd &F : fills) owned += F.n_nodes;
    if (owned < n_nodes) Z2D_CUDA(cudaMemsetAsync(d_nfill, 0xFF, sizeof(int32_t) * (size_t)n_nodes, c.stream));
    k_node_owner<<<grid_for(n_fills, 8), 256, 0, c.stream>>>(d_fills, n_fills, d_nfill);
    c.launches++;

    // ---- flatten
    const unsigned flat_blocks =
        (unsigned)std::min<long long>(grid_for((n_nodes + 31) / 32, kFlattenWarps), (long long)c.sm_count * 64);
    // one warp per queued curve, as many as there could be curves up to the
    // blocks the SMs hold at once: a grid of one wave, so the grid-stride
    // loop over the queue has no partial second wave
    static std::atomic<int> curve_occ{0};
    int curve_res = curve_occ.load(std::memory_order_relaxed);
    if (curve_res <= 0) {
        int a = 0, b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_curve_count_w, 32 * kFlattenWarps, 0) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_curve_emit_w, 32 * kFlattenWarps, 0) != cudaSuccess)
            a = b = 4;
        curve_res = std::max(1, std::min(a, b));
        curve_occ.store(curve_res, std::memory_order_relaxed);
    }
    const unsigned curve_blocks =
        (unsigned)std::min<long long>(grid_for(n_nodes, kFlattenWarps), (long long)c.sm_count * curve_res);
    // per curve warp: kScratch leaf points per lane; then the curve pool
    const size_t scratch_pts = (size_t)curve_blocks * kFlattenWarps * 32 * kScratch;
    // pool capacity: 32 points per node, or what the previous call asked for
    const int32_t pool_cap = (int32_t)std::min<long long>(
        64ll << 20, std::max<long long>({1ll << 20, 32ll * n_nodes, c.pool_demand + c.pool_demand / 4}));
    if (c.curve_pool.ensure(sizeof(double2) * (scratch_pts + (size_t)pool_cap))) return Z2D_ERR_OUT_OF_MEMORY;
    double2 *d_scratch = c.curve_pool.as<double2>();
    double2 *d_pool = d_scratch + scratch_pts;
    cudaEvent_t tf = c.timer_begin(c.t_flatten);
    k_node_count_w<<<flat_blocks, 32 * kFlattenWarps, 0, c.stream>>>(d_nodes, d_nfill, d_fills, d_info, n_nodes,
                                                                    d_curves, d_cnt);
    k_curve_count_w<<<curve_blocks, 32 * kFlattenWarps, 0, c.stream>>>(d_nodes, d_nfill, d_fills, d_info, n_nodes,
                                                                      d_curves, d_cnt, d_cnt + CNT_STATUS, d_scratch,
                                                                      d_pool, pool_cap);
    StrokeRun srun;
    if (n_sk > 0) {
        srun.nodes = d_nodes;
        srun.strokes = reinterpret_cast<const StrokeDev *>(dv + o_sk);
        srun.subs = reinterpret_cast<const SubpathDev *>(dv + o_sb);
        srun.trig = reinterpret_cast<const double *>(dv + o_tr);
        srun.n_strokes = (int32_t)n_sk;
        srun.n_subs = (int32_t)n_sb;
        srun.n_local = strokes->n_local;
        srun.n_pen = strokes->n_pen;
        const int rc = stroke_count(c, srun, d_cnt + CNT_STATUS);
        if (rc) return rc;
    }
    k_fill_scan<<<grid_for(n_fills, kScanWarps), 32 * kScanWarps, 0, c.stream>>>(
        d_nodes, d_fills, d_info, d_st, n_fills, d_cnt, d_cnt + CNT_STATUS, srun.stroke_edges,
        reinterpret_cast<const int32_t *>(dv + o_pe));
    c.timer_end(c.t_flatten, tf);
    c.launches += 3;
    const size_t rb_jobs_off = al(sizeof(int32_t) * CNT_COUNT + 2 * sizeof(long long));
    const size_t rb_bytes = rb_jobs_off + sizeof(DevJob) * (size_t)n_jobs;
    if (c.readback.ensure(rb_bytes)) return Z2D_ERR_OUT_OF_MEMORY;
    int32_t *rb = c.readback.as<int32_t>();
    long long *rb_tot = reinterpret_cast<long long *>(rb + CNT_COUNT);  // stroke contour totals (8-aligned: CNT_COUNT even)
    DevJob *rb_jobs = reinterpret_cast<DevJob *>(c.readback.as<uint8_t>() + rb_jobs_off);
    Z2D_CUDA(cudaMemcpyAsync(rb, d_cnt, sizeof(int32_t) * CNT_COUNT, cudaMemcpyDeviceToHost, c.stream));
    if (n_sk > 0)
        Z2D_CUDA(cudaMemcpyAsync(rb_tot, stroke_totals_dev(srun), 2 * sizeof(long long), cudaMemcpyDeviceToHost,
                                 c.stream));
    Z2D_CUDA(cudaStreamSynchronize(c.stream));
    c.pool_demand = (long long)std::min<unsigned long long>(
        64ull << 20, ((unsigned long long)(uint32_t)rb[CNT_POOL + 1] << 32) | (uint32_t)rb[CNT_POOL]);
    if (rb[CNT_STATUS] != 0) {
        set_error(rb[CNT_STATUS] == Z2D_ERR_INVALID_STATE ? "curve subdivision exceeded its depth bound"
                                                          : "batch too large: more than 2^31 edges in one polygon");
        return rb[CNT_STATUS];
    }
    if (n_sk > 0) {
        srun.n_a = rb_tot[0];
        srun.n_b = rb_tot[1];
    }
    const int32_t n_edges = rb[CNT_EDGES];
    if (n_edges < 0) return Z2D_ERR_OUT_OF_MEMORY;
    if (c.edges.ensure(sizeof(DEdge) * (size_t)std::max(n_edges, 1) + sizeof(int32_t) * (size_t)std::max(n_edges, 1)))
        return Z2D_ERR_OUT_OF_MEMORY;
    DEdge *d_edges = c.edges.as<DEdge>();
    int32_t *d_edge_fill = reinterpret_cast<int32_t *>(d_edges + std::max(n_edges, 1));
    // extents start at +inf/-inf keys: min slots 0xFF.., max slots 0
    tf = c.timer_begin(c.t_flatten);
    k_node_emit_w<<<flat_blocks, 32 * kFlattenWarps, 0, c.stream>>>(d_nodes, d_nfill, d_fills, d_info, d_st, d_edges,
                                                                   n_nodes, d_curves_emit, d_cnt);
    k_curve_emit_w<<<curve_blocks, 32 * kFlattenWarps, 0, c.stream>>>(d_nodes, d_nfill, d_fills, d_info, d_st,
                                                                     d_edges, d_curves_emit, d_cnt, d_pool);
    if (n_sk > 0) {
        const int rc = stroke_emit(c, srun, d_fills, d_st, d_edges);
        if (rc) return rc;
    }
    if (n_ctr > 0) {
        PolyRun pr;
        pr.pts = reinterpret_cast<const double2 *>(dv + o_pt);
        pr.start = reinterpret_cast<const long long *>(dv + o_cs);
        pr.n = reinterpret_cast<const int32_t *>(dv + o_cn);
        pr.fill = reinterpret_cast<const int32_t *>(dv + o_cf);
        pr.edge_off = reinterpret_cast<const int32_t *>(dv + o_ce);
        pr.n_contours = (int32_t)n_ctr;
        pr.n_points = n_pts;
        const int rc = poly_emit(c, pr, d_fills, d_st, d_edges);
        if (rc) return rc;
    }
    k_edge_fill<<<n_fills, 128, 0, c.stream>>>(d_st, d_fills, d_jobs, d_edge_fill, d_luts);
    k_fill_setup<<<grid_for(n_fills, 64), 64, 0, c.stream>>>(d_fills, d_st, n_fills, d_jobs, d_cnt, d_rf);
    c.timer_end(c.t_flatten, tf);
    c.launches += 4;
    Z2D_CUDA(cudaMemcpyAsync(rb, d_cnt, sizeof(int32_t) * CNT_COUNT, cudaMemcpyDeviceToHost, c.stream));
    Z2D_CUDA(cudaMemcpyAsync(rb_jobs, d_jobs, sizeof(DevJob) * (size_t)n_jobs, cudaMemcpyDeviceToHost, c.stream));
    Z2D_CUDA(cudaStreamSynchronize(c.stream));
    const int32_t n_fb = rb[CNT_FILL_BANDS];
    const long long mask_bytes = (long long)(((unsigned long long)(uint32_t)rb[CNT_MASK_LO + 1] << 32) | (uint32_t)rb[CNT_MASK_LO]);
    const int32_t n_exact = rb[CNT_EXACT];
    // ---- layout: global bands, raster CTAs and band-list slots, job after job
    long long n_gbands = 0, n_tiles = 0, n_slots = 0;
    for (int32_t j = 0; j < n_jobs; j++) {
        DevJob &J = jobs[j];
        J.band_lo = rb_jobs[j].band_lo;
        J.band_hi = rb_jobs[j].band_hi;
        J.tcol_lo = rb_jobs[j].tcol_lo;
        J.tcol_hi = rb_jobs[j].tcol_hi;
        J.gband_base = (int32_t)n_gbands;
        J.tile_base = (int32_t)n_tiles;
        J.list_base = n_slots;
        if (J.band_hi < J.band_lo || J.tcol_hi < J.tcol_lo) {  // nothing is drawn on this surface
            J.band_lo = 0;
            J.band_hi = -1;
            J.tcol_lo = 0;
            J.tcol_hi = -1;
            continue;
        }
        const long long nb = J.band_hi - J.band_lo + 1, nc = J.tcol_hi - J.tcol_lo + 1;
        n_gbands += nb;
        n_tiles += nb * nc;
        n_slots += nb * (J.fill1 - J.fill0);
    }
    if (n_gbands == 0) return pads.finish(c);  // nothing is drawn
    if (n_tiles > 0x7FFFFFFFll || n_gbands > 0x7FFFFFFFll) {
        set_error("batch too large: more than 2^31 tiles");
        return Z2D_ERR_INVALID_ARGUMENT;
    }
    memcpy(rb_jobs, jobs.data(), sizeof(DevJob) * (size_t)n_jobs);
    Z2D_CUDA(cudaMemcpyAsync(d_jobs, rb_jobs, sizeof(DevJob) * (size_t)n_jobs, cudaMemcpyHostToDevice, c.stream));

    // ---- bins: counts, exclusive scan, scatter
    if (c.bin_offsets.ensure(sizeof(int32_t) * (2 * (size_t)n_fb + 2))) return Z2D_ERR_OUT_OF_MEMORY;
    int32_t *d_fb_cnt = c.bin_offsets.as<int32_t>();
    int32_t *d_fb_off = d_fb_cnt + (n_fb + 1);
    Z2D_CUDA(cudaMemsetAsync(d_fb_cnt, 0, sizeof(int32_t) * (size_t)(n_fb + 1), c.stream));
    cudaEvent_t tb = c.timer_begin(c.t_bins);
    if (n_edges > 0) {
        k_bin_count<<<grid_for(n_edges, 256), 256, 0, c.stream>>>(d_fills, d_st, d_edges, d_edge_fill, n_edges, d_fb_cnt,
                                                                   d_cnt + CNT_STATUS);
        c.launches++;
    }
    size_t tmp_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, d_fb_cnt, d_fb_off, n_fb + 1, c.stream);
    if (c.scan_tmp.ensure(tmp_bytes + 16)) return Z2D_ERR_OUT_OF_MEMORY;
    Z2D_CUDA(cub::DeviceScan::ExclusiveSum(c.scan_tmp.ptr, tmp_bytes, d_fb_cnt, d_fb_off, n_fb + 1, c.stream));
    c.timer_end(c.t_bins, tb);
    c.launches++;
    Z2D_CUDA(cudaMemcpyAsync(rb, d_fb_off + n_fb, sizeof(int32_t), cudaMemcpyDeviceToHost, c.stream));
    Z2D_CUDA(cudaMemcpyAsync(rb + 1, d_cnt + CNT_STATUS, sizeof(int32_t), cudaMemcpyDeviceToHost, c.stream));
    Z2D_CUDA(cudaStreamSynchronize(c.stream));
    const int32_t n_bin_entries = rb[0];
    if (rb[1] != 0) {
        set_error("a fill has more than 32000 edges inside one 4-row band");
        return rb[1];
    }
    // the band lists and the exact path's masks, then the bins: what is left
    // decides whether they hold records or, an eighth of them, indices
    const size_t count_bytes = ((sizeof(int32_t) * (size_t)n_gbands) + 15) & ~(size_t)15;
    const size_t tile_bytes = n_jobs > 1 ? sizeof(TileRec) * (size_t)n_tiles : 0;
    if (c.band_fills.ensure(count_bytes + tile_bytes + sizeof(int4) * (size_t)std::max(n_slots, 1ll)))
        return Z2D_ERR_OUT_OF_MEMORY;
    // masks plus per-fill work arrays
    if (n_exact > 0 && c.masks.ensure((size_t)mask_bytes + 64)) return Z2D_ERR_OUT_OF_MEMORY;
    BinKind bin_kind = kBinRecords;
    if (c.bins.ensure(sizeof(BinEdge) * (size_t)std::max(n_bin_entries, 1))) {
        bin_kind = kBinIndex;
        if (c.bins.ensure(sizeof(int32_t) * (size_t)std::max(n_bin_entries, 1))) return Z2D_ERR_OUT_OF_MEMORY;
    }
    // scatter with the counts array reused as cursors
    Z2D_CUDA(cudaMemcpyAsync(d_fb_cnt, d_fb_off, sizeof(int32_t) * (size_t)(n_fb + 1), cudaMemcpyDeviceToDevice, c.stream));
    tb = c.timer_begin(c.t_bins);
    if (n_edges > 0 && n_bin_entries > 0) {
        const auto bin_fill = bin_kind == kBinRecords ? k_bin_fill<true> : k_bin_fill<false>;
        bin_fill<<<grid_for(n_edges, 256), 256, 0, c.stream>>>(d_fills, d_st, d_edges, d_edge_fill, n_edges, d_fb_cnt,
                                                                c.bins.ptr);
        c.launches++;
    }

    // ---- ordered fill lists per global band
    int32_t *d_band_count = c.band_fills.as<int32_t>();
    TileRec *d_tiles = n_jobs > 1 ? reinterpret_cast<TileRec *>(c.band_fills.as<uint8_t>() + count_bytes) : nullptr;
    int4 *d_band_fills = reinterpret_cast<int4 *>(c.band_fills.as<uint8_t>() + count_bytes + tile_bytes);
    // A warp per band where the jobs have few fills on average, and then a CTA
    // for the bands of the jobs of more than kWarpFills: 2,000 surfaces of one
    // fill beside one of n, all bins and lists: n = 256 by warps 50.5 us, by
    // CTAs 54.7; 512 58.1 and 54.4; 1,024 68.9 and 57.8; 4,096 142 and 75.
    const int32_t max_fills = n_slots <= 256 * n_gbands ? kWarpFills : 0;
    if (max_fills > 0) {
        k_band_lists_w<<<grid_for(32 * n_gbands, 256), 256, 0, c.stream>>>(d_st, d_jobs, n_jobs, (int32_t)n_gbands,
                                                                            max_fills, d_band_count, d_band_fills,
                                                                            d_tiles);
        c.launches++;
    }
    long long gb0 = n_gbands, gb1 = 0;  // from the first of the other jobs' bands to the last
    for (const DevJob &J : jobs)
        if (J.fill1 - J.fill0 > max_fills && J.band_hi >= J.band_lo) {
            gb0 = std::min<long long>(gb0, J.gband_base);
            gb1 = (long long)J.gband_base + (J.band_hi - J.band_lo + 1);
        }
    if (gb0 < gb1) {
        k_band_lists<<<(unsigned)(gb1 - gb0), 256, 0, c.stream>>>(d_st, d_jobs, n_jobs, (int32_t)gb0, max_fills,
                                                                 d_band_count, d_band_fills, d_tiles);
        c.launches++;
    }

    // ---- exact path
    if (n_exact > 0) {
        Z2D_CUDA(cudaMemsetAsync(c.masks.ptr, 0, (size_t)mask_bytes, c.stream));
        k_exact<<<grid_for(n_fills, 32), 32, 0, c.stream>>>(d_fills, d_st, d_edges, n_fills, d_jobs, c.masks.as<uint8_t>());
        c.launches++;
    }
    c.timer_end(c.t_bins, tb);

    // ---- raster
    RasterArgs A;
    A.jobs = d_jobs;
    A.fills = d_fills;
    A.st = d_st;
    A.edges = d_edges;
    A.bins = c.bins.ptr;
    A.bin_off = d_fb_off;
    A.band_count = d_band_count;
    A.band_fills = d_band_fills;
    A.rfills = d_rf;
    A.luts = d_luts;
    A.tiles = d_tiles;
    A.masks = c.masks.as<uint8_t>();
    A.job0 = jobs[0];
    {
        const int rc = c.await_surface();  // a host surface's upload
        if (rc) return rc;
    }
    // persistent grid: every SM filled to the kernel's residency (or the
    // tuned CTAs per SM), never more CTAs than tiles
    RasterVariant variant{n_jobs > 1, false, bin_kind, raster_mode(fills.data(), fills.size(), n_exact > 0)};
    if (bin_kind == kBinIndex) variant.mode = kGeneral;
    int occ = 1;
    {
        const int rc = raster_occupancy(c, variant, occ);
        if (rc) return rc;
    }
    // the schedule: forced on the context, or the tuner's for this kind of pass
    const TuneKey key = tune_key(n_jobs, variant.mode, n_tiles, n_slots, n_gbands);
    c.last_key = key;
    RasterPlan plan{c.raster_ctas_per_sm, c.raster_order, c.raster_cta_items, -1};
    if (bin_kind == kBinIndex) {  // (one schedule: its variants draw rows)
        plan = RasterPlan{0, 0, 0, -1};
    } else if (!c.raster_forced) {
        c.tune_collect(false);
        plan = tune_pick(key);
    }
    cudaEvent_t tune_t0 = nullptr, tune_t1 = nullptr;
    if (plan.candidate >= 0) {
        if (cudaEventCreate(&tune_t0) != cudaSuccess || cudaEventCreate(&tune_t1) != cudaSuccess) {
            if (tune_t0) cudaEventDestroy(tune_t0);
            tune_t0 = tune_t1 = nullptr;
            plan.candidate = -1;
        } else {
            Z2D_CUDA(cudaEventRecord(tune_t0, c.stream));
        }
    }
    // ctas < 0: one CTA per tile (a tile per item), else a persistent grid
    const int per_sm = plan.ctas > 0 ? std::min(plan.ctas, occ) : occ;
    const bool one_per_tile = plan.ctas < 0;
    const unsigned grid =
        one_per_tile ? (unsigned)n_tiles : (unsigned)std::min<long long>(n_tiles, (long long)c.sm_count * per_sm);
    if (one_per_tile) plan.cta_items = 1;
    A.one_per_tile = one_per_tile ? 1 : 0;
    A.queue = reinterpret_cast<unsigned long long *>(d_cnt + CNT_QUEUE);
    A.n_items = (unsigned long long)n_tiles * (plan.cta_items ? 1 : kTileRows);
    A.order = nullptr;
    if (plan.order == 1 && n_tiles > 1) {
        // longest bands first: tiles sorted by their band's fill count (in tile
        // order where there is no room to sort them)
        const size_t nt = (size_t)n_tiles;
        size_t sort_bytes = 0;
        cub::DeviceRadixSort::SortPairsDescending(nullptr, sort_bytes, (const int32_t *)nullptr, (int32_t *)nullptr,
                                                  (const int32_t *)nullptr, (int32_t *)nullptr, (int)nt, 0, 32,
                                                  c.stream);
        const size_t arr = (sizeof(int32_t) * nt + 255) & ~(size_t)255;
        if (c.tile_order.ensure(4 * arr + sort_bytes) == 0) {
            uint8_t *b = c.tile_order.as<uint8_t>();
            int32_t *cost = reinterpret_cast<int32_t *>(b), *idx = reinterpret_cast<int32_t *>(b + arr);
            int32_t *cost_s = reinterpret_cast<int32_t *>(b + 2 * arr), *order = reinterpret_cast<int32_t *>(b + 3 * arr);
            k_tile_cost<<<grid_for((long long)nt, 256), 256, 0, c.stream>>>(d_jobs, n_jobs, d_band_count, (int32_t)nt,
                                                                             cost, idx);
            Z2D_CUDA(cub::DeviceRadixSort::SortPairsDescending(b + 4 * arr, sort_bytes, cost, cost_s, idx, order,
                                                               (int)nt, 0, 32, c.stream));
            c.launches += 2;
            A.order = order;
        }
    }
    cudaEvent_t t0 = c.timer_begin(c.t_raster);
    variant.cta_items = plan.cta_items != 0;
    {
        const int rc = raster_launch(c, variant, A, grid);
        if (rc) return rc;
    }
    c.timer_end(c.t_raster, t0);
    if (plan.candidate >= 0) {
        Z2D_CUDA(cudaEventRecord(tune_t1, c.stream));
        c.tune_pending.push_back(TunePending{key, plan.candidate, tune_t0, tune_t1});
    }
    return pads.finish(c);
}

// ------------------------------------------------------- small fills
// One fill of a short path: everything up to the rasteriser runs on the
// host (a few microseconds for a few hundred edges) and reaches the device
// with the rasteriser's one launch (tables of up to 8 KB, its parameters) or
// in one copy in front of it, instead of the pipeline's launches and size
// readbacks.  The host steps restate the same
// z2d code as the device kernels, with the same f64 operations in the same
// order (the host is compiled without FP contraction), so the edges, the
// fill's box and the tiles are the device pipeline's; bins list a band's
// edges in any order (the rasteriser's sums do not depend on it).
namespace {

// The host's work grows with the edges (about 20-30 ns each to flatten and
// bin) while the pipeline's cost is mostly fixed (~100 us of launches and
// readbacks for a small call), so the path takes calls whose edge count,
// estimated before and counted while flattening, stays below a budget:
// one surface up to 4,096 edges; several (as in the server's passes under
// load, where the pipeline's fixed cost is shared) up to 1,024 on at most
// 8 surfaces.
constexpr int32_t kSmallMaxNodes = 4096;       // nodes of all the call's fills
constexpr size_t kSmallEdgesOne = 4096;        // edge budget, one surface
constexpr size_t kSmallEdgesMany = 1024;       // edge budget, several surfaces
constexpr size_t kSmallMaxJobs = 8;
constexpr size_t kSmallMaxBins = 1 << 17;      // (edge, band) pairs
constexpr long long kSmallMaxBands = 1 << 16;  // (fill, band) slots and band-list entries
constexpr int kSmallMaxDepth = 40;  // below the device subdivision bound

struct HostFlatten {
    const FillCmd &F;
    std::vector<SmallEdge> &edges;
    size_t max_edges;
    double et = 0, eb = 0, el = 0, er = 0;
    bool any = false, overflow = false;
    // PointBuffer(1, 3) of fill_plotter: its first and last points and length
    double fx = 0, fy = 0, lx = 0, ly = 0;
    int count = 0;

    // Polygon.addEdge (Polygon.zig:61-109), as add_edge in edges.cuh
    void edge(double x0, double y0, double x1, double y1) {
        if (edges.size() >= max_edges) {
            overflow = true;
            return;
        }
        const double ax = x0 * F.edge_scale, ay = y0 * F.edge_scale, bx = x1 * F.edge_scale, by = y1 * F.edge_scale;
        SmallEdge e{};
        if (ay < by) {
            e.top = ay;
            e.x_start = ax;
            e.x_inc = (bx - ax) / (by - ay);
            e.rb2 = 2 * (int32_t)std::round(by) + 1;
        } else if (ay > by) {
            e.top = by;
            e.x_start = bx;
            e.x_inc = (ax - bx) / (ay - by);
            e.rb2 = 2 * (int32_t)std::round(ay);
        } else {
            e.rt = 1;  // rb = 0: never active
            edges.push_back(e);
            return;
        }
        e.rt = (int32_t)std::round(e.top);
        const double bot = ay < by ? by : ay;
        const double l = ax < bx ? ax : bx, r = ax < bx ? bx : ax;
        if (!any) {
            et = e.top, eb = bot, el = l, er = r;
            any = true;
        } else {
            if (e.top < et) et = e.top;
            if (bot > eb) eb = bot;
            if (l < el) el = l;
            if (r > er) er = r;
        }
        edges.push_back(e);
    }
    // lineTo through the point buffer (fill_plotter.zig:44-51, 100-118)
    void line_to(double x, double y) {
        if (lx == x && ly == y) return;
        edge(lx, ly, x, y);
        lx = x;
        ly = y;
        count = count < 3 ? count + 1 : 3;
    }
    struct K {
        double ax, ay, bx, by, cx, cy, dx, dy;
    };
    static double error_sq(const K &k) {  // Spline.Knots.errorSq (Spline.zig:83-123)
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
    // Spline.decompose / decomposeInto (Spline.zig:37-79): depth-first, the
    // first half before the second, leaves' start points then d
    bool curve(const double *p) {
        const double ax = lx, ay = ly;
        if (ax == p[0] && ay == p[1] && p[2] == p[4] && p[3] == p[5]) {
            line_to(p[4], p[5]);
            return true;
        }
        const double tol2 = F.tol * F.tol;
        struct Item {
            K k;
            int depth;
        };
        Item stack[kSmallMaxDepth + 2];
        int top = 0;
        stack[top++] = Item{K{ax, ay, p[0], p[1], p[2], p[3], p[4], p[5]}, 0};
        auto half = [](double a, double b) { return a + ((b - a) / 2); };
        while (top > 0) {
            Item it = stack[--top];
            K &k = it.k;
            if (error_sq(k) < tol2) {
                if (!(k.ax == ax && k.ay == ay)) line_to(k.ax, k.ay);
                if (overflow) return true;
                continue;
            }
            if (it.depth >= kSmallMaxDepth) return false;
            // deCasteljau: k becomes the first half, s2 the second
            const double abx = half(k.ax, k.bx), aby = half(k.ay, k.by);
            const double bcx = half(k.bx, k.cx), bcy = half(k.by, k.cy);
            const double cdx = half(k.cx, k.dx), cdy = half(k.cy, k.dy);
            const double abbcx = half(abx, bcx), abbcy = half(aby, bcy);
            const double bccdx = half(bcx, cdx), bccdy = half(bcy, cdy);
            const double fx_ = half(abbcx, bccdx), fy_ = half(abbcy, bccdy);
            const K s2{fx_, fy_, bccdx, bccdy, cdx, cdy, k.dx, k.dy};
            const K s1{k.ax, k.ay, abx, aby, abbcx, abbcy, fx_, fy_};
            stack[top++] = Item{s2, it.depth + 1};
            stack[top++] = Item{s1, it.depth + 1};
        }
        line_to(p[4], p[5]);
        return true;
    }
    // fill_plotter.plot (fill_plotter.zig:21-97); false: not for this path
    bool plot(const z2d_node *nodes, int32_t n, bool &open_chain) {
        for (int32_t i = 0; i < n && !overflow; i++) {
            const z2d_node &nd = nodes[i];
            switch (nd.tag) {
                case Z2D_MOVE_TO:
                    if (i == n - 1) return true;  // the auto-added move_to after close_path
                    fx = lx = nd.p[0];
                    fy = ly = nd.p[1];
                    count = 1;
                    break;
                case Z2D_LINE_TO:
                    if (count == 0) return false;  // InvalidState: the pipeline reports it
                    line_to(nd.p[0], nd.p[1]);
                    break;
                case Z2D_CURVE_TO:
                    if (count == 0) return false;
                    if (!curve(nd.p)) return false;
                    break;
                default:  // close_path
                    if (count >= 3) {
                        if (!(lx == fx && ly == fy)) {
                            edge(lx, ly, fx, fy);
                            lx = fx;
                            ly = fy;
                        }
                    } else if (count > 0 && !(lx == fx && ly == fy)) {
                        open_chain = true;
                    }
                    break;
            }
        }
        return !overflow;
    }
};

// An estimate of a path's edges before flattening it: one per line_to and
// close_path, and for a curve 2^k leaves with k the levels of halving that
// bring the initial knots' errorSq below tol^2 (each halving divides it by
// about 16).
size_t estimate_edges(const z2d_node *nodes, int32_t n, double tol) {
    size_t est = 0;
    double lx = 0, ly = 0;
    const double tol2 = tol * tol;
    for (int32_t i = 0; i < n; i++) {
        const z2d_node &nd = nodes[i];
        if (nd.tag == Z2D_CURVE_TO) {
            const HostFlatten::K k{lx, ly, nd.p[0], nd.p[1], nd.p[2], nd.p[3], nd.p[4], nd.p[5]};
            const double e = HostFlatten::error_sq(k);
            size_t leaves = 1;
            if (e >= tol2) {
                const double lv = std::ceil(std::log2(e / tol2) / 4.0);
                leaves = lv >= 20.0 ? ((size_t)1 << 20) : ((size_t)1 << (size_t)std::max(0.0, lv));
            }
            est += leaves;
            lx = nd.p[4];
            ly = nd.p[5];
        } else {
            est += 1;
            if (nd.tag != Z2D_CLOSE_PATH) {
                lx = nd.p[0];
                ly = nd.p[1];
            }
        }
    }
    return est;
}

}  // namespace

int run_small_jobs(Ctx &c, std::vector<DevJob> &jobs, const z2d_node *nodes, const std::vector<FillCmd> &fills,
                   const std::vector<DevGradient> &grads, const std::vector<int32_t> &grad_of_fill, bool &done) {
    done = false;
    const size_t n_fills = fills.size(), n_jobs = jobs.size();
    if (n_fills == 0 || n_jobs == 0 || n_jobs > kSmallMaxJobs) return Z2D_OK;
    const size_t budget = n_jobs == 1 ? kSmallEdgesOne : kSmallEdgesMany;
    long long total_nodes = 0;
    for (const FillCmd &F : fills) {
        if (F.aa != Z2D_AA_MULTISAMPLE_4X || F.stroke >= 0 || F.poly >= 0 || F.n_nodes <= 0) return Z2D_OK;
        total_nodes += F.n_nodes;
    }
    if (total_nodes > kSmallMaxNodes) return Z2D_OK;
    size_t est = 0;
    for (const FillCmd &F : fills) {
        est += estimate_edges(nodes + F.node_off, F.n_nodes, F.tol);
        if (est > budget) return Z2D_OK;
    }
    for (const DevJob &J : jobs)
        if (fmt_packed(J.sfc.fmt)) return Z2D_OK;
    for (const DevGradient &g : grads)
        if (g.n_stops > kMaxStops) return Z2D_OK;
    // ---- flatten every fill (fill_plotter.plot)
    static thread_local std::vector<SmallEdge> edges;
    static thread_local std::vector<FillState> st;
    static thread_local std::vector<RasterFill> rf;
    static thread_local std::vector<double> ext;  // et, eb, el, er per fill
    edges.clear();
    st.assign(n_fills, FillState{});
    rf.assign(n_fills, RasterFill{});
    ext.assign(4 * n_fills, 0.0);
    for (size_t f = 0; f < n_fills; f++) {
        const size_t e0 = edges.size();
        HostFlatten H{fills[f], edges, budget};
        bool open_chain = false;
        if (!H.plot(nodes + fills[f].node_off, fills[f].n_nodes, open_chain) || open_chain) return Z2D_OK;
        st[f].edge_base = (int32_t)e0;
        st[f].n_edges = (int32_t)(edges.size() - e0);
        st[f].has_edges = H.any ? 1 : 0;
        ext[4 * f] = H.et, ext[4 * f + 1] = H.eb, ext[4 * f + 2] = H.el, ext[4 * f + 3] = H.er;
    }
    // ---- k_fill_setup per fill: Polygon.inBox, multisample.run's draw box,
    // the bands and tile columns it touches
    auto clampi_h = [](int32_t v, int32_t lo, int32_t hi) { return std::max(lo, std::min(v, hi)); };
    static thread_local std::vector<DevJob> J;
    J = jobs;
    for (DevJob &jb : J) {
        jb.band_lo = jb.tcol_lo = 0x7FFFFFFF;
        jb.band_hi = jb.tcol_hi = -1;
        jb.gband_base = jb.tile_base = 0;
        jb.list_base = 0;
    }
    long long n_fb = 0;
    for (size_t f = 0; f < n_fills; f++) {
        const FillCmd &F = fills[f];
        FillState &S = st[f];
        DevJob &jb = J[(size_t)F.job];
        const int32_t sw = jb.sfc.w, sh = jb.sfc.h;
        const double et = ext[4 * f], eb = ext[4 * f + 1], el = ext[4 * f + 2], er = ext[4 * f + 3];
        if (!S.has_edges || er < 0.0 || eb < 0.0) continue;
        const double sc = F.scale;
        const int32_t psx = (int32_t)std::floor(el / sc), psy = (int32_t)std::floor(et / sc);
        const int32_t pex = (int32_t)std::ceil(er / sc), pey = (int32_t)std::ceil(eb / sc);
        const int32_t pw = pex - psx, ph = pey - psy;
        if (pw == 0 || ph == 0 || psx + pw < 0 || psy + ph < 0 || psx >= sw || psy >= sh) continue;
        S.active = 1;
        S.start_y = clampi_h((int32_t)std::floor(et / 4.0), 0, sh - 1);
        S.end_y = clampi_h((int32_t)std::ceil(eb / 4.0), S.start_y, sh - 1);
        S.start_x = clampi_h((int32_t)std::floor(el / 4.0), 0, sw - 1);
        S.end_x = clampi_h((int32_t)std::ceil(er / 4.0), S.start_x, sw);
        const bool bounded = is_bounded(F.op);
        S.band0 = (bounded ? S.start_y : 0) / kTileRows;
        S.band1 = (bounded ? S.end_y : sh - 1) / kTileRows;
        S.fb_base = (int32_t)n_fb;
        n_fb += S.band1 - S.band0 + 1;
        S.cull_x0 = bounded ? S.start_x : 0;
        S.cull_x1 = bounded ? S.end_x : sw;
        jb.band_lo = std::min(jb.band_lo, S.band0);
        jb.band_hi = std::max(jb.band_hi, S.band1);
        jb.tcol_lo = std::min(jb.tcol_lo, S.cull_x0 / kTileCols);
        jb.tcol_hi = std::max(jb.tcol_hi, (std::max(S.cull_x1, S.cull_x0 + 1) - 1) / kTileCols);
        RasterFill &R = rf[f];
        R.start_x = S.start_x;
        R.end_x = S.end_x;
        R.start_y = S.start_y;
        R.end_y = S.end_y;
        R.meta = ((uint32_t)F.op & RF_OP_MASK) | ((uint32_t)F.aa << RF_AA_SHIFT) |
                 (F.rule == Z2D_FILL_EVEN_ODD ? RF_EVEN_ODD : 0u) | ((uint32_t)F.fast_kind << RF_FAST_SHIFT) |
                 (bounded ? RF_BOUNDED : 0u);
    }
    done = true;
    if (n_fb == 0) return Z2D_OK;  // nothing is drawn
    if (n_fb > kSmallMaxBands) {
        done = false;
        return Z2D_OK;
    }
    // ---- layout: global bands, tiles and band-list storage, job after job
    long long n_gbands = 0, n_tiles = 0, n_slots = 0;
    for (DevJob &jb : J) {
        jb.gband_base = (int32_t)n_gbands;
        jb.tile_base = (int32_t)n_tiles;
        jb.list_base = n_slots;
        if (jb.band_hi < jb.band_lo || jb.tcol_hi < jb.tcol_lo) {
            jb.band_lo = 0;
            jb.band_hi = -1;
            jb.tcol_lo = 0;
            jb.tcol_hi = -1;
            continue;
        }
        const long long nb = jb.band_hi - jb.band_lo + 1, nc = jb.tcol_hi - jb.tcol_lo + 1;
        n_gbands += nb;
        n_tiles += nb * nc;
        n_slots += nb * (jb.fill1 - jb.fill0);
    }
    if (n_slots > kSmallMaxBands || n_tiles > 0x7FFFFFFF) {
        done = false;
        return Z2D_OK;
    }
    // ---- bins: each edge in the bands of its active sample rows (edge_bands)
    static thread_local std::vector<int32_t> cnt, off, bins, bcount;
    static thread_local std::vector<TileRec> tiles;
    static thread_local std::vector<int4> blist;
    cnt.assign((size_t)n_fb + 1, 0);
    auto for_bands = [&](auto &&visit) {
        for (size_t f = 0; f < n_fills; f++) {
            const FillState &S = st[f];
            if (!S.active) continue;
            const int32_t S_ = (int32_t)fills[f].scale;
            for (int32_t k = 0; k < S.n_edges; k++) {
                const SmallEdge &e = edges[(size_t)(S.edge_base + k)];
                const int32_t lo = std::max(e.rt, S.start_y * S_), hi = std::min(e.rb2 >> 1, (S.end_y + 1) * S_);
                if (lo >= hi) continue;
                const int32_t b0 = lo / (kTileRows * S_), b1 = (hi - 1) / (kTileRows * S_);
                for (int32_t b = b0; b <= b1; b++) visit(S.fb_base + (b - S.band0), S.edge_base + k);
            }
        }
    };
    size_t n_bins = 0;
    for_bands([&](int32_t fb, int32_t) {
        cnt[(size_t)fb]++;
        n_bins++;
    });
    if (n_bins > kSmallMaxBins) {
        done = false;
        return Z2D_OK;
    }
    for (long long fb = 0; fb < n_fb; fb++)
        if (cnt[(size_t)fb] > kMaxBandEdges) {
            done = false;  // the pipeline reports it
            return Z2D_OK;
        }
    off.assign((size_t)n_fb + 1, 0);
    for (long long fb = 0; fb < n_fb; fb++) off[(size_t)fb + 1] = off[(size_t)fb] + cnt[(size_t)fb];
    bins.assign(std::max<size_t>(n_bins, 1), 0);
    for (long long fb = 0; fb < n_fb; fb++) cnt[(size_t)fb] = off[(size_t)fb];
    for_bands([&](int32_t fb, int32_t e) { bins[(size_t)cnt[(size_t)fb]++] = e; });
    // ---- band lists (k_band_lists): the job's fills touching each band, in order
    bcount.assign(std::max<long long>(n_gbands, 1), 0);
    blist.assign(std::max<long long>(n_slots, 1), make_int4(0, 0, 0, 0));
    tiles.clear();
    for (const DevJob &jb : J) {
        if (jb.band_hi < jb.band_lo) continue;
        const int32_t nf = jb.fill1 - jb.fill0;
        for (int32_t b = jb.band_lo; b <= jb.band_hi; b++) {
            const int32_t lb = b - jb.band_lo;
            if (n_jobs > 1)  // (tiles are numbered in this order)
                for (int32_t t = 0; t <= jb.tcol_hi - jb.tcol_lo; t++)
                    tiles.push_back(TileRec{(int32_t)(&jb - J.data()), lb, t, 0});
            int4 *out = blist.data() + jb.list_base + (long long)lb * nf;
            int32_t k = 0;
            for (int32_t f = jb.fill0; f < jb.fill1; f++) {
                const FillState &S = st[(size_t)f];
                if (S.active && b >= S.band0 && b <= S.band1)
                    out[k++] = make_int4(f, S.cull_x0, S.cull_x1, S.fb_base + (b - S.band0));
            }
            bcount[(size_t)(jb.gband_base + lb)] = k;
        }
    }
    // ---- the tables, laid out as the device reads them
    auto al = [](size_t v) { return (v + 15) & ~(size_t)15; };
    const size_t o_jobs = 0, o_fill = al(sizeof(DevJob) * n_jobs);
    const size_t o_st = o_fill + al(sizeof(FillCmd) * n_fills), o_rf = o_st + al(sizeof(FillState) * n_fills);
    const size_t o_edges = o_rf + al(sizeof(RasterFill) * n_fills);
    const size_t o_bins = o_edges + al(sizeof(SmallEdge) * std::max<size_t>(edges.size(), 1));
    const size_t o_off = o_bins + al(sizeof(int32_t) * bins.size());
    const size_t o_cnt = o_off + al(sizeof(int32_t) * ((size_t)n_fb + 1));
    const size_t o_list = o_cnt + al(sizeof(int32_t) * bcount.size());
    const size_t o_grad = o_list + al(sizeof(int4) * blist.size());
    const size_t o_tile = o_grad + al(sizeof(DevGradient) * grads.size());
    const size_t o_lut = o_tile + al(sizeof(TileRec) * tiles.size());
    const size_t total = o_lut + al(32 * sizeof(uint32_t) * n_fills);
    // (as the launch's parameters, or by a copy: k_raster_small)
    const bool by_param = total <= kParamBytes;
    ParamBlob blob;
    uint8_t *h;
    uintptr_t dv = 0;  // the device's tables (parameters: offsets)
    int slot = 0;
    if (by_param) {
        h = reinterpret_cast<uint8_t *>(blob.v);
    } else {
        if (c.small_params.ensure(total)) return Z2D_ERR_OUT_OF_MEMORY;
        dv = reinterpret_cast<uintptr_t>(c.small_params.ptr);
        slot = c.small_slot;
        c.small_slot ^= 1;
        HostBuf &hb = c.small_stage[slot];
        if (!c.small_done[slot]) Z2D_CUDA(cudaEventCreateWithFlags(&c.small_done[slot], cudaEventDisableTiming));
        Z2D_CUDA(cudaEventSynchronize(c.small_done[slot]));  // the slot's previous upload has been read
        if (hb.ensure(total)) return Z2D_ERR_OUT_OF_MEMORY;
        h = hb.as<uint8_t>();
    }
    memcpy(h + o_jobs, J.data(), sizeof(DevJob) * n_jobs);
    FillCmd *hf = reinterpret_cast<FillCmd *>(h + o_fill);
    memcpy(hf, fills.data(), sizeof(FillCmd) * n_fills);
    const DevGradient *dgrads = reinterpret_cast<const DevGradient *>(dv + o_grad);
    for (size_t f = 0; f < n_fills; f++)
        hf[f].src.grad = grad_of_fill[f] >= 0 ? dgrads + grad_of_fill[f] : nullptr;
    memcpy(h + o_st, st.data(), sizeof(FillState) * n_fills);
    memcpy(h + o_rf, rf.data(), sizeof(RasterFill) * n_fills);
    if (!edges.empty()) memcpy(h + o_edges, edges.data(), sizeof(SmallEdge) * edges.size());
    memcpy(h + o_bins, bins.data(), sizeof(int32_t) * bins.size());
    if (!tiles.empty()) memcpy(h + o_tile, tiles.data(), sizeof(TileRec) * tiles.size());
    memcpy(h + o_off, off.data(), sizeof(int32_t) * ((size_t)n_fb + 1));
    memcpy(h + o_cnt, bcount.data(), sizeof(int32_t) * bcount.size());
    memcpy(h + o_list, blist.data(), sizeof(int4) * blist.size());
    if (!grads.empty()) memcpy(h + o_grad, grads.data(), sizeof(DevGradient) * grads.size());
    uint32_t *lut = reinterpret_cast<uint32_t *>(h + o_lut);
    for (size_t f = 0; f < n_fills; f++) {
        if (fills[f].fast_kind != FAST_PIXEL_SRC_OVER) continue;  // (not read)
        for (int k = 0; k <= 16; k++) lut[32 * f + k] = coverage_word(fills[f], J[(size_t)fills[f].job].sfc.fmt, k);
    }
    if (!by_param) {
        Z2D_CUDA(cudaMemcpyAsync(c.small_params.ptr, h, total, cudaMemcpyHostToDevice, c.stream));
        Z2D_CUDA(cudaEventRecord(c.small_done[slot], c.stream));
    }
    if (n_tiles == 0) return Z2D_OK;
    // ---- the rasteriser, one CTA per tile
    RasterArgs A{};
    A.job0 = J[0];
    A.jobs = reinterpret_cast<const DevJob *>(dv + o_jobs);
    A.fills = reinterpret_cast<const FillCmd *>(dv + o_fill);
    A.st = reinterpret_cast<const FillState *>(dv + o_st);
    A.edges = reinterpret_cast<const SmallEdge *>(dv + o_edges);
    A.bins = reinterpret_cast<const int32_t *>(dv + o_bins);
    A.bin_off = reinterpret_cast<const int32_t *>(dv + o_off);
    A.band_count = reinterpret_cast<const int32_t *>(dv + o_cnt);
    A.band_fills = reinterpret_cast<const int4 *>(dv + o_list);
    A.rfills = reinterpret_cast<const RasterFill *>(dv + o_rf);
    A.tiles = reinterpret_cast<const TileRec *>(dv + o_tile);
    A.luts = reinterpret_cast<const uint32_t *>(dv + o_lut);
    A.masks = nullptr;
    A.queue = nullptr;
    A.n_items = (unsigned long long)n_tiles;
    A.order = nullptr;
    A.one_per_tile = 1;
    {
        const int rs = c.await_surface();
        if (rs) return rs;
    }
    const int mode = raster_mode(fills.data(), n_fills, false);
    cudaEvent_t t0 = c.timer_begin(c.t_raster);
    const int rc = by_param ? raster_launch_small(c, n_jobs > 1, mode, A, blob, (int32_t)(total / sizeof(uint4)),
                                                  (int32_t)n_fills, (unsigned)n_tiles)
                            : raster_launch(c, RasterVariant{n_jobs > 1, true, kBinSmall, mode}, A, (unsigned)n_tiles);
    if (rc) return rc;
    c.timer_end(c.t_raster, t0);
    return Z2D_OK;
}

}  // namespace z2dg
