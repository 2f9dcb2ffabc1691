// stroke_gpu.cu -- the stroke polygon of painter.stroke, tessellated on the
// device (solid strokes; the stages are listed in stroke_gpu.cuh).
//
// The polygon is the one stroke_plotter.Plotter builds
// (src/internal/tess/stroke_plotter.zig:77-403): per subpath, an outer
// contour that joins append to and an inner contour that joins prepend to;
// closed subpaths give both as separate contours, open ones one contour
// [start cap, outer, end cap, inner].  Every join and cap writes its points
// straight into their final contour positions, found by prefix sums over
// the elements' point counts, so the edges (consecutive contour points) are
// the reference's in its order.  Geometry is stroke_geom.h, shared with the
// host builder; the curve subdivision is spline.cuh, shared with fills.
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include "edges.cuh"
#include "spline.cuh"
#include "stroke_geom.h"
#include "stroke_gpu.cuh"
#include "z2d_internal.h"

namespace z2dg {

using sg::Face;
using sg::PenVertex;
using sg::Pt;
using sg::Slope;
using sg::Tf;

namespace {

enum : int32_t { SK_NONE = 0, SK_OPEN = 1, SK_CLOSED = 2, SK_SINGLE = 3, SK_DOT = 4 };

// per subpath, after deduplication
struct SubState {
    int32_t q0, n;   // kept points [q0, q0 + n)
    int32_t kind;    // SK_*
    int32_t pcw;     // direction of the first join (the plotter's `clockwise`)
};
// counts or offsets of outer (a) and inner (b) contour points
struct Count2 {
    long long a, b;
};
struct Sum2 {
    __host__ __device__ __forceinline__ Count2 operator()(const Count2 &x, const Count2 &y) const {
        return Count2{x.a + y.a, x.b + y.b};
    }
};
// per subpath: its outer points [ra, ra + sa) and inner points
// [rb, rb + sb), the fill that draws it and what turns a point's position
// into its edge's index within that fill
struct Region {
    int32_t ra, sa, rb, sb;
    int32_t fill, edge_a, edge_b, closed;
};
// The points of an element that is a join, found when it is counted: the
// outer side's first and last point with a run of pen vertices around the
// join's point between them, the inner side's first and last point with the
// join's point between them.
enum : int32_t { EL_JOIN = 1, EL_SWITCHED = 2, EL_CW = 4, EL_TWO_OUTER = 8, EL_THREE_INNER = 16 };
struct Elem {
    Pt o1, o2, i1, i2;
    int32_t start, cnt;  // pen vertices
    int32_t flags, _pad;
};

// device pointers of one run
struct State {
    long long *raw_cnt, *raw_off;   // (n_local << g) + 1
    int g;                          // log2 of the lanes that share a node
    PenVertex *pen;                 // n_pen
    SubState *sub;                  // n_subs
    Region *region;                 // n_subs
    long long *totals;              // outer, inner totals (read back)
    // sized by the raw point count R
    double2 *raw_pt;
    int32_t *raw_sub;
    uint8_t *raw_mode;
    int32_t *keep, *kept_off;       // R + 1
    double2 *q_pt;
    int32_t *q_sub;
    uint8_t *q_mode;
    Elem *elem;                     // R, or null: not kept
    Count2 *cnt, *off;              // R + 1
    // contour points, and each one's subpath
    double2 *pa, *pb;
    int32_t *a_sub, *b_sub;
};

__device__ __forceinline__ Tf tf_of(const StrokeDev &s) {
    return Tf{s.ctm[0], s.ctm[1], s.ctm[2], s.ctm[3], s.ctm[4], s.ctm[5]};
}
__device__ __forceinline__ Pt node_end(const z2d_node &nd) {
    return nd.tag == Z2D_CURVE_TO ? Pt{nd.p[4], nd.p[5]} : Pt{nd.p[0], nd.p[1]};
}

// ----------------------------------------------------------------- pens
// Pen.init (Pen.zig:25-88) from the host's cos/sin table: vertex points
// through the CTM, then the slopes to either neighbour.
// A block per stroke, a thread per vertex (each evaluates its neighbours'
// points again, which gives the same bits).
__global__ void ks_pen(const StrokeDev *__restrict__ strokes, const double *__restrict__ trig,
                       PenVertex *__restrict__ pen) {
    const StrokeDev &S = strokes[blockIdx.x];
    const int32_t n = S.pen_n;
    const Tf ctm = tf_of(S);
    const double radius = S.thickness / 2;
    PenVertex *v = pen + S.pen_off;
    const double *t = trig + 2 * (size_t)S.pen_tab;
    auto point = [&](int32_t i) {
        double dx = radius * t[2 * i], dy = radius * t[2 * i + 1];
        sg::user_to_device_distance(ctm, dx, dy);
        return Pt{dx, dy};
    };
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const int32_t next = (i >= n - 1) ? 0 : i + 1;
        const int32_t prev = max(0, i == 0 ? n - 1 : i - 1);
        PenVertex p;
        p.point = point(i);
        p.slope_cw = sg::slope(point(prev), p.point);
        p.slope_ccw = sg::slope(p.point, point(next));
        v[i] = p;
    }
}

// ------------------------------------------------------------ raw points
// A warp per subpath.
__global__ void ks_local_sub(const SubpathDev *__restrict__ subs, int32_t n_subs, int32_t *__restrict__ local_sub) {
    const long long sp = warp_number(blockIdx.x, blockDim.x, threadIdx.x);
    if (sp >= n_subs) return;
    const int32_t l0 = subs[sp].local0, n = subs[sp].n_nodes;
    for (int32_t j = threadIdx.x & 31; j < n; j += 32) local_sub[l0 + j] = (int32_t)sp;
}

// The points one node hands to the plotter: move_to its point, line_to its
// end, curve_to Spline.decompose's lineTo calls (stroke_plotter.zig:126-150).
// 2^g neighbouring lanes share a node: a curve's subdivision tree as in
// lane_subtree (one thread walking a curve of 500 leaves took 0.68 ms, most
// of a single stroke's call; 32 lanes take 0.03), the other nodes' point is
// lane 0's.  emit(x, y) is called for the lane's points in order; false if
// the subdivision gave up.
template <class Emit>
__device__ __forceinline__ bool node_points(const z2d_node *__restrict__ nodes, const SubpathDev &S, int32_t n, int g,
                                           int j, double tol, Emit &&emit) {
    const z2d_node nd = nodes[S.node0 + n];
    if (n == 0 || nd.tag == Z2D_LINE_TO) {
        if (j == 0) emit(nd.p[0], nd.p[1]);
        return true;
    }
    const Pt a = node_end(nodes[S.node0 + n - 1]);
    const double *p = nd.p;
    const int last = (1 << g) - 1;
    bool ok = true;
    if (!(pt_eq(a.x, a.y, p[0], p[1]) && pt_eq(p[2], p[3], p[4], p[5]))) {  // Spline.zig:39-42
        Knots k{a.x, a.y, p[0], p[1], p[2], p[3], p[4], p[5]};
        const Tol t = make_tol(tol, k);
        bool is_leaf;
        int open;
        if (lane_subtree(k, g, j, t, is_leaf, open))
            ok = walk_leaves(k, is_leaf, open, t, [&](const Knots &q) {
                if (!pt_eq(q.ax, q.ay, a.x, a.y)) emit(q.ax, q.ay);
            });
    }
    if (j == last) emit(p[4], p[5]);
    return ok;
}

// Points per (node, lane), node after node.
__global__ void ks_raw_count(const z2d_node *__restrict__ nodes, const SubpathDev *__restrict__ subs,
                             const int32_t *__restrict__ local_sub, const StrokeDev *__restrict__ strokes,
                             long long n_local, int g, long long *__restrict__ raw_cnt, int32_t *__restrict__ status) {
    const long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = at >> g;
    if (i >= n_local) {
        if (at == lane_slot(n_local, g)) raw_cnt[at] = 0;
        return;
    }
    const SubpathDev S = subs[local_sub[i]];
    int32_t cnt = 0;
    if (!node_points(nodes, S, (int32_t)(i - S.local0), g, (int)(at & ((1 << g) - 1)), strokes[S.stroke].tolerance,
                     [&](double, double) { cnt++; }))
        atomicExch(status, Z2D_ERR_INVALID_STATE);
    raw_cnt[at] = cnt;
}

__global__ void ks_raw_emit(const z2d_node *__restrict__ nodes, const SubpathDev *__restrict__ subs,
                            const int32_t *__restrict__ local_sub, const StrokeDev *__restrict__ strokes,
                            long long n_local, int g, const long long *__restrict__ raw_off,
                            double2 *__restrict__ raw_pt, int32_t *__restrict__ raw_sub,
                            uint8_t *__restrict__ raw_mode) {
    const long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = at >> g;
    if (i >= n_local) return;
    long long r = raw_off[at];
    const long long r_end = raw_off[at + 1];
    if (r == r_end) return;
    const int32_t sp = local_sub[i];
    const SubpathDev S = subs[sp];
    const int32_t n = (int32_t)(i - S.local0);
    const StrokeDev &T = strokes[S.stroke];
    const uint8_t mode =
        (n > 0 && nodes[S.node0 + n].tag == Z2D_CURVE_TO) ? (uint8_t)Z2D_JOIN_ROUND : (uint8_t)T.join;
    node_points(nodes, S, n, g, (int)(at & ((1 << g) - 1)), T.tolerance, [&](double x, double y) {
        if (r < r_end) {
            raw_pt[r] = make_double2(x, y);
            raw_sub[r] = sp;
            raw_mode[r] = mode;
        }
        r++;
    });
}

// Whether the plotter keeps raw point r: the degenerate-node check against
// the point before it of the same subpath.
__global__ void ks_keep(const double2 *__restrict__ raw_pt, const int32_t *__restrict__ raw_sub, long long n_raw,
                        int32_t *__restrict__ keep) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r > n_raw) return;
    int32_t k = 0;
    if (r < n_raw) {
        k = 1;
        if (r > 0 && raw_sub[r] == raw_sub[r - 1]) {
            const double2 a = raw_pt[r - 1], b = raw_pt[r];
            k = pt_eq(a.x, a.y, b.x, b.y) ? 0 : 1;
        }
    }
    keep[r] = k;
}

__global__ void ks_compact(const double2 *__restrict__ raw_pt, const int32_t *__restrict__ raw_sub,
                           const uint8_t *__restrict__ raw_mode, const int32_t *__restrict__ keep,
                           const int32_t *__restrict__ kept_off, long long n_raw, double2 *__restrict__ q_pt,
                           int32_t *__restrict__ q_sub, uint8_t *__restrict__ q_mode) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_raw || !keep[r]) return;
    const int32_t q = kept_off[r];
    q_pt[q] = raw_pt[r];
    q_sub[q] = raw_sub[r];
    q_mode[q] = raw_mode[r];
}

// close_path / finish of the plotter (stroke_plotter.zig:152-230): what a
// subpath of n kept points draws.
__global__ void ks_sub_setup(const SubpathDev *__restrict__ subs, int32_t n_subs, const StrokeDev *__restrict__ strokes,
                             int g, const long long *__restrict__ raw_off, const int32_t *__restrict__ kept_off,
                             const double2 *__restrict__ q_pt, SubState *__restrict__ sub) {
    const int32_t sp = blockIdx.x * blockDim.x + threadIdx.x;
    if (sp >= n_subs) return;
    const SubpathDev S = subs[sp];
    const long long r0 = raw_off[lane_slot(S.local0, g)], r1 = raw_off[lane_slot((long long)S.local0 + S.n_nodes, g)];
    SubState st;
    st.q0 = kept_off[r0];
    st.n = kept_off[r1] - st.q0;
    if (st.n >= 3) st.kind = S.closed ? SK_CLOSED : SK_OPEN;
    else if (st.n == 2) st.kind = SK_SINGLE;
    else if (st.n == 1 && S.closed && strokes[S.stroke].cap == Z2D_CAP_ROUND) st.kind = SK_DOT;
    else st.kind = SK_NONE;
    st.pcw = 1;
    if (st.n >= 3) {
        const double2 a = q_pt[st.q0], b = q_pt[st.q0 + 1], c = q_pt[st.q0 + 2];
        const Slope in = sg::normalized(Slope{b.x - a.x, b.y - a.y});
        const Slope out = sg::normalized(Slope{c.x - b.x, c.y - b.y});
        st.pcw = sg::compare(in, out) < 0 ? 1 : 0;
    }
    sub[sp] = st;
}

// ------------------------------------------------------------- elements
// Receives an element's points: A = appended to the outer contour, B =
// prepended to the inner one (in plot order).  Counting only when !EMIT.
template <bool EMIT>
struct Out {
    long long na = 0, nb = 0;
    double2 *pa = nullptr;      // A point k goes to pa[k]
    double2 *pb_end = nullptr;  // B point k goes to pb_end[-1 - k]
    double scale = 1;
    __device__ __forceinline__ void A(Pt p) {
        if (EMIT) pa[na] = make_double2(p.x * scale, p.y * scale);
        na++;
    }
    __device__ __forceinline__ void B(Pt p) {
        if (EMIT) pb_end[-1 - nb] = make_double2(p.x * scale, p.y * scale);
        nb++;
    }
    // pen vertices around c, to A or B
    __device__ __forceinline__ void pen(bool to_a, Pt c, const PenVertex *v, int32_t len, int32_t start,
                                        int32_t cnt, bool cw) {
        if (!EMIT) {
            (to_a ? na : nb) += cnt;
            return;
        }
        for (int32_t k = 0; k < cnt; k++) {
            const Pt p = v[sg::pen_step(start, k, len, cw)].point;
            const Pt q{c.x + p.x, c.y + p.y};
            if (to_a) A(q);
            else B(q);
        }
    }
};

// join (stroke_plotter.zig:405-545) at p1 between p0->p1 and p1->p2, with
// the subpath's first-join direction pcw: where outer and inner trade places
// (EL_SWITCHED) the outer points go to the inner contour.
__device__ __forceinline__ Elem join(const StrokeDev &T, const Tf &ctm, const PenVertex *pen, int mode, Pt p0, Pt p1,
                                     Pt p2, bool pcw) {
    Elem e;
    e.start = e.cnt = 0;
    e.flags = 0;
    if (sg::eq(p0, p1) || sg::eq(p1, p2)) return e;
    const Face in = sg::face_init(p0, p1, T.thickness, ctm);
    const Face out = sg::face_init(p1, p2, T.thickness, ctm);
    const int cmp = sg::compare(in.dev_slope, out.dev_slope);
    const bool jcw = cmp < 0;
    e.flags = EL_JOIN | (jcw != pcw ? EL_SWITCHED : 0) | (jcw ? EL_CW : 0);
    e.o1 = jcw ? in.p1_ccw : in.p1_cw;
    e.i1 = jcw ? in.p1_cw : in.p1_ccw;
    if (cmp == 0) return e;
    e.flags |= EL_THREE_INNER;
    e.i2 = jcw ? out.p0_cw : out.p0_ccw;
    if (mode == Z2D_JOIN_MITER && sg::compare_for_miter_limit(in.dev_slope, out.dev_slope, T.miter_limit)) {
        e.o1 = sg::intersect(in, out, jcw);
        return e;
    }
    e.flags |= EL_TWO_OUTER;
    e.o2 = jcw ? out.p0_ccw : out.p0_cw;
    if (mode != Z2D_JOIN_MITER && mode != Z2D_JOIN_BEVEL)
        e.cnt = sg::pen_range(pen, T.pen_n, in.dev_slope, out.dev_slope, jcw, e.start);
    return e;
}
__device__ __forceinline__ Count2 join_count(const Elem &e) {
    if (!(e.flags & EL_JOIN)) return Count2{0, 0};
    const long long o = 1 + e.cnt + ((e.flags & EL_TWO_OUTER) ? 1 : 0), i = (e.flags & EL_THREE_INNER) ? 3 : 1;
    return (e.flags & EL_SWITCHED) ? Count2{i, o} : Count2{o, i};
}

// Face.cap (Face.zig:156-246), to A
template <class O>
__device__ __forceinline__ void cap(O &o, const StrokeDev &T, const Tf &ctm, const PenVertex *pen, const Face &f,
                                    bool cw) {
    if (T.cap == Z2D_CAP_BUTT) {
        o.A(cw ? f.p1_ccw : f.p1_cw);
        o.A(cw ? f.p1_cw : f.p1_ccw);
    } else if (T.cap == Z2D_CAP_SQUARE) {
        double ox = f.user_slope.dx * f.half_width, oy = f.user_slope.dy * f.half_width;
        sg::user_to_device_distance(ctm, ox, oy);
        const Pt a = cw ? f.p1_ccw : f.p1_cw, b = cw ? f.p1_cw : f.p1_ccw;
        o.A(a);
        o.A(Pt{a.x + ox, a.y + oy});
        o.A(Pt{b.x + ox, b.y + oy});
        o.A(b);
    } else {
        o.A(cw ? f.p1_ccw : f.p1_cw);
        int32_t start;
        const int32_t cnt =
            sg::pen_range(pen, T.pen_n, f.dev_slope, Slope{-f.dev_slope.dx, -f.dev_slope.dy}, cw, start);
        o.pen(true, f.p1, pen, T.pen_n, start, cnt, cw);
        o.A(cw ? f.p1_cw : f.p1_ccw);
    }
}

// What element k of a subpath contributes (see stroke_gpu.cuh): caps and dots
// go to `o`, a join is returned (flags 0: none).
template <class O>
__device__ __forceinline__ Elem element(O &o, const StrokeDev &T, const PenVertex *pen, const SubState &st,
                                        const double2 *__restrict__ q_pt, const uint8_t *__restrict__ q_mode,
                                        int32_t k) {
    const int32_t n = st.n;
    auto P = [&](int32_t i) {
        const double2 v = q_pt[st.q0 + i];
        return Pt{v.x, v.y};
    };
    const Tf ctm = tf_of(T);
    const bool pcw = st.pcw != 0;
    // Every case below draws at most two caps or one join; they are
    // gathered into one cap call and one join call, so that the kernel
    // holds a single copy of each.
    Elem none;
    none.flags = none.cnt = 0;
    int n_caps = 0, jmode = -1;
    Pt c0{}, c1{}, j0{}, j1{}, j2{};
    bool ccw = pcw;
    switch (st.kind) {
        case SK_DOT:  // plot_dot of stroke_plotter (round caps only)
            if (k == 0) {
                const Pt c = P(0);
                for (int32_t i = 0; i < T.pen_n; i++) o.A(Pt{c.x + pen[i].point.x, c.y + pen[i].point.y});
            }
            return none;
        case SK_SINGLE:  // plotSingle (stroke_plotter.zig:232-279): caps of b->a, then a->b
            if (k != 0) return none;
            n_caps = 2;
            c0 = P(1);
            c1 = P(0);
            ccw = true;
            break;
        case SK_OPEN:  // plotOpenJoined (stroke_plotter.zig:281-363)
            if (k == 0) {
                n_caps = 1;
                c0 = P(1);
                c1 = P(0);
            } else if (k == n - 1) {
                n_caps = 1;
                c0 = P(n - 2);
                c1 = P(n - 1);
            } else {
                jmode = q_mode[st.q0 + k + 1];
                j0 = P(k - 1);
                j1 = P(k);
                j2 = P(k + 1);
            }
            break;
        case SK_CLOSED: {  // plotClosedJoined (stroke_plotter.zig:365-403)
            const bool back_to_start = sg::eq(P(n - 1), P(0));
            if (k >= 1 && k <= n - 2) {
                jmode = q_mode[st.q0 + k + 1];
                j0 = P(k - 1);
                j1 = P(k);
                j2 = P(k + 1);
            } else if (k == n - 1) {
                if (back_to_start) return none;
                jmode = T.join;
                j0 = P(n - 2);
                j1 = P(n - 1);
                j2 = P(0);
            } else {
                jmode = T.join;
                j0 = back_to_start ? P(n - 2) : P(n - 1);
                j1 = P(0);
                j2 = P(1);
            }
            break;
        }
        default: return none;
    }
#pragma unroll 1
    for (int i = 0; i < n_caps; i++) {
        cap(o, T, ctm, pen, sg::face_init(c0, c1, T.thickness, ctm), ccw);
        const Pt t = c0;  // the second cap of plotSingle runs the other way
        c0 = c1;
        c1 = t;
    }
    if (jmode >= 0) return join(T, ctm, pen, jmode, j0, j1, j2, pcw);
    return none;
}

__global__ void ks_elem_count(const SubpathDev *__restrict__ subs, const StrokeDev *__restrict__ strokes,
                              const PenVertex *__restrict__ pen, const SubState *__restrict__ sub,
                              const double2 *__restrict__ q_pt, const int32_t *__restrict__ q_sub,
                              const uint8_t *__restrict__ q_mode, const int32_t *__restrict__ kept_off,
                              long long n_raw, Elem *__restrict__ elem, Count2 *__restrict__ cnt) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q > n_raw) return;
    const long long n_kept = kept_off[n_raw];
    if (q >= n_kept) {
        cnt[q] = Count2{0, 0};
        return;
    }
    const int32_t sp = q_sub[q];
    const SubState st = sub[sp];
    const StrokeDev T = strokes[subs[sp].stroke];
    Out<false> o;
    const Elem e = element(o, T, pen + T.pen_off, st, q_pt, q_mode, (int32_t)(q - st.q0));
    if (elem) elem[q] = e;
    cnt[q] = (e.flags & EL_JOIN) ? join_count(e) : Count2{o.na, o.nb};
}

// Per stroke its edge count, per subpath its regions of the contour arrays.
__global__ void ks_stroke_tot(const StrokeDev *__restrict__ strokes, int32_t n_strokes,
                              const SubpathDev *__restrict__ subs, int32_t n_subs, const SubState *__restrict__ sub,
                              const Count2 *__restrict__ off, long long n_raw, Region *__restrict__ region,
                              int32_t *__restrict__ stroke_edges, long long *__restrict__ totals) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        totals[0] = off[n_raw].a;
        totals[1] = off[n_raw].b;
    }
    // the stroke's points: [first, last) of the kept points
    auto ends = [&](const StrokeDev &S, Count2 &c0, Count2 &c1) {
        const SubState last = sub[S.sub0 + S.n_sub - 1];
        c0 = off[sub[S.sub0].q0];
        c1 = off[last.q0 + last.n];
    };
    if (i < n_strokes) {
        const StrokeDev &S = strokes[i];
        Count2 c0{0, 0}, c1{0, 0};
        if (S.n_sub > 0) ends(S, c0, c1);
        const long long e = (c1.a - c0.a) + (c1.b - c0.b);
        stroke_edges[i] = e > 0x7FFFFFFFll ? -1 : (int32_t)e;
    }
    if (i < n_subs) {
        const StrokeDev &S = strokes[subs[i].stroke];
        const SubState st = sub[i];
        Count2 c0, c1;
        ends(S, c0, c1);
        const Count2 r0 = off[st.q0], r1 = off[st.q0 + st.n];
        Region R;
        R.ra = (int32_t)r0.a;
        R.sa = (int32_t)(r1.a - r0.a);
        R.rb = (int32_t)r0.b;
        R.sb = (int32_t)(r1.b - r0.b);
        R.fill = S.fill;
        R.edge_a = (int32_t)-c0.a;
        R.edge_b = (int32_t)(c1.a - c0.a - c0.b);
        R.closed = st.kind == SK_CLOSED ? 1 : 0;
        region[i] = R;
    }
}

// Writes every element's points to their contour positions: outer points in
// element order, inner points in reverse (B points are prepended); a closed
// subpath's closing joins come last: elements 1..n-1, then 0.  KEPT: the joins
// are in `elem`; without (scarce), they are found a second time.
template <bool KEPT>
__global__ void ks_elem_emit(const SubpathDev *__restrict__ subs, const StrokeDev *__restrict__ strokes,
                             const PenVertex *__restrict__ pen, const SubState *__restrict__ sub,
                             const Region *__restrict__ region, const double2 *__restrict__ q_pt,
                             const int32_t *__restrict__ q_sub, const uint8_t *__restrict__ q_mode,
                             const int32_t *__restrict__ kept_off, long long n_raw, const Elem *__restrict__ elem,
                             const Count2 *__restrict__ off, double2 *__restrict__ pa, double2 *__restrict__ pb,
                             int32_t *__restrict__ a_sub, int32_t *__restrict__ b_sub) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= kept_off[n_raw]) return;
    const int32_t sp = q_sub[q];
    const SubState st = sub[sp];
    const Region R = region[sp];
    const int32_t k = (int32_t)(q - st.q0);
    const StrokeDev &T = strokes[subs[sp].stroke];
    const Count2 at = off[q], next = off[q + 1];
    const long long na = next.a - at.a, nb = next.b - at.b;
    long long pos_a = at.a, t_b = at.b - R.rb;
    if (st.kind == SK_CLOSED) {
        const Count2 o1 = off[st.q0 + 1];
        const long long a0 = o1.a - R.ra, b0 = o1.b - R.rb;
        pos_a = k >= 1 ? at.a - a0 : R.ra + R.sa - a0;
        t_b = k >= 1 ? at.b - R.rb - b0 : R.sb - b0;
    }
    const long long end_b = (long long)R.rb + R.sb - t_b;
    for (long long i = 0; i < na; i++) a_sub[pos_a + i] = sp;
    for (long long i = 0; i < nb; i++) b_sub[end_b - 1 - i] = sp;
    Elem e;
    if constexpr (KEPT) e = elem[q];
    Out<true> o;
    o.pa = pa + pos_a;
    o.pb_end = pb + end_b;
    o.scale = T.scale;
    if (!KEPT || !(e.flags & EL_JOIN)) {  // caps and dots
        if (na + nb == 0) return;
        const StrokeDev S = T;
        e = element(o, S, pen + S.pen_off, st, q_pt, q_mode, k);
        if (!(e.flags & EL_JOIN)) return;
    }
    const bool sw = (e.flags & EL_SWITCHED) != 0;
    auto outer = [&](Pt p) {
        if (sw) o.B(p);
        else o.A(p);
    };
    auto inner = [&](Pt p) {
        if (sw) o.A(p);
        else o.B(p);
    };
    const double2 c = q_pt[q];
    const Pt p1{c.x, c.y};
    outer(e.o1);
    if (e.cnt > 0) o.pen(!sw, p1, pen + T.pen_off, T.pen_n, e.start, e.cnt, (e.flags & EL_CW) != 0);
    if (e.flags & EL_TWO_OUTER) outer(e.o2);
    inner(e.i1);
    if (e.flags & EL_THREE_INNER) {
        inner(p1);
        inner(e.i2);
    }
}

// Polygon.addEdgesFromContour: every contour point to the next one (the
// last back to the first), a thread per point.  An open subpath's contour is
// its outer region followed by its inner region.
__global__ void ks_edges(const Region *__restrict__ region, const double2 *__restrict__ pa,
                         const double2 *__restrict__ pb, const int32_t *__restrict__ a_sub,
                         const int32_t *__restrict__ b_sub, long long n_a, long long n_b,
                         const FillCmd *__restrict__ fills, FillState *__restrict__ st_fill,
                         DEdge *__restrict__ edges) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int32_t f = -1;
    double et = 0, eb = 0, el = 0, er = 0;
    bool any = false;
    if (t < n_a + n_b) {
        const bool outer = t < n_a;
        const int32_t pos = (int32_t)(outer ? t : t - n_a);
        const Region R = region[outer ? a_sub[pos] : b_sub[pos]];
        f = R.fill;
        double2 a, b;
        if (outer) {
            a = pa[pos];
            b = pos + 1 < R.ra + R.sa ? pa[pos + 1] : !R.closed && R.sb > 0 ? pb[R.rb] : pa[R.ra];
        } else {
            a = pb[pos];
            b = pos + 1 < R.rb + R.sb ? pb[pos + 1] : !R.closed ? pa[R.ra] : pb[R.rb];
        }
        DEdge *out = edges + st_fill[f].edge_base + (pos + (outer ? R.edge_a : R.edge_b));
        add_edge(fills[f], out, a.x, a.y, b.x, b.y, et, eb, el, er, any);
    }
    merge_extents(st_fill, f, any, et, eb, el, er);
}

// Host-built polygons: each warp takes 32 consecutive points; lane k
// finds its contour among the (at most 32) contours the chunk touches.
__global__ void kp_edges(PolyRun run, const FillCmd *__restrict__ fills, FillState *__restrict__ st_fill,
                         DEdge *__restrict__ edges) {
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const long long n_pts = run.n_points;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long base = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; base < n_pts;
         base += warps * 32) {
        // the contour holding `base`: the last one starting at or before it
        int32_t c0 = 0;
        if (lane == 0) {
            int32_t lo = 0, hi = run.n_contours - 1;
            while (lo < hi) {
                const int32_t mid = (lo + hi + 1) >> 1;
                if (run.start[mid] <= base) lo = mid;
                else hi = mid - 1;
            }
            c0 = lo;
        }
        c0 = __shfl_sync(all, c0, 0);
        const int32_t ck = c0 + lane;
        const long long end_k = ck < run.n_contours ? run.start[ck] + run.n[ck] : 0x7FFFFFFFFFFFFFFFll;
        const long long pt = base + lane;
        int32_t my = c0;
#pragma unroll 8
        for (int k = 0; k < 32; k++) my += __shfl_sync(all, end_k, k) <= pt ? 1 : 0;
        int32_t f = -1;
        double et = 0, eb = 0, el = 0, er = 0;
        bool any = false;
        if (pt < n_pts) {
            const long long s0 = run.start[my];
            const int32_t n = run.n[my];
            f = run.fill[my];
            const long long nx = pt + 1 == s0 + n ? s0 : pt + 1;
            const double2 a = run.pts[pt], b = run.pts[nx];
            add_edge(fills[f], edges + st_fill[f].edge_base + run.edge_off[my] + (pt - s0), a.x, a.y, b.x, b.y, et, eb,
                     el, er, any);
        }
        merge_extents(st_fill, f, any, et, eb, el, er);
    }
}

inline unsigned blocks_for(long long n, int threads) { return (unsigned)((n + threads - 1) / threads); }

// carves aligned sub-buffers out of one allocation
struct Carve {
    size_t off = 0;
    template <class T>
    size_t take(long long count) {
        const size_t at = off;
        off = (off + sizeof(T) * (size_t)count + 255) & ~(size_t)255;
        return at;
    }
};

// Whether scratch that a call can do without would leave the device too little
// for the rest of it: the rest of a stroke takes three to six times as much.
bool scarce(size_t bytes) {
    if (bytes < ((size_t)1 << 30)) return false;
    size_t free_bytes = 0, total = 0;
    if (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess) return false;
    return bytes > free_bytes / 8;
}

}  // namespace

int poly_emit(Ctx &c, const PolyRun &run, const FillCmd *d_fills, FillState *d_st, DEdge *d_edges) {
    if (run.n_points == 0 || run.n_contours == 0) return Z2D_OK;
    constexpr int T = 128;
    const unsigned blocks = (unsigned)std::min<long long>(blocks_for((run.n_points + 31) / 32, T / 32),
                                                          (long long)c.sm_count * 32);
    cudaEvent_t ts = c.timer_begin(c.t_stroke);
    kp_edges<<<blocks, T, 0, c.stream>>>(run, d_fills, d_st, d_edges);
    c.timer_end(c.t_stroke, ts);
    c.launches += 1;
    return Z2D_OK;
}

const long long *stroke_totals_dev(const StrokeRun &run) {
    return reinterpret_cast<const State *>(run.state)->totals;
}

int stroke_count(Ctx &c, StrokeRun &run, int32_t *d_status) {
    if (run.n_strokes == 0) return Z2D_OK;
    static thread_local State st;  // device pointers of this thread's current run
    st = State{};
    run.state = &st;
    constexpr int T = 128;
    // ---- buffers known before counting
    // A warp per node while the device has room for all of them, else 8 lanes;
    // one where the lanes' counts are scarce memory.
    Carve ca;
    long long n_lanes = 0;
    size_t o_cnt, o_off, o_lsub, o_pen, o_sub, o_reg, o_edges, o_totals;
    auto carve = [&](int g) {
        ca = Carve{};
        st.g = g;
        n_lanes = lane_slot(run.n_local, g);
        o_cnt = ca.take<long long>(n_lanes + 1), o_off = ca.take<long long>(n_lanes + 1);
        o_lsub = ca.take<int32_t>(run.n_local + 1), o_pen = ca.take<PenVertex>(run.n_pen + 1);
        o_sub = ca.take<SubState>(run.n_subs + 1), o_reg = ca.take<Region>(run.n_subs + 1);
        o_edges = ca.take<int32_t>(run.n_strokes + 1), o_totals = ca.take<long long>(2);
    };
    carve(run.n_local * 32 <= (long long)c.sm_count * 2048 ? 5 : 3);
    if (c.stroke_a.cap < ca.off && (scarce(2 * sizeof(long long) * (size_t)n_lanes) || c.stroke_a.ensure(ca.off)))
        carve(0);
    if (c.stroke_a.ensure(ca.off)) return Z2D_ERR_OUT_OF_MEMORY;
    uint8_t *A = c.stroke_a.as<uint8_t>();
    st.raw_cnt = reinterpret_cast<long long *>(A + o_cnt);
    st.raw_off = reinterpret_cast<long long *>(A + o_off);
    int32_t *local_sub = reinterpret_cast<int32_t *>(A + o_lsub);
    st.pen = reinterpret_cast<PenVertex *>(A + o_pen);
    st.sub = reinterpret_cast<SubState *>(A + o_sub);
    st.region = reinterpret_cast<Region *>(A + o_reg);
    run.stroke_edges = reinterpret_cast<int32_t *>(A + o_edges);
    st.totals = reinterpret_cast<long long *>(A + o_totals);

    cudaEvent_t ts = c.timer_begin(c.t_stroke);
    ks_pen<<<(unsigned)run.n_strokes, 64, 0, c.stream>>>(run.strokes, run.trig, st.pen);
    ks_local_sub<<<blocks_for(32ll * run.n_subs, T), T, 0, c.stream>>>(run.subs, run.n_subs, local_sub);
    ks_raw_count<<<blocks_for(n_lanes + 1, T), T, 0, c.stream>>>(run.nodes, run.subs, local_sub, run.strokes,
                                                                  run.n_local, st.g, st.raw_cnt, d_status);
    size_t tmp = 0;
    Z2D_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, st.raw_cnt, st.raw_off, n_lanes + 1, c.stream));
    if (c.scan_tmp.ensure(tmp + 16)) return Z2D_ERR_OUT_OF_MEMORY;
    Z2D_CUDA(cub::DeviceScan::ExclusiveSum(c.scan_tmp.ptr, tmp, st.raw_cnt, st.raw_off, n_lanes + 1, c.stream));
    c.launches += 4;
    long long *rb = nullptr;
    if (c.readback.ensure(64)) return Z2D_ERR_OUT_OF_MEMORY;
    rb = c.readback.as<long long>();
    Z2D_CUDA(cudaMemcpyAsync(rb, st.raw_off + n_lanes, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
    Z2D_CUDA(cudaStreamSynchronize(c.stream));
    const long long R = rb[0];
    if (R < 0 || R >= 0x7FFFFFFFll) {
        set_error("batch too large: more than 2^31 stroke points");
        return Z2D_ERR_INVALID_ARGUMENT;
    }
    run.raw = R;
    // ---- buffers sized by the point count
    Carve cb;
    const size_t o_rpt = cb.take<double2>(R + 1), o_rsub = cb.take<int32_t>(R + 1), o_rmode = cb.take<uint8_t>(R + 1);
    const size_t o_keep = cb.take<int32_t>(R + 1), o_kept = cb.take<int32_t>(R + 1);
    const size_t o_qpt = cb.take<double2>(R + 1), o_qsub = cb.take<int32_t>(R + 1), o_qmode = cb.take<uint8_t>(R + 1);
    const size_t o_c = cb.take<Count2>(R + 1), o_o = cb.take<Count2>(R + 1);
    // the joins are kept where the device has room for them (a stroke of 500
    // leaves 449 us without, with them and an edge per contour point 335)
    const size_t without = cb.off, o_el = cb.take<Elem>(R + 1);
    bool kept = c.stroke_b.cap >= cb.off || !scarce(cb.off - without);
    if (kept && c.stroke_b.ensure(cb.off)) kept = false;
    if (!kept && c.stroke_b.ensure(without)) return Z2D_ERR_OUT_OF_MEMORY;
    uint8_t *B = c.stroke_b.as<uint8_t>();
    st.raw_pt = reinterpret_cast<double2 *>(B + o_rpt);
    st.raw_sub = reinterpret_cast<int32_t *>(B + o_rsub);
    st.raw_mode = B + o_rmode;
    st.keep = reinterpret_cast<int32_t *>(B + o_keep);
    st.kept_off = reinterpret_cast<int32_t *>(B + o_kept);
    st.q_pt = reinterpret_cast<double2 *>(B + o_qpt);
    st.q_sub = reinterpret_cast<int32_t *>(B + o_qsub);
    st.q_mode = B + o_qmode;
    st.elem = kept ? reinterpret_cast<Elem *>(B + o_el) : nullptr;
    st.cnt = reinterpret_cast<Count2 *>(B + o_c);
    st.off = reinterpret_cast<Count2 *>(B + o_o);

    ks_raw_emit<<<blocks_for(n_lanes + 1, T), T, 0, c.stream>>>(run.nodes, run.subs, local_sub, run.strokes, run.n_local,
                                                            st.g, st.raw_off, st.raw_pt, st.raw_sub, st.raw_mode);
    ks_keep<<<blocks_for(R + 1, T), T, 0, c.stream>>>(st.raw_pt, st.raw_sub, R, st.keep);
    size_t t1 = 0, t2 = 0;
    Z2D_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, t1, st.keep, st.kept_off, R + 1, c.stream));
    Z2D_CUDA(cub::DeviceScan::ExclusiveScan(nullptr, t2, st.cnt, st.off, Sum2{}, Count2{0, 0}, R + 1, c.stream));
    if (c.scan_tmp.ensure(std::max(t1, t2) + 16)) return Z2D_ERR_OUT_OF_MEMORY;
    Z2D_CUDA(cub::DeviceScan::ExclusiveSum(c.scan_tmp.ptr, t1, st.keep, st.kept_off, R + 1, c.stream));
    ks_compact<<<blocks_for(R, T), T, 0, c.stream>>>(st.raw_pt, st.raw_sub, st.raw_mode, st.keep, st.kept_off, R,
                                                      st.q_pt, st.q_sub, st.q_mode);
    ks_sub_setup<<<blocks_for(run.n_subs, T), T, 0, c.stream>>>(run.subs, run.n_subs, run.strokes, st.g, st.raw_off,
                                                                 st.kept_off, st.q_pt, st.sub);
    ks_elem_count<<<blocks_for(R + 1, T), T, 0, c.stream>>>(run.subs, run.strokes, st.pen, st.sub, st.q_pt, st.q_sub,
                                                             st.q_mode, st.kept_off, R, st.elem, st.cnt);
    Z2D_CUDA(cub::DeviceScan::ExclusiveScan(c.scan_tmp.ptr, t2, st.cnt, st.off, Sum2{}, Count2{0, 0}, R + 1, c.stream));
    ks_stroke_tot<<<blocks_for(std::max(run.n_strokes, run.n_subs), T), T, 0, c.stream>>>(
        run.strokes, run.n_strokes, run.subs, run.n_subs, st.sub, st.off, R, st.region, run.stroke_edges, st.totals);
    c.timer_end(c.t_stroke, ts);
    c.launches += 9;
    return Z2D_OK;
}

int stroke_emit(Ctx &c, StrokeRun &run, const FillCmd *d_fills, FillState *d_st, DEdge *d_edges) {
    if (run.n_strokes == 0) return Z2D_OK;
    State &st = *reinterpret_cast<State *>(run.state);
    if (run.n_a < 0 || run.n_b < 0 || run.n_a + run.n_b > 0x7FFFFFFFll) {
        set_error("batch too large: more than 2^31 stroke polygon points");
        return Z2D_ERR_INVALID_ARGUMENT;
    }
    Carve cc;
    const size_t o_pa = cc.take<double2>(run.n_a + 1), o_pb = cc.take<double2>(run.n_b + 1);
    const size_t o_as = cc.take<int32_t>(run.n_a + 1), o_bs = cc.take<int32_t>(run.n_b + 1);
    if (c.stroke_c.ensure(cc.off)) return Z2D_ERR_OUT_OF_MEMORY;
    st.pa = reinterpret_cast<double2 *>(c.stroke_c.as<uint8_t>() + o_pa);
    st.pb = reinterpret_cast<double2 *>(c.stroke_c.as<uint8_t>() + o_pb);
    st.a_sub = reinterpret_cast<int32_t *>(c.stroke_c.as<uint8_t>() + o_as);
    st.b_sub = reinterpret_cast<int32_t *>(c.stroke_c.as<uint8_t>() + o_bs);
    constexpr int T = 128;
    const long long R = run.raw;
    cudaEvent_t ts = c.timer_begin(c.t_stroke);
    const auto elem_emit = st.elem ? ks_elem_emit<true> : ks_elem_emit<false>;
    elem_emit<<<blocks_for(R, T), T, 0, c.stream>>>(run.subs, run.strokes, st.pen, st.sub, st.region, st.q_pt, st.q_sub,
                                                     st.q_mode, st.kept_off, R, st.elem, st.off, st.pa, st.pb, st.a_sub,
                                                     st.b_sub);
    if (run.n_a + run.n_b > 0)
        ks_edges<<<blocks_for(run.n_a + run.n_b, T), T, 0, c.stream>>>(st.region, st.pa, st.pb, st.a_sub, st.b_sub,
                                                                        run.n_a, run.n_b, d_fills, d_st, d_edges);
    c.timer_end(c.t_stroke, ts);
    c.launches += 2;
    return Z2D_OK;
}

}  // namespace z2dg
