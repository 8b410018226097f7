// 2D Laguerre-cell kernels (sm_100a), FP64.
//
// One thread builds one cell.  Threads take Diracs in Morton (sorted) order so
// a warp works on 32 neighbouring cells and walks nearly the same tree nodes.
// The fast tier keeps the cell polygon in shared memory (one column per thread,
// coordinates relative to the Dirac, the order of the vertices in a register);
// cells that outgrow it, and all those of a small diagram, are built by the warp
// tier, a warp per cell, with polygons in shared memory or, past 64 vertices, in
// global scratch.  The fast tier's traversal stack lives in local memory.
//
// Reference behaviour restated here:
//  * traversal, eviction test and bisector cuts: SpZGrid::for_each_laguerre_cell
//    (src/sdot/PowerDiagram/Visitors/SpZGrid.tcc:494-719, eviction :475-480,
//    bisector :506-522); the reference pops boxes best-first from a priority
//    queue keyed on the float distance to the box centre, here a depth-first
//    walk pushes children farthest-first so the nearest is visited first.
//  * disc clipping (InBallW05, ball_cut after all plane cuts): :633-634.
//  * integrals: ConvexPolyhedron2::integration(Constant,Unit)
//    (ConvexPolyhedron2.tcc:1791-1843), add_centroid_contrib (:1047-1074),
//    for_each_boundary_item (:437-478).
//  * Hessian row: get_der_integrals_wrt_weights (get_der_integrals_wrt_weights.h:43-88):
//    off-diagonal -1/2 * len_ij / |x_i - x_j|, diagonal the sum of those plus
//    1/2 * arc_len / sqrt(w_i).
//  * bounds: ConvexPolyhedronAssembly::for_each_intersection
//    (ConvexPolyhedronAssembly.tcc:132-142) and ScaledImage::for_each_intersection
//    (ScaledImage.tcc:98-149).  A piece (cell intersected with an item or a
//    pixel) is produced by clipping the cell by the item/pixel half-planes,
//    which is the same convex set the reference gets by clipping the item by
//    the cell's lines.
#include "cell2d.cuh"
#include "geom2d.cuh"

namespace sdot {

// Counting builds (-DSDOT_COUNT) add up the work of the fast tier's walks,
// the terms of the per-cell operation count: [0] cut attempts, [1] vertices
// classified at them, [2] node tests, [3] vertices tested at them, [4]
// effective cuts, [5] final vertices, [6] cells built.  Release builds
// compile the counting away.
#ifdef SDOT_COUNT
static __device__ unsigned long long sdot_work[8];
#define SDOT_WORK_ADD(k, v) atomicAdd(&sdot_work[k], (unsigned long long)(v))
#else
#define SDOT_WORK_ADD(k, v) ((void)0)
#endif

namespace {

constexpr int STACK = 64;   // traversal stack (depth <= 17 levels, <= 3 pending siblings each)
// Warps (blocks) per SM of the warp tier in shared memory: 12 / 16 / 20 / 24 /
// 28 solve 60,000 clustered Diracs in 321 / 313 / 309 / 306 / 308 ms.
constexpr int MID_BLOCKS = 24;
constexpr int MID_WARPS = 148 * MID_BLOCKS;
constexpr int WTIER_WARPS = 148 * 4;  // warps of the warp tier in global scratch (few cells)

// Records the first failed consistency guard and flags the error word; the
// caller then skips the access.  Guards cover every index that comes from
// data (tree nodes, leaf ranges, item offsets), so a corrupt input gives an
// error status instead of a fault.
__device__ void guard_fail(const Cell2DArgs &A, int code, long long s, long long value) {
#ifdef __CUDA_ARCH__
    const bool first = A.guard && atomicCAS(&A.guard[0], 0, code) == 0;
#else
    const bool first = A.guard && A.guard[0] == 0;
    if (first) A.guard[0] = code;
#endif
    if (first) {
        A.guard[1] = int(s);
        A.guard[2] = int(value);
    }
    flag_error(A.err, DE_GUARD);
}

// Destination of one row (or id list): element k at col[k * stride]
// (col == nullptr: the output is not wanted, only counted).
struct Out {
    int *col;
    double *val;
    long long stride;
    int cap;
    int cnt = 0;
    SDOT_HDI Out(int *c, double *v, long long st, int cp) : col(c), val(v), stride(st), cap(cp) {}
    SDOT_HDI void emit(int j, double v) {
        if (col && cnt < cap) {
            col[cnt * stride] = j;
            if (val) val[cnt * stride] = v;
        }
        ++cnt;
    }
    SDOT_HDI bool ok() const { return !col || cnt <= cap; }
};

// Integrates a streamed polygon (one piece at a time) and collects the
// boundary measures for the Hessian row.  P: the cell's polygon view (its
// ids name the neighbours).  POLY: the density of a piece is the quadratic
// c0 + c1 x + c2 y + c3 x^2 + c4 x y + c5 y^2 (absolute coordinates) of a
// piecewise-quadratic image (ScaledImage with nb_coeffs = 6), integrated
// exactly: the edge-midpoint rule on each fan triangle for the mass (exact
// for quadratics), the 7-point rule (vertices 1/20, edge midpoints 2/15,
// centroid 9/20 of the area; exact for cubics) for the first moments, and
// Simpson's rule along each edge for the boundary measures (exact for
// quadratics).  The reference evaluates the same integrals from expanded
// closed forms (ConvexPolyhedron2.tcc:2181-2225 integration, :980-1044
// add_centroid_contrib, :180-214 for_each_boundary_item).
template <bool DIRECT, class P = PolyView<double>, bool POLY = false>
struct Sink {
    const P &cell;
    const double *pos;
    double c0x, c0y, sqw0;
    double cx, cy, r;
    double coeff = 1.0;
    // piece state
    double fx = 0, fy = 0, px = 0, py = 0;
    int pt = 0, cnt = 0;
    double tr2 = 0, arcs = 0, pm = 0, pcx = 0, pcy = 0;
    // cell totals
    double mass = 0, mass_c = 0, momx = 0, momy = 0, der0 = 0;
    // rows: DIRECT emits one item per line edge; otherwise measures are
    // summed per cell edge in acc (negative = edge not seen yet)
    double *acc;
    int acc_st;
    Out &row;
    long long n_diracs = 1LL << 40;
    const double *trans = nullptr;  // periodic domains: translation k of id j + (k + 1) n

    SDOT_HDI Sink(const P &c, const double *p, double x0, double y0, double sw, double r_, double *a, int ast,
                  Out &ro)
        : cell(c), pos(p), c0x(x0), c0y(y0), sqw0(sw), cx(x0), cy(y0), r(r_), acc(a), acc_st(ast), row(ro) {}

    double q[6] = {0, 0, 0, 0, 0, 0};  // POLY: the piece's density coefficients

    SDOT_HDI void begin_piece(double c) {
        coeff = c;
        cnt = 0;
        tr2 = arcs = pm = pcx = pcy = 0;
    }
    // POLY: the coefficients of pixel p, plane k at c[p + k * plane]
    SDOT_HDI void begin_piece_poly(const double *c, long long plane) {
        for (int k = 0; k < 6; ++k) q[k] = c[k * plane];
        begin_piece(1.0);
    }
    SDOT_HDI double f(double x, double y) const {
        return q[0] + q[1] * x + q[2] * y + q[3] * x * x + q[4] * x * y + q[5] * y * y;
    }
    SDOT_HDI void line(int t, double len) {
        if (t < 0) return;
        const int id = cell.I(t);
        if (id < 0) return;
        const double m = coeff * len;
        if (DIRECT) {
            // the neighbour, or the image of Dirac j under translation k for
            // an id j + (k + 1) n (get_der_integrals_wrt_weights.h:61-62)
            int j = id;
            double qx, qy;
            if (id >= n_diracs) {
                const int k = int(id / n_diracs) - 1;
                j = int(id % n_diracs);
                qx = pos[2 * j] + trans[2 * k];
                qy = pos[2 * j + 1] + trans[2 * k + 1];
            } else {
                qx = pos[2 * SDOT_CHECK_IDX(id, n_diracs, 3)];
                qy = pos[2 * id + 1];
            }
            const double dx = c0x - qx, dy = c0y - qy;
            const double dist = sqrt(dx * dx + dy * dy);
            if (dist != 0) {
                const double b = 0.5 * m / dist;
                row.emit(j, -b);
                der0 += b;
            }
        } else {
            double &a = acc[SDOT_CHECK_IDX(t, cell.cap, 2) * acc_st];
            a = a < 0 ? m : a + m;
        }
    }
    __device__ __forceinline__ void edge(double ax, double ay, int t, double bx, double by) {
        if (t == ID_ARC) {
            const Arc a = arc_segment(ax, ay, bx, by, cx, cy, r);
            arcs += a.area;
            pm += coeff * a.area;
            pcx += coeff * a.mx;
            pcy += coeff * a.my;
            der0 += 0.5 * (coeff * a.angle * r) / sqw0;
        } else {
            const double dx = bx - ax, dy = by - ay;
            double len = sqrt(dx * dx + dy * dy);
            if (POLY)  // Simpson along the edge; line() multiplies by coeff = 1
                len *= (1.0 / 6.0) * (f(ax, ay) + 4.0 * f(0.5 * (ax + bx), 0.5 * (ay + by)) + f(bx, by));
            line(t, len);
        }
    }
    // closing: the first vertex once more, for the edge back to it
    __device__ __forceinline__ void push(double x, double y, int tag, bool closing) {
        if (cnt == 0) {
            fx = x; fy = y;
        } else {
            edge(px, py, pt, x, y);
        }
        if (closing) return;
        if (++cnt >= 3) {
            const double t2 = fx * (py - y) + px * (y - fy) + x * (fy - py);
            tr2 += t2;
            if (POLY) {
                const double a = 0.5 * t2;
                const double m1x = 0.5 * (fx + px), m1y = 0.5 * (fy + py), m2x = 0.5 * (px + x), m2y = 0.5 * (py + y);
                const double m3x = 0.5 * (x + fx), m3y = 0.5 * (y + fy);
                const double gx = (1.0 / 3.0) * (fx + px + x), gy = (1.0 / 3.0) * (fy + py + y);
                const double f1 = f(m1x, m1y), f2 = f(m2x, m2y), f3 = f(m3x, m3y);
                const double fa = f(fx, fy), fb = f(px, py), fc = f(x, y), fg = f(gx, gy);
                pm += a * (1.0 / 3.0) * (f1 + f2 + f3);
                pcx += a * ((1.0 / 20.0) * (fx * fa + px * fb + x * fc) +
                            (2.0 / 15.0) * (m1x * f1 + m2x * f2 + m3x * f3) + (9.0 / 20.0) * gx * fg);
                pcy += a * ((1.0 / 20.0) * (fy * fa + py * fb + y * fc) +
                            (2.0 / 15.0) * (m1y * f1 + m2y * f2 + m3y * f3) + (9.0 / 20.0) * gy * fg);
            } else {
                const double lea = 0.5 * t2 * coeff;
                const double f = (1.0 / 3.0) * lea;
                pcx += f * (fx + px + x);
                pcy += f * (fy + py + y);
                pm += lea;
            }
        }
        px = x; py = y; pt = tag;
    }
    // radius: the disc radius after clipping (> 0 keeps a vertex-free piece
    // as the full disc), or -1 when there is no disc.
    SDOT_HDI void end_piece(double radius) {
        if (cnt == 0) {
            if (radius > 0) {
                const double lea = kPi * (radius * radius) * coeff;
                mass += lea;
                mass_c += lea;
                momx += lea * cx;
                momy += lea * cy;
                der0 += 0.5 * (coeff * 2 * kPi * radius) / sqw0;
            }
            return;
        }
        mass += POLY ? pm : coeff * (tr2 * 0.5 + arcs);
        mass_c += pm;
        momx += pcx;
        momy += pcy;
    }
};

// Area of a streamed (clipped) polygon, segments of the clipping disc
// included (fan from the first vertex plus the arc segments, as Sink).
struct AreaSink {
    double cx, cy, r;
    double fx = 0, fy = 0, px = 0, py = 0;
    int pt = 0, cnt = 0;
    double tr2 = 0, arcs = 0;
    __device__ AreaSink(double x, double y, double rr) : cx(x), cy(y), r(rr) {}
    __device__ __forceinline__ void push(double x, double y, int tag, bool closing) {
        if (cnt == 0) {
            fx = x;
            fy = y;
        } else if (pt == ID_ARC) {
            arcs += arc_segment(px, py, x, y, cx, cy, r).area;
        }
        if (closing) return;
        if (++cnt >= 3) tr2 += fx * (py - y) + px * (y - fy) + x * (fy - py);
        px = x;
        py = y;
        pt = tag;
    }
    // radius: the disc radius after clipping (> 0 keeps a vertex-free piece
    // as the full disc), or -1 when there is no disc
    SDOT_HDI double area(double radius) const {
        if (cnt == 0) return radius > 0 ? kPi * radius * radius : 0.0;
        return 0.5 * tr2 + arcs;
    }
};

// The cell (n vertices; box [xmin, xmax] x [ymin, ymax], or what of it its disc
// reaches) cut to a pixel, into `piece`; an edge keeps its vertex number in the
// cell as its id, a pixel's edge gets PID_OWN.  Only the pixel's lines that
// pass through the box cut.  Returns the number of vertices (piece.cap, at least
// n + 4, at most).
// The piece lies in memory of its own (shared in the fast tier) between short
// loops; streamed through four nested clip stages and the disc's, each holding
// its state in local memory, with 4 to 8 KB of spills a thread, 500,000 cells
// over a 512 x 512 image took 36.5 ms, now 4.3 ms (B200).
template <class P>
__device__ __forceinline__ int clip_to_pixel(const PolyView<double> &piece, const P &cell, int n, double x0, double x1,
                                             double y0, double y1, double xmin, double xmax, double ymin, double ymax) {
    for (int k = 0; k < n; ++k) {
        piece.X(k) = cell.X(k);
        piece.Y(k) = cell.Y(k);
        piece.I(k) = k;
    }
    int m = n;
#pragma unroll 1
    for (int side = 0; side < 4; ++side) {
        const bool y = side >= 2, hi = side & 1;
        const double c = y ? (hi ? y1 : y0) : (hi ? x1 : x0);
        // (the other lines' room is kept)
        if (hi ? (y ? ymax : xmax) > c : (y ? ymin : xmin) < c)
            m = axis_cut(piece, m, y, c, hi ? -1.0 : 1.0, PID_OWN, piece.cap - 3 + side);
    }
    return m;
}

// Integrates the cell of sorted Dirac s (its polygon before disc clipping,
// n vertices) over the pixels of the raster that its bounding box meets:
// get_image_integrals / get_image_of_cell_nums
// (get_image_integrals.h:16-78, get_image_of_cell_nums.h:13-80) clip each
// pixel box by the cell and integrate; here the cell is clipped by the pixel's
// four lines (and the disc), the same convex set.
template <bool BALL, class P>
__device__ void raster_cell(const Cell2DArgs &A, long long s, const P &cell, int n, double c0x, double c0y, double r,
                            const PolyView<double> &piece) {
    if (n <= 0) return;
    double xmin = cell.X(0), xmax = xmin, ymin = cell.Y(0), ymax = ymin;
    for (int k = 1; k < n; ++k) {
        xmin = fmin(xmin, cell.X(k)); xmax = fmax(xmax, cell.X(k));
        ymin = fmin(ymin, cell.Y(k)); ymax = fmax(ymax, cell.Y(k));
    }
    if (BALL) {
        xmin = fmax(xmin, c0x - r); xmax = fmin(xmax, c0x + r);
        ymin = fmax(ymin, c0y - r); ymax = fmin(ymax, c0y + r);
    }
    const double psx = (A.ras_hi[0] - A.ras_lo[0]) / A.ras_nx, psy = (A.ras_hi[1] - A.ras_lo[1]) / A.ras_ny;
    const double fx0 = floor((xmin - A.ras_lo[0]) / psx), fx1 = floor((xmax - A.ras_lo[0]) / psx);
    const double fy0 = floor((ymin - A.ras_lo[1]) / psy), fy1 = floor((ymax - A.ras_lo[1]) / psy);
    if (!(fx1 >= 0 && fy1 >= 0 && fx0 < A.ras_nx && fy0 < A.ras_ny)) return;  // outside the raster (or NaN)
    const int ix0 = int(fmax(fx0, 0.0)), ix1 = int(fmin(fx1, double(A.ras_nx - 1)));
    const int iy0 = int(fmax(fy0, 0.0)), iy1 = int(fmin(fy1, double(A.ras_ny - 1)));
    const long long orig = A.perm ? A.perm[s] : s;
    for (int iy = iy0; iy <= iy1; ++iy) {
        const double y0 = A.ras_lo[1] + psy * double(iy), y1 = A.ras_lo[1] + psy * double(iy + 1);
        for (int ix = ix0; ix <= ix1; ++ix) {
            const double x0 = A.ras_lo[0] + psx * double(ix), x1 = A.ras_lo[0] + psx * double(ix + 1);
            AreaSink as(c0x, c0y, r);
            const int np = clip_to_pixel(piece, cell, n, x0, x1, y0, y1, xmin, xmax, ymin, ymax);
            const double m = A.coeff * as.area(stream_piece<BALL, true>(
                                           piece, np, [&](int k) { return piece.I(k); }, c0x, c0y, r, as));
            if (m == 0) continue;
            const long long pix = (long long)iy * A.ras_nx + ix;
#ifdef __CUDA_ARCH__
            if (A.ras) {
                atomicAdd(&A.ras[3 * pix], m * c0x);
                atomicAdd(&A.ras[3 * pix + 1], m * c0y);
                atomicAdd(&A.ras[3 * pix + 2], m);
            }
            if (A.ras_nums) atomicMax(&A.ras_nums[pix], orig);
#else
            if (A.ras) {
                A.ras[3 * pix] += m * c0x;
                A.ras[3 * pix + 1] += m * c0y;
                A.ras[3 * pix + 2] += m;
            }
            if (A.ras_nums && A.ras_nums[pix] < orig) A.ras_nums[pix] = orig;
#endif
        }
    }
}

// Records the ids of the streamed (disc-clipped) cell boundary.
template <class P>
struct NbSink {
    const P &cell;
    Out &out;
    __device__ NbSink(const P &c, Out &o) : cell(c), out(o) {}
    __device__ void push(double, double, int tag, bool) { out.emit(tag == ID_ARC ? ID_ARC : cell.I(tag), 0.0); }
};

// The children [first, first + nch) of a box (2 <= nch <= 4) in ch[0 ..
// nch), farthest first by the float squared distance from c0 to their box
// centres (the key of the reference's queue), the box shifted by (tx, ty)
// when PER.  A fixed network of five exchanges over four slots (missing
// children keyed -1, after every real key) keeps the arrays in registers.
template <bool PER>
SDOT_HDI void order_children(const Cell2DArgs &A, int first, int nch, double c0x, double c0y, double tx, double ty,
                             int ch[4]) {
    float key[4] = {-1.f, -1.f, -1.f, -1.f};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        ch[c] = first + c;
        if (c < nch) {
            const TreeNode<2> &cn = A.nodes[SDOT_CHECK_IDX(first + c, A.max_nodes, 5)];
            const double cx = 0.5 * (cn.lo[0] + cn.hi[0]), cy = 0.5 * (cn.lo[1] + cn.hi[1]);
            const double mx = c0x - (PER ? cx + tx : cx);
            const double my = c0y - (PER ? cy + ty : cy);
            key[c] = float(mx * mx + my * my);
        }
    }
    auto cx = [&](int a, int b) {
        if (key[a] < key[b]) {
            const float tk = key[a];
            key[a] = key[b];
            key[b] = tk;
            const int tc = ch[a];
            ch[a] = ch[b];
            ch[b] = tc;
        }
    };
    cx(0, 1);
    cx(2, 3);
    cx(0, 2);
    cx(1, 3);
    cx(1, 2);
}

// The polygon of one thread's cell in the fast tier: up to CAP vertices in
// shared memory (slot k of thread t at [k * BS + t]) in coordinates relative to
// the cell's Dirac, and the order of the slots in a register: nibble k of
// `order` is the slot of vertex k, the nibbles past the last vertex are the free
// slots.  A cut then moves no vertex: it writes the two new ones and rearranges
// nibbles (the copy loops it takes the place of ran as long as the longest of
// the warp).
template <int CAP, int BS>
struct Ring {
    static_assert(CAP <= 16, "slots of four bits in a 64-bit word");
    static constexpr unsigned long long ALL = CAP == 16 ? ~0ull : (1ull << (4 * CAP)) - 1;
    double *x, *y;
    int *id;
    unsigned long long order = 0xfedcba9876543210ull & ALL;
    double c0x, c0y;
    int cap = CAP;  // bound of the debug checks

    __device__ int slot(int k) const { return int(order >> (4 * SDOT_CHECK_IDX(k, CAP, 1))) & 15; }
    __device__ double &ux(int k) const { return x[slot(k) * BS]; }
    __device__ double &uy(int k) const { return y[slot(k) * BS]; }
    __device__ int &I(int k) const { return id[slot(k) * BS]; }
    // absolute coordinates, for the streaming stages
    __device__ double X(int k) const { return c0x + ux(k); }
    __device__ double Y(int k) const { return c0y + uy(k); }

    // The mask of a cut's farthest run, where rounding gives more than one.
    __device__ __noinline__ unsigned one_run(int n, double nx, double ny, double b) const {
        int i1, gone;
        farthest_run(n, [&](int k) { return b - (ux(k) * nx + uy(k) * ny); }, i1, gone);
        const unsigned run = (1u << gone) - 1u;
        return (run << i1 | run >> (n - i1)) & ((1u << n) - 1u);
    }

    // Cuts the polygon (n vertices) by nx ux + ny uy <= b; bit k of mask:
    // vertex k is outside.  Same new vertices at the same places as
    // plane_cut_apply: with i1 the first and i2 the last vertex removed, A on
    // the edge into i1 takes the cut's id, B on the edge out of i2 keeps that
    // edge's.  Returns the new count, or -1 past CAP.
    __device__ int cut(int n, unsigned mask, double nx, double ny, double b, int cut_id) {
        const unsigned starts = mask & ~(mask << 1 | mask >> (n - 1));
        if (starts & (starts - 1)) mask = one_run(n, nx, ny, b);
        const CutFacts f = cut_facts(mask, n);
        if (f.nb_out == n) return 0;
        const int nb_in = n - f.nb_out;
        if (f.nb_out == 1 && n + 1 > CAP) return -1;
        const bool wrap = f.out_last && f.first_out == 0;
        const int i3 = wrap ? f.first_in : f.first_out + f.nb_out;  // may be n: vertex 0
        const int i1 = wrap ? f.first_in + nb_in : f.first_out;
        const int s1 = slot(i1), s0 = slot(i1 == 0 ? n - 1 : i1 - 1);
        const int s2 = slot(i3 == 0 ? n - 1 : i3 - 1), s3 = slot(i3 == n ? 0 : i3);
        const double p0x = x[s0 * BS], p0y = y[s0 * BS], p1x = x[s1 * BS], p1y = y[s1 * BS];
        const double p2x = x[s2 * BS], p2y = y[s2 * BS], p3x = x[s3 * BS], p3y = y[s3 * BS];
        const double d0 = b - (p0x * nx + p0y * ny), d1 = b - (p1x * nx + p1y * ny);
        const double d2 = b - (p2x * nx + p2y * ny), d3 = b - (p3x * nx + p3y * ny);
        // the two edge ratios d0 / (d1 - d0) and d3 / (d2 - d3) by one division
        const double u = d1 - d0, v = d2 - d3, r = 1.0 / (u * v);
        const double m1 = d0 * v * r, m2 = d3 * u * r;
        const int id2 = id[s2 * BS];
        int sa, sb;  // slots of A and B
        if (wrap) {
            // [B, kept run, A]: B takes the place before the kept run, A the
            // one after it, and the order is turned to start at B
            sa = s1;
            sb = s2;
            const int t = 4 * (i3 - 1);
            order = ((order >> t) | (order << (4 * CAP - t))) & ALL;
        } else if (f.nb_out == 1) {
            // A in the removed place, B in a free slot after it
            sa = s1;
            sb = slot(n);
            const unsigned long long low = (1ull << (4 * (i1 + 1))) - 1;
            const unsigned long long used = n + 1 == 16 ? ~0ull : (1ull << (4 * (n + 1))) - 1;
            order = (order & (low | ~used)) | ((unsigned long long)sb << (4 * (i1 + 1))) |
                    (((order & ~low) << 4) & used & ~((1ull << (4 * (i1 + 2))) - 1));
        } else {
            // A and B in the first two removed places, the other removed ones
            // to the end
            sa = s1;
            sb = slot(i1 + 1);
            if (f.nb_out > 2) {
                const int keep = 4 * (i1 + 2), gone = 4 * (f.nb_out - 2);
                const unsigned long long low = (1ull << keep) - 1;
                const unsigned long long run = (order >> keep) & ((1ull << gone) - 1);
                order = (order & low) | (((order >> gone) & ~low) & ALL) | (run << (4 * CAP - gone));
            }
        }
        x[sa * BS] = p0x - m1 * (p1x - p0x);
        y[sa * BS] = p0y - m1 * (p1y - p0y);
        id[sa * BS] = cut_id;
        x[sb * BS] = p3x - m2 * (p2x - p3x);
        y[sb * BS] = p3y - m2 * (p2y - p3y);
        id[sb * BS] = id2;
        return nb_in + 2;
    }
};

// Builds the Laguerre cells of the warp's 32 sorted Diracs, one per lane
// (before any disc clipping).  The walk of each is
// SpZGrid::for_each_laguerre_cell's (SpZGrid.tcc:494-719): boxes popped
// nearest-first (children pushed farthest-first, keyed on the float squared
// distance from c0 to the box centre as the reference's queue), skipped when
// the eviction test holds for every vertex (SpZGrid.tcc:475-480), a leaf's
// Diracs cut in index order (bisector SpZGrid.tcc:506-522).
// The lanes run node tests together and cuts together: node steps go on until
// at most WAIT of 32 lanes still look for a leaf while others hold one, then
// the leaves are cut out of every cell that holds one.  (With one loop in which
// each lane took whichever step its walk was at, every turn ran the node test,
// the ordering of children, the cut test and the cut for some of the lanes:
// 6.2 of 32 lanes active.)
// Returns per lane the vertex count, -1 on capacity (or stack / visit cap)
// overflow, -2 on a failed guard; every lane of the warp calls it (live: it has
// a cell).
// PER (periodic domains): after the tree, the walk visits it again once per
// translation t, as the tree of the Diracs x_j + t (SpZGrid.tcc:558-561:
// every translation's root enters the front; boxes and Diracs are shifted by
// t, :396-397 and :608-611); a cut by the image of Dirac j under translation
// k carries the id j + (k + 1) n, and the Dirac's own images cut it too.
// WAIT 4 / 8 / 12 / 16 / 22: 3.47 / 3.29 / 3.26 / 3.26 / 3.30 ms at 1M Diracs,
// 0.75 / 0.69 / 0.66 / 0.65 / 0.67 ms at 147,000.
constexpr int WAIT = 12;

template <bool PER, int CAP, int BS>
__device__ int build_cell(const Cell2DArgs &A, long long s, bool live, Ring<CAP, BS> &cell, double w0) {
    constexpr unsigned FULL = 0xffffffffu;
    const double c0x = cell.c0x, c0y = cell.c0y;
    int n = live ? A.start_n : 0;
    for (int k = 0; k < n; ++k) {
        cell.ux(k) = A.start_xy[2 * k] - c0x;
        cell.uy(k) = A.start_xy[2 * k + 1] - c0y;
        cell.I(k) = domain_id(k);
    }
    // The walk's memory reads are issued a step before their use: the node
    // popped next is kept in a register (the stack holds the others), and the
    // position and weight of the next Dirac of a leaf are loaded while the
    // current one cuts.
    int stack[STACK];
    int sp = 0;                 // stack entries below `top`
    int top = 0;                // the node the next node step pops
    bool has_top = true;
    bool done = !live;
    int j = 0, je = 0;          // Diracs of the current leaf still to cut by
    double cjx = 0, cjy = 0, cjw = 0;  // Dirac j
    int visits = 0;
    int sym = -1;               // PER: the translation of the current walk (-1: none)
    double tx = 0, ty = 0;      // and its vector
    auto skip_self = [&](int k) { return (!PER || sym < 0) && k == s ? k + 1 : k; };
    // shifted by the current translation (PER only: adding a zero would not
    // be free, it turns -0 into +0)
    auto tr = [&](double v, double t) { return PER ? v + t : v; };
    auto load = [&](int k) {
        (void)SDOT_CHECK_IDX(k, A.n, 6);
        const double2 p = reinterpret_cast<const double2 *>(A.pos)[k];
        cjx = tr(p.x, tx);
        cjy = tr(p.y, ty);
        cjw = A.w[k];
    };
    auto stop = [&](int result) {
        n = result;
        done = true;
        j = je = 0;
    };
    while (true) {
        // ---- node steps
        while (true) {
            const bool want = !done && j >= je;
            const unsigned wm = __ballot_sync(FULL, want), hm = __ballot_sync(FULL, j < je);
            if (!wm || (hm && 32 * __popc(wm) <= WAIT * A.lanes)) break;
            if (!want) continue;
            if (!has_top) {
                if (!PER || sym + 1 >= A.ntrans) {
                    done = true;
                    continue;
                }
                // the next translation's walk starts from the root again
                ++sym;
                tx = A.trans[2 * sym];
                ty = A.trans[2 * sym + 1];
                top = 0;
                has_top = true;
            }
            if (++visits > (PER ? (A.ntrans + 1) * A.max_nodes : A.max_nodes)) {  // each tree walk visits a node once
                flag_error(A.err, DE_ITER);
                stop(-1);
                continue;
            }
            const int node = top;
            if (sp > 0)
                top = stack[--sp];
            else
                has_top = false;
            const TreeNode<2> nd = A.nodes[SDOT_CHECK_IDX(node, A.max_nodes, 4)];
            const double lo0 = tr(nd.lo[0], tx) - c0x, lo1 = tr(nd.lo[1], ty) - c0y;
            const double hi0 = tr(nd.hi[0], tx) - c0x, hi1 = tr(nd.hi[1], ty) - c0y;
            // the eviction test, left at the first vertices that fail it, as
            // the reference's all_pos does
            bool need = false;
            for (int k = 0; k < n && !need; k += 2) {
                const int a = cell.slot(k), b = cell.slot(k + 1 < n ? k + 1 : k);
                const double ax = cell.x[a * BS], ay = cell.y[a * BS], bx = cell.x[b * BS], by = cell.y[b * BS];
                const double gx = gap(lo0, hi0, ax), gy = gap(lo1, hi1, ay);
                const double hx = gap(lo0, hi0, bx), hy = gap(lo1, hi1, by);
                need = !(ax * ax + ay * ay - w0 <= gx * gx + gy * gy - nd.maxw) ||
                       !(bx * bx + by * by - w0 <= hx * hx + hy * hy - nd.maxw);
                // (the second one's is no work of the algorithm's if the first fails)
                SDOT_WORK_ADD(3, k + 1 < n && ax * ax + ay * ay - w0 <= gx * gx + gy * gy - nd.maxw ? 2 : 1);
            }
            SDOT_WORK_ADD(2, 1);
            if (!need) continue;  // every vertex passes: the box is evicted
            if (nd.b < 0) {
                const int first = nd.a, nch = -nd.b;
                if (nch < 2 || nch > 4 || first < 1 || first + nch > A.max_nodes) {
                    guard_fail(A, 1, s, node);
                    stop(-2);
                    continue;
                }
                if (sp + nch > STACK) {
                    flag_error(A.err, DE_STACK);
                    stop(-1);
                    continue;
                }
                int ch[4];
                order_children<PER>(A, first, nch, c0x, c0y, tx, ty, ch);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (c < nch) {
                        if (has_top) stack[sp++] = top;
                        top = ch[c];
                        has_top = true;
                    }
                }
            } else {
                if (nd.a < 0 || nd.b > A.n) {
                    guard_fail(A, 2, s, node);
                    stop(-2);
                    continue;
                }
                j = skip_self(nd.a);
                je = nd.b;
                if (j < je) load(j);
            }
        }
        if (!__any_sync(FULL, j < je)) break;  // no leaf, and no walk goes on
        // ---- cuts
        while (__any_sync(FULL, j < je)) {
            if (!(j < je)) continue;
            // the bisector (SpZGrid.tcc:506-522) relative to c0: n . u <= b.
            // One position twice has none (the reference's is not a number)
            const double nx = cjx - c0x, ny = cjy - c0y;
            const double b = 0.5 * (nx * nx + ny * ny) + 0.5 * (w0 - cjw);
            const int jc = j;
            j = skip_self(j + 1);
            if (j < je) load(j);
            unsigned mask = 0;
            for (int k0 = 0; k0 < n; k0 += 4) {
                const unsigned h = unsigned(cell.order >> (4 * k0));
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int a = int(h >> (4 * k)) & 15;
                    const double d = b - (cell.x[a * BS] * nx + cell.y[a * BS] * ny);
                    mask |= unsigned(d < 0.0) << (k0 + k);
                }
            }
            mask &= (1u << n) - 1u;
            SDOT_WORK_ADD(0, 1);
            SDOT_WORK_ADD(1, n);
            if (mask && (nx != 0 || ny != 0)) {
                SDOT_WORK_ADD(4, 1);
                n = cell.cut(n, mask, nx, ny, b, PER ? jc + (sym + 1) * int(A.n) : jc);
                if (n <= 0) stop(n);
            }
        }
    }
    return n;
}

// Vertex k relative to the Dirac at c0.
template <class P>
__device__ double rel_x(const P &cell, int k, double c0x) { return cell.X(k) - c0x; }
template <class P>
__device__ double rel_y(const P &cell, int k, double c0y) { return cell.Y(k) - c0y; }
template <int CAP, int BS>
__device__ double rel_x(const Ring<CAP, BS> &cell, int k, double) { return cell.ux(k); }
template <int CAP, int BS>
__device__ double rel_y(const Ring<CAP, BS> &cell, int k, double) { return cell.uy(k); }

// Per-cell work once the polygon of Dirac s is built (n vertices; -1: a
// capacity was exceeded, -2: a guard failed).  Returns false when a capacity
// was exceeded (the cell is then rebuilt by the next tier, which rewrites
// every output of it).
// piece: room for n + 4 vertices (image and raster modes).
template <int MODE, bool BALL, class P>
__device__ bool finish_cell(const Cell2DArgs &A, long long s, const P &cell, int n, double *acc, int acc_st, Out &row,
                            Out &nbo, const PolyView<double> &piece) {
    const double c0x = A.pos[2 * s], c0y = A.pos[2 * s + 1], w0 = A.w[s];
    if (n == -2) {
        // failed guard: report a NaN cell, not an overflow
        if (A.mass) A.mass[s] = nan("");
        if (A.mass_c) A.mass_c[s] = nan("");
        if (A.ctd) A.ctd[2 * s] = A.ctd[2 * s + 1] = nan("");
        row.emit(int(s), 0.0);
        return true;
    }
    if (n < 0) return false;

    const double r = BALL ? sqrt(w0) : -1.0;
    if (MODE == DM_RASTER) {
        raster_cell<BALL>(A, s, cell, n, c0x, c0y, r, piece);
        return true;
    }
    constexpr bool DIRECT = MODE == DM_SINGLE || MODE == DM_PERIODIC;
    using SinkT = Sink<DIRECT, P, MODE == DM_IMAGE6>;
    SinkT sink(cell, A.pos, c0x, c0y, BALL ? r : sqrt(w0), r, acc, acc_st, row);
    sink.n_diracs = A.n;
    sink.trans = A.trans;

    if (DIRECT && !BALL) {
        // reference order: fan from vertex 0, boundary items from edge (n-1 ->
        // 0), in coordinates about the Dirac (no cancellation of positions of
        // the domain's size)
        sink.begin_piece(A.coeff);
        if (n > 0) {
            const double ax = rel_x(cell, 0, c0x), ay = rel_y(cell, 0, c0y);
            double px = rel_x(cell, n - 1, c0x), py = rel_y(cell, n - 1, c0y);
            double bx = ax, by = ay, tr2 = 0;
            for (int i = 0; i < n; ++i) {
                const double cx = i ? rel_x(cell, i, c0x) : ax, cy = i ? rel_y(cell, i, c0y) : ay;
                sink.line(i ? i - 1 : n - 1, sqrt((cx - px) * (cx - px) + (cy - py) * (cy - py)));
                px = cx;
                py = cy;
                if (i >= 2) {
                    const double t2 = ax * (by - cy) + bx * (cy - ay) + cx * (ay - by);
                    tr2 += t2;
                    const double lea = 0.5 * t2 * A.coeff;
                    const double f = (1.0 / 3.0) * lea;
                    sink.momx += f * (ax + bx + cx);
                    sink.momy += f * (ay + by + cy);
                    sink.mass_c += lea;
                }
                bx = cx;
                by = cy;
            }
            sink.mass = A.coeff * (tr2 * 0.5);
            // moments about the origin, as the other modes leave them
            sink.momx += c0x * sink.mass_c;
            sink.momy += c0y * sink.mass_c;
        }
    } else if (DIRECT) {
        sink.begin_piece(A.coeff);
        sink.end_piece(stream_piece<true, true>(cell, n, [](int k) { return k; }, c0x, c0y, r, sink));
    } else {
        for (int k = 0; k < n; ++k) acc[k * acc_st] = -1.0;
        if (n > 0) {
            if (MODE == DM_IMAGE || MODE == DM_IMAGE6) {
                double xmin = cell.X(0), xmax = xmin, ymin = cell.Y(0), ymax = ymin;
                for (int k = 1; k < n; ++k) {
                    xmin = fmin(xmin, cell.X(k)); xmax = fmax(xmax, cell.X(k));
                    ymin = fmin(ymin, cell.Y(k)); ymax = fmax(ymax, cell.Y(k));
                }
                if (BALL) {
                    xmin = fmax(xmin, c0x - r); xmax = fmin(xmax, c0x + r);
                    ymin = fmax(ymin, c0y - r); ymax = fmin(ymax, c0y + r);
                }
                const double psx = (A.img_hi[0] - A.img_lo[0]) / A.img_nx;
                const double psy = (A.img_hi[1] - A.img_lo[1]) / A.img_ny;
                // pixels outside the cell's bounding box give empty pieces
                int ix0 = int(floor((xmin - A.img_lo[0]) / psx)), ix1 = int(floor((xmax - A.img_lo[0]) / psx));
                int iy0 = int(floor((ymin - A.img_lo[1]) / psy)), iy1 = int(floor((ymax - A.img_lo[1]) / psy));
                ix0 = max(ix0, 0); iy0 = max(iy0, 0);
                ix1 = min(ix1, A.img_nx - 1); iy1 = min(iy1, A.img_ny - 1);
                for (int iy = iy0; iy <= iy1; ++iy) {
                    const double y0 = A.img_lo[1] + psy * double(iy), y1 = A.img_lo[1] + psy * double(iy + 1);
                    for (int ix = ix0; ix <= ix1; ++ix) {
                        const double x0 = A.img_lo[0] + psx * double(ix), x1 = A.img_lo[0] + psx * double(ix + 1);
                        if (MODE == DM_IMAGE6)
                            sink.begin_piece_poly(A.img + (long long)iy * A.img_nx + ix,
                                                  (long long)A.img_nx * A.img_ny);
                        else
                            sink.begin_piece(A.img[(long long)iy * A.img_nx + ix]);
                        const int m = clip_to_pixel(piece, cell, n, x0, x1, y0, y1, xmin, xmax, ymin, ymax);
                        sink.end_piece(stream_piece<BALL && MODE == DM_IMAGE, true>(
                            piece, m, [&](int k) { return piece.I(k); }, c0x, c0y, r, sink));
                    }
                }
            }
        }
        if (A.rows.cnt) {
            for (int i1 = 0, i0 = n - 1; i1 < n; i0 = i1++) {
                const double m = acc[i0 * acc_st];
                if (m < 0) continue;
                const int id = cell.I(i0);
                if (id < 0 || id >= A.n) {
                    guard_fail(A, 4, s, id);
                    continue;
                }
                const double dx = c0x - A.pos[2 * id], dy = c0y - A.pos[2 * id + 1];
                const double dist = sqrt(dx * dx + dy * dy);
                if (dist != 0) {
                    const double b = 0.5 * m / dist;
                    row.emit(id, -b);
                    sink.der0 += b;
                }
            }
        }
    }

    if (A.rows.cnt) {
        row.emit(int(s), sink.der0);
        if (!row.ok()) return false;
    }
    if (A.nb.cnt) {
        if (BALL) {
            NbSink<P> nbs(cell, nbo);
            stream_piece<true, false>(cell, n, [](int k) { return k; }, c0x, c0y, r, nbs);
        } else {
            for (int k = 0; k < n; ++k) nbo.emit(cell.I(k), 0.0);
        }
        if (!nbo.ok()) return false;
    }
    if (A.mass) A.mass[s] = sink.mass;
    if (A.mass_c) A.mass_c[s] = sink.mass_c;
    if (A.ctd) {
        const double d = sink.mass_c + (sink.mass_c == 0);
        A.ctd[2 * s] = sink.momx / d;
        A.ctd[2 * s + 1] = sink.momy / d;
    }
    return true;
}

// Hands cell s to the warp tier.  The list holds n entries and one launch
// appends each cell at most once; the bound check turns a count that was not
// reset between launches into an error instead of a write past the list.
__device__ void push_overflow(const Cell2DArgs &A, long long s) {
    const int k = atomicAdd(A.ovf_cnt, 1);
    if (k < A.n)
        A.ovf_list[k] = int(s);
    else
        flag_error(A.err, DE_CAPACITY);
}

// Shared memory of a fast-tier block: the polygons, in the image modes the
// per-edge accumulators, and in these and the raster mode the piece of a pixel.
// Measured (1M clustered mix, FP64): 4.12 ms with one loop of mixed steps and
// polygons moved in shared memory -> 3.25 ms; 77k warp instructions per warp
// (95k), 7.6 of 32 lanes active, issue 71%: bound by instruction issue, over
// half of it the vertex loops of the node tests.  Blocks of 32 / 64 / 128: 3.22
// / 3.26 / 3.48 ms; 10 instead of 12 of them per SM: 3.40 ms.
constexpr int BS = 64;  // threads of a fast-tier block
constexpr int fast_blocks(int mode, bool ball) {
    return mode == DM_IMAGE || mode == DM_IMAGE6 || mode == DM_RASTER ? 5 : ball ? 8 : 12;
}
constexpr bool has_acc(int mode) { return mode == DM_IMAGE || mode == DM_IMAGE6; }
constexpr bool has_piece(int mode) { return has_acc(mode) || mode == DM_RASTER; }
constexpr int PCAP = CAP_FAST_2D + 4;  // four lines of a pixel add a vertex each
template <int MODE>
constexpr size_t fast_smem() {
    return size_t(BS) * (CAP_FAST_2D * (20 + (has_acc(MODE) ? 8 : 0)) + (has_piece(MODE) ? PCAP * 20 : 0));
}

template <int MODE, bool BALL>
__global__ void __launch_bounds__(BS, fast_blocks(MODE, BALL)) k_cells2d(const Cell2DArgs A) {
    extern __shared__ double smem[];
    constexpr int CAP = CAP_FAST_2D;
    const int t = threadIdx.x;
    // the doubles, then the ids
    double *acc = smem + 2 * CAP * BS;
    double *px = acc + (has_acc(MODE) ? CAP * BS : 0);
    int *sid = reinterpret_cast<int *>(px + (has_piece(MODE) ? 2 * PCAP * BS : 0));
    const PolyView<double> piece{px + t, px + PCAP * BS + t, sid + CAP * BS + t, BS, PCAP};
    const long long s = (blockIdx.x * (long long)BS + t) / 32 * A.lanes + (t & 31);
    const bool live = (t & 31) < A.lanes && s < A.n;
    Ring<CAP, BS> cell;
    cell.x = smem + t;
    cell.y = smem + CAP * BS + t;
    cell.id = sid + t;
    cell.c0x = live ? A.pos[2 * s] : 0;
    cell.c0y = live ? A.pos[2 * s + 1] : 0;
    const int n = build_cell<MODE == DM_PERIODIC, CAP, BS>(A, s, live, cell, live ? A.w[s] : 0);
    if (!live) return;
    SDOT_WORK_ADD(5, n > 0 ? n : 0);
    SDOT_WORK_ADD(6, 1);
    Out row(A.rows.cnt ? A.rows.col + s : nullptr, A.rows.cnt ? A.rows.val + s : nullptr, A.rows.stride, A.rows.cap);
    Out nbo(A.nb.cnt ? A.nb.col + s : nullptr, nullptr, A.nb.stride, A.nb.cap);
    if (finish_cell<MODE, BALL>(A, s, cell, n, acc + t, BS, row, nbo, piece)) {
        if (A.rows.cnt) A.rows.cnt[s] = row.cnt;
        if (A.nb.cnt) A.nb.cnt[s] = nbo.cnt;
    } else {
        push_overflow(A, s);
    }
}

// Polygon, accumulators and row buffers of one warp of the warp tier,
// contiguous (vertex k at index k) so that the lanes read 32 vertices at once.
struct WarpScratch {
    PolyView<double> cell, piece;
    double *acc, *row_val;
    int *row_col, *nb_id;
    __device__ WarpScratch(double *base, int cap) {
        double *p = base;
        cell = PolyView<double>{p, p + cap, reinterpret_cast<int *>(p + 2 * cap), 1, cap};
        p += 3 * cap;
        acc = p;
        p += cap;
        row_val = p;
        p += cap + 1;
        row_col = reinterpret_cast<int *>(p);
        p += cap + 1;
        nb_id = reinterpret_cast<int *>(p);  // 2 cap ints
        p += cap;
        const int pc = cap + 4;
        piece = PolyView<double>{p, p + pc, reinterpret_cast<int *>(p + 2 * pc), 1, pc};
    }
};
// doubles of one warp's scratch: cell (3 cap), acc (cap), row values (cap + 1),
// row columns (cap + 1), ids (2 cap ints), a pixel's piece (3 (cap + 4))
__host__ __device__ constexpr long long warp_scratch_doubles(int cap) {
    return (5LL * cap + 2LL * (cap + 1) + 3LL * (cap + 4) + 31) / 32 * 32;
}

// Copies a finished row from scratch to its ELL slot or the side buffer.
__device__ bool commit(const Rows &R, long long s, const int *col, const double *val, long long st, int cnt) {
    if (cnt <= R.cap) {
        for (int k = 0; k < cnt; ++k) {
            R.col[k * R.stride + s] = col[k * st];
            if (R.val) R.val[k * R.stride + s] = val[k * st];
        }
    } else {
        const unsigned long long off = atomicAdd(R.side_used, (unsigned long long)cnt);
        if ((long long)(off + cnt) > R.side_cap) return false;  // the caller flags DE_SIDE
        R.side[s] = (long long)off;
        for (int k = 0; k < cnt; ++k) {
            R.side_col[off + k] = col[k * st];
            if (R.side_val) R.side_val[off + k] = val[k * st];
        }
    }
    R.cnt[s] = cnt;
    return true;
}

// The polygon of a warp's cell: contiguous, in coordinates about the Dirac.
struct RelView {
    PolyView<double> p;
    double c0x, c0y;
    int cap;
    __device__ RelView(const PolyView<double> &q, double x, double y) : p(q), c0x(x), c0y(y), cap(q.cap) {}
    __device__ double X(int k) const { return c0x + p.X(k); }
    __device__ double Y(int k) const { return c0y + p.Y(k); }
    __device__ int I(int k) const { return p.I(k); }
};
__device__ double rel_x(const RelView &cell, int k, double) { return cell.p.X(k); }
__device__ double rel_y(const RelView &cell, int k, double) { return cell.p.Y(k); }

// Warp-per-cell build of one cell (all lanes, same s): the walk of build_cell.
// A popped box and a cut have the vertices spread over the lanes; when a box is
// opened each of its children, and in a leaf each Dirac, is first tried by a
// lane of its own against every vertex (polygons of at most 64), and only the
// children that are needed now and the Diracs that cut go on, in their order:
// most do not, and one after the other each waited for its reads.
template <bool PER = false>
__device__ int build_cell_warp(const Cell2DArgs &A, long long s, const PolyView<double> &cell, int cap, double c0x,
                               double c0y, double w0, int *wstack) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int n = A.start_n;
    for (int k = lane; k < n; k += 32) {
        cell.X(k) = A.start_xy[2 * k] - c0x;
        cell.Y(k) = A.start_xy[2 * k + 1] - c0y;
        cell.I(k) = domain_id(k);
    }
    __syncwarp();
    int visits = 0;
    // PER: one walk of the tree per translation after the untranslated one
    // (see build_cell)
    for (int sym = -1; sym < (PER ? A.ntrans : 0); ++sym) {
        const double tx = sym >= 0 ? A.trans[2 * sym] : 0.0, ty = sym >= 0 ? A.trans[2 * sym + 1] : 0.0;
        // the box of a node about the Dirac, and whether vertex k needs it
        struct Box {
            double lo0, lo1, hi0, hi1, maxw;
        };
        auto box_of = [&](const TreeNode<2> &nd) {
            return Box{(PER ? nd.lo[0] + tx : nd.lo[0]) - c0x, (PER ? nd.lo[1] + ty : nd.lo[1]) - c0y,
                       (PER ? nd.hi[0] + tx : nd.hi[0]) - c0x, (PER ? nd.hi[1] + ty : nd.hi[1]) - c0y, nd.maxw};
        };
        auto fails = [&](const Box &b, int k) {
            const double px = cell.X(k), py = cell.Y(k);
            const double gx = gap(b.lo0, b.hi0, px), gy = gap(b.lo1, b.hi1, py);
            return !(px * px + py * py - w0 <= gx * gx + gy * gy - b.maxw);
        };
        if (lane == 0) wstack[0] = 0;
        __syncwarp();
        int sp = 1;
        for (; sp > 0; ++visits) {
            if (visits > (PER ? (A.ntrans + 1) * A.max_nodes : A.max_nodes)) {
                if (lane == 0) flag_error(A.err, DE_ITER);
                return -1;
            }
            const int node = wstack[--sp];
            __syncwarp();
            const TreeNode<2> nd = A.nodes[SDOT_CHECK_IDX(node, A.max_nodes, 4)];
            const Box box = box_of(nd);
            bool need = false;
            for (int base = 0; base < n && !need; base += 32)
                need = __any_sync(FULL, base + lane < n && fails(box, base + lane));
            if (!need) continue;
            if (nd.b < 0) {
                const int first = nd.a, nch = -nd.b;
                if (nch < 2 || nch > 4 || first < 1 || first + nch > A.max_nodes) {
                    if (lane == 0) guard_fail(A, 1, s, node);
                    return -2;
                }
                if (sp + nch > STACK) {
                    if (lane == 0) flag_error(A.err, DE_STACK);
                    return -1;
                }
                float key = -1;
                bool keep = false;
                if (lane < nch) {
                    const TreeNode<2> &cn = A.nodes[first + lane];
                    const double cx = 0.5 * (cn.lo[0] + cn.hi[0]), cy = 0.5 * (cn.lo[1] + cn.hi[1]);
                    const double mx = c0x - (PER ? cx + tx : cx), my = c0y - (PER ? cy + ty : cy);
                    key = float(mx * mx + my * my);
                    const Box b = box_of(cn);
                    keep = n > 64;
                    for (int k = 0; k < n && !keep; ++k) keep = fails(b, k);
                }
                // farthest first (nearest popped first)
                const unsigned km = __ballot_sync(FULL, keep);
                int rank = 0;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float kc = __shfl_sync(FULL, key, c);
                    rank += (km >> c & 1u) && (kc > key || (kc == key && c < lane));
                }
                if (keep) wstack[sp + rank] = first + lane;
                sp += __popc(km);
                __syncwarp();
            } else {
                if (nd.a < 0 || nd.b > A.n) {
                    if (lane == 0) guard_fail(A, 2, s, node);
                    return -2;
                }
                for (int j0 = nd.a; j0 < nd.b; j0 += 32) {
                    // lane: Dirac j0 + lane, its bisector relative to c0
                    const int j = j0 + lane;
                    double ox = 0, oy = 0, nx = 0, ny = 0;
                    bool cuts = false;
                    if (j < nd.b && !(j == s && sym < 0)) {
                        const double2 p = reinterpret_cast<const double2 *>(A.pos)[j];
                        bisector(0.0, 0.0, w0, (PER ? p.x + tx : p.x) - c0x, (PER ? p.y + ty : p.y) - c0y, A.w[j], ox, oy,
                                 nx, ny);
                        cuts = n > 64;
                        for (int k = 0; k < n && !cuts; ++k)
                            cuts = (ox - cell.X(k)) * nx + (oy - cell.Y(k)) * ny < 0.0;
                    }
                    for (unsigned cm = __ballot_sync(FULL, cuts); cm; cm &= cm - 1) {
                        const int l = __ffs(int(cm)) - 1;
                        n = plane_cut_warp(cell, n, cap, __shfl_sync(FULL, ox, l), __shfl_sync(FULL, oy, l),
                                           __shfl_sync(FULL, nx, l), __shfl_sync(FULL, ny, l),
                                           PER ? j0 + l + (sym + 1) * int(A.n) : j0 + l);
                        if (n <= 0) return n;
                    }
                }
            }
        }
    }
    return n;
}

// finish_cell by a warp (single shapes without the disc clip): the lanes take
// the edges.  Returns 0, 1 (a capacity was exceeded) or 2 (no room for the row).
__device__ int finish_warp(const Cell2DArgs &A, long long s, const PolyView<double> &cell, int n) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const double c0x = A.pos[2 * s], c0y = A.pos[2 * s + 1];
    if (n == -1) return 1;
    const bool failed = n < 0;  // a failed guard: a NaN cell, not an overflow
    if (failed) n = 0;
    // a neighbour, or the image of Dirac j under translation k for an id j + (k + 1) n
    auto site = [&](int id, int &j, double &x, double &y) {
        const int k = int(id / A.n) - 1;
        j = int(id % A.n);
        x = A.pos[2 * j] + (k >= 0 ? A.trans[2 * k] : 0.0);
        y = A.pos[2 * j + 1] + (k >= 0 ? A.trans[2 * k + 1] : 0.0);
    };
    int nrow = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int id = k0 + lane < n ? cell.I(k0 + lane) : -1;
        int j;
        double x = c0x, y = c0y;
        if (id >= 0) site(id, j, x, y);
        const double dx = c0x - x, dy = c0y - y;
        nrow += __popc(__ballot_sync(FULL, sqrt(dx * dx + dy * dy) != 0));
    }
    RowPut row(A.rows, s, nrow + 1), nb(A.nb, s, n);
    if (!row.ok || !nb.ok) return 2;
    double tr2 = 0, mx = 0, my = 0, mass = 0, der0 = 0;
    const double ax = n > 0 ? cell.X(0) : 0, ay = n > 0 ? cell.Y(0) : 0;
    int at = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        bool entry = false;
        int j = 0;
        double v = 0;
        if (k < n) {
            const int k1 = k + 1 < n ? k + 1 : 0, id = cell.I(k);
            const double bx = cell.X(k), by = cell.Y(k), cx = cell.X(k1), cy = cell.Y(k1);
            if (id >= 0) {
                double x, y;
                site(id, j, x, y);
                const double dx = c0x - x, dy = c0y - y, dist = sqrt(dx * dx + dy * dy);
                entry = dist != 0;
                v = entry ? 0.5 * (A.coeff * sqrt((cx - bx) * (cx - bx) + (cy - by) * (cy - by))) / dist : 0.0;
                der0 += v;
            }
            nb.put(k, id, 0.0);
            if (k >= 1 && k1) {  // triangle (0, k, k + 1)
                const double t2 = ax * (by - cy) + bx * (cy - ay) + cx * (ay - by);
                tr2 += t2;
                const double lea = 0.5 * t2 * A.coeff;
                mx += (1.0 / 3.0) * lea * (ax + bx + cx);
                my += (1.0 / 3.0) * lea * (ay + by + cy);
                mass += lea;
            }
        }
        const unsigned em = __ballot_sync(FULL, entry);
        if (entry) row.put(at + __popc(em & ((1u << lane) - 1u)), j, -v);
        at += __popc(em);
    }
    for (int o = 16; o > 0; o >>= 1) {
        tr2 += __shfl_xor_sync(FULL, tr2, o);
        mx += __shfl_xor_sync(FULL, mx, o);
        my += __shfl_xor_sync(FULL, my, o);
        mass += __shfl_xor_sync(FULL, mass, o);
        der0 += __shfl_xor_sync(FULL, der0, o);
    }
    if (lane == 0) {
        row.put(at, int(s), der0);
        row.cnt = at + 1;
        row.finish();
        nb.finish();
        const double none = nan("");
        if (A.mass) A.mass[s] = failed ? none : A.coeff * (tr2 * 0.5);
        if (A.mass_c) A.mass_c[s] = failed ? none : mass;
        if (A.ctd) {
            const double d = mass + (mass == 0);
            A.ctd[2 * s] = failed ? none : (mx + c0x * mass) / d;
            A.ctd[2 * s + 1] = failed ? none : (my + c0y * mass) / d;
        }
    }
    return 0;
}

// Cells that overflowed the fast tier, one warp per cell: polygons of up to
// CAP vertices in shared memory (MID), or in global scratch for those that
// overflow that too.  The warp integrates a cell of a single shape; the disc
// clip and the image and raster modes are done by lane 0.
// 60,000 clustered Diracs: 8,700 cells pass 13 vertices while they are built (23
// at most at their end).  With every polygon in global scratch, lane 0
// integrating and one Dirac at a time, the cells took 3.1 ms at the starting
// weights and 7.7 ms at the solved ones, then 1.4 and 3.8 ms; with one warp a
// block, more of them and a cursor in place of fixed shares 3.5 ms at the solved
// ones (the longest walks last: a cell takes up to a millisecond).
template <int MODE, bool BALL, bool MID>
__global__ void __launch_bounds__(32, !MID ? 4 : BALL || (MODE != DM_SINGLE && MODE != DM_PERIODIC) ? 16 : MID_BLOCKS)
    k_cells2d_wtier(const Cell2DArgs A, double *scratch, const int *list, const int *list_cnt, int *cursor,
                    int *next_list, int *next_cnt) {
    constexpr int CAP = MID ? CAP_MID_2D : CAP_HUGE_2D;
    extern __shared__ double wmem[];
    __shared__ int wstack[STACK];
    const int lane = threadIdx.x;
    WarpScratch W(MID ? wmem : scratch + (long long)blockIdx.x * warp_scratch_doubles(CAP), CAP);
    const int cnt = list ? *list_cnt : int(A.n);
    // the first cells by block, the others as blocks come free
    auto fetch = [&] {
        int k = 0;
        if (lane == 0) k = atomicAdd(cursor, 1);
        return int(gridDim.x) + __shfl_sync(0xffffffffu, k, 0);
    };
    for (int i = blockIdx.x; i < cnt; i = fetch()) {
        const long long s = list ? list[i] : i;
        const double c0x = A.pos[2 * s], c0y = A.pos[2 * s + 1];
        const int n = build_cell_warp<MODE == DM_PERIODIC>(A, s, W.cell, CAP, c0x, c0y, A.w[s], wstack);
        int failed = 0;  // 1: a capacity was exceeded, 2: no room for the row
        if constexpr ((MODE == DM_SINGLE || MODE == DM_PERIODIC) && !BALL) {
            failed = finish_warp(A, s, W.cell, n);
        } else if (lane == 0) {
            Out row(A.rows.cnt ? W.row_col : nullptr, W.row_val, 1, CAP + 1);
            Out nbo(A.nb.cnt ? W.nb_id : nullptr, nullptr, 1, 2 * CAP);
            if (!finish_cell<MODE, BALL>(A, s, RelView(W.cell, c0x, c0y), n, W.acc, 1, row, nbo, W.piece)) failed = 1;
            if (!failed && A.rows.cnt && !commit(A.rows, s, W.row_col, W.row_val, 1, row.cnt)) failed = 2;
            if (!failed && A.nb.cnt && !commit(A.nb, s, W.nb_id, nullptr, 1, nbo.cnt)) failed = 2;
        }
        if (lane == 0 && failed) {
            if (MID && failed == 1) {
                const int k = atomicAdd(next_cnt, 1);
                if (k < A.n) next_list[k] = int(s);  // as push_overflow
            } else {
                atomicOr(A.err, failed == 2 ? DE_SIDE : DE_CAPACITY);
                if (A.mass) A.mass[s] = nan("");
                if (A.rows.cnt) A.rows.cnt[s] = 0;
                if (A.nb.cnt) A.nb.cnt[s] = 0;
            }
        }
        __syncwarp();
    }
}

// Every cell into the warp tier's list (domain polygons larger than the fast
// tier's polygons).
__global__ void k_all_cells(int *list, int *cnt, long long n) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s < n) list[s] = int(s);
    if (s == 0) *cnt = int(n);
}

// Counters the fast kernel appends to: zeroed before every launch of it.
void reset_overflow(const Cell2DArgs &a, cudaStream_t st) {
    SDOT_CUDA(cudaMemsetAsync(a.ovf_cnt, 0, sizeof(int), st));
    SDOT_CUDA(cudaMemsetAsync(a.ovf_cnt2, 0, 3 * sizeof(int), st));  // and the cursors
    if (a.rows.side_used) SDOT_CUDA(cudaMemsetAsync(a.rows.side_used, 0, sizeof(unsigned long long), st));
    if (a.nb.side_used) SDOT_CUDA(cudaMemsetAsync(a.nb.side_used, 0, sizeof(unsigned long long), st));
}

// Up to this many Diracs a cell gets a warp from the start (single shapes
// without the disc clip, whose cells a warp integrates): the walk of one thread
// takes 100 to 200 us whatever their number.  Cells of 1,000 / 3,000 / 10,000
// uniform Diracs: 150 / 190 / 203 us by threads, 62 / 94 / 199 us by warps (whose
// 15 ns per cell lose to 2 ns beyond).
constexpr long long WARP_CELLS = 6000;
// Cells per warp of the fast tier: where there are too few warps to fill the
// device, fewer cells per warp end sooner (10,000 Diracs: 201 -> 182 us with 12;
// 30,000: 283 -> 291).
int warp_lanes(long long n) { return n <= 16384 ? 12 : 32; }

template <int MODE, bool BALL>
void launch_all(const Cell2DArgs &a, void *scratch, cudaStream_t st) {
    static PerDevice<int> attr_set;
    attr_set.once([] {
        // room for the twelve blocks per SM that the registers allow (2%
        // faster than 72%, which holds ten)
        SDOT_CUDA(cudaFuncSetAttribute(k_cells2d<MODE, BALL>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    });
    reset_overflow(a, st);
    constexpr bool BY_WARP = (MODE == DM_SINGLE || MODE == DM_PERIODIC) && !BALL;
    const int *list = a.ovf_list, *cnt = a.ovf_cnt;
    if (BY_WARP && a.start_n <= CAP_FAST_2D && a.n <= WARP_CELLS) {
        list = cnt = nullptr;  // every cell
    } else if (a.start_n <= CAP_FAST_2D) {
        Cell2DArgs b = a;
        b.lanes = warp_lanes(a.n);
        k_cells2d<MODE, BALL><<<ceil_div(ceil_div(a.n, b.lanes), BS / 32), BS, fast_smem<MODE>(), st>>>(b);
        note_launch();
    } else {
        // the starting polygon alone overflows the fast tier
        k_all_cells<<<ceil_div(a.n, 256), 256, 0, st>>>(a.ovf_list, a.ovf_cnt, a.n);
        note_launch();
    }
    // a starting polygon that nearly fills the warps' shared memory goes on to
    // the last tier at once
    const bool mid = a.start_n <= CAP_MID_2D - 16;
    if (mid) {
        k_cells2d_wtier<MODE, BALL, true><<<MID_WARPS, 32, warp_scratch_doubles(CAP_MID_2D) * sizeof(double), st>>>(
            a, nullptr, list, cnt, a.ovf_cnt2 + 1, a.ovf_list2, a.ovf_cnt2);
        note_launch();
    }
    k_cells2d_wtier<MODE, BALL, false><<<WTIER_WARPS, 32, 0, st>>>(
        a, static_cast<double *>(scratch), mid ? a.ovf_list2 : a.ovf_list, mid ? a.ovf_cnt2 : a.ovf_cnt, a.ovf_cnt2 + 2,
        nullptr, nullptr);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

}  // namespace

void cells2d_read_checks(unsigned long long out[3]) {
#ifdef SDOT_CHECKS
    SDOT_CUDA(cudaMemcpyFromSymbol(out, sdot_dbg_word, 3 * sizeof(unsigned long long)));
#else
    out[0] = out[1] = out[2] = 0;
#endif
}

void cells2d_read_work(unsigned long long out[8], bool reset) {
#ifdef SDOT_COUNT
    SDOT_CUDA(cudaMemcpyFromSymbol(out, sdot_work, 8 * sizeof(unsigned long long)));
    if (reset) {
        const unsigned long long z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        SDOT_CUDA(cudaMemcpyToSymbol(sdot_work, z, sizeof z));
    }
#else
    (void)reset;
    for (int k = 0; k < 8; ++k) out[k] = 0;
#endif
}

size_t cells2d_scratch_bytes() {
    return size_t(warp_scratch_doubles(CAP_HUGE_2D)) * WTIER_WARPS * sizeof(double) + 256;
}

void cells2d_launch(const Cell2DArgs &a, void *scratch, cudaStream_t st) {
    if (a.n == 0) return;
    const bool ball = a.ball != 0;
    if (a.mode == DM_SINGLE) {
        if (ball) launch_all<DM_SINGLE, true>(a, scratch, st); else launch_all<DM_SINGLE, false>(a, scratch, st);
    } else if (a.mode == DM_PERIODIC) {
        if (ball) launch_all<DM_PERIODIC, true>(a, scratch, st); else launch_all<DM_PERIODIC, false>(a, scratch, st);
    } else if (a.mode == DM_IMAGE) {
        if (ball) launch_all<DM_IMAGE, true>(a, scratch, st); else launch_all<DM_IMAGE, false>(a, scratch, st);
    } else if (a.mode == DM_RASTER) {
        if (ball) launch_all<DM_RASTER, true>(a, scratch, st); else launch_all<DM_RASTER, false>(a, scratch, st);
    } else if (a.mode == DM_IMAGE6) {
        // the reference integrates no piecewise-quadratic density over disc arcs
        if (ball) throw CudaError{cudaErrorInvalidValue, "cells2d_launch: no disc clip with nb_coeffs = 6"};
        launch_all<DM_IMAGE6, false>(a, scratch, st);
    } else {
        throw CudaError{cudaErrorInvalidValue, "cells2d_launch: a domain of several shapes runs one pass per shape"};
    }
}

}  // namespace sdot
