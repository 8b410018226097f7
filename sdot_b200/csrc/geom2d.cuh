// 2D convex-polygon geometry shared by the cell kernels (device) and the
// host-side domain builder.  Polygons are counter-clockwise vertex lists; the
// edge leaving vertex k carries id[k] (see common.cuh for id meanings).
//
// plane_cut restates ConvexPolyhedron2::plane_cut (reference
// src/sdot/Geometry/ConvexPolyhedron2.tcc:687-924) including its index
// bookkeeping (where the two new vertices land, and the rotation when the
// removed run wraps over vertex 0), so that a cell built from the same cut
// sequence has the same vertex order, hence the same fan triangulation.
#pragma once
#include "common.cuh"
#include <cmath>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace sdot {

#define SDOT_HD __host__ __device__ __forceinline__
#define SDOT_HDI __host__ __device__

constexpr double kPi = 3.141592653589793238462643383279502884;

// Vertex storage with an element stride (SoA in shared or global memory).
template <class T>
struct PolyView {
    T *x;
    T *y;
    int *id;
    int st;
    int cap = 1 << 30;  // vertex slots (bound of the debug checks)
    SDOT_HDI T &X(int k) const { return x[SDOT_CHECK_IDX(k, cap, 1) * st]; }
    SDOT_HDI T &Y(int k) const { return y[SDOT_CHECK_IDX(k, cap, 1) * st]; }
    SDOT_HDI int &I(int k) const { return id[SDOT_CHECK_IDX(k, cap, 1) * st]; }
    SDOT_HDI void copy(int dst, int src) const {
        X(dst) = X(src);
        Y(dst) = Y(src);
        I(dst) = I(src);
    }
};

// Cut the polygon (n vertices, capacity cap) by the half-plane
// {p : (o - p) . nrm >= 0}; the new edge gets `cut_id`.  The reference
// divides its distances by |nrm| for un-normalised normals (N<0>); the
// interpolation ratios are the same without it.
// Returns the new vertex count, or -1 if the result would exceed `cap`.
// The facts read from the vertices' sides: how many are outside, the first one
// outside, the first one inside, and the last one's side.
struct CutFacts {
    int nb_out = 0, first_out = -1, first_in = -1;
    bool out_last = false;
    SDOT_HD void add(int k, int n, bool o) {
        nb_out += o;
        if (o && first_out < 0) first_out = k;
        if (!o && first_in < 0) first_in = k;
        if (k == n - 1) out_last = o;
    }
};

SDOT_HD int popcount(unsigned v) {
#ifdef __CUDA_ARCH__
    return __popc(v);
#else
    return __builtin_popcount(v);
#endif
}
// The place of the lowest bit set (-1: none).
SDOT_HD int first_bit(unsigned v) {
#ifdef __CUDA_ARCH__
    return __ffs(int(v)) - 1;
#else
    return __builtin_ffs(int(v)) - 1;
#endif
}

// The same facts from a bit mask of the outside vertices (bit k: vertex k;
// polygons of at most 32 vertices).
SDOT_HD CutFacts cut_facts(unsigned mask, int n) {
    CutFacts f;
    const unsigned valid = n >= 32 ? 0xffffffffu : ((1u << n) - 1u);
    const unsigned in = ~mask & valid;
    f.nb_out = popcount(mask);
    f.first_out = first_bit(mask);
    f.first_in = first_bit(in);
    f.out_last = (mask >> (n - 1)) & 1u;
    return f;
}

// The run [i1, i1 + gone) (cyclic) of vertices with d(k) < 0 that holds the
// lowest, for a polygon with some such vertices and some others.  A convex
// polygon has one run but for rounding: where several vertices lie at one place
// (the corners of a lattice's cells), others may be outside by an ulp here and
// there, and the run of the farthest is the one that a cut removes.
template <class D>
SDOT_HDI void farthest_run(int n, const D &d, int &i1, int &gone) {
    double low = 0;
    i1 = 0;
    for (int k = 0; k < n; ++k) {
        const double v = d(k);
        if (v < low) {
            low = v;
            i1 = k;
        }
    }
    gone = 1;
    while (gone < n && d(i1 == 0 ? n - 1 : i1 - 1) < 0) {
        i1 = i1 == 0 ? n - 1 : i1 - 1;
        ++gone;
    }
    while (gone < n && d((i1 + gone) % n) < 0) ++gone;
}

template <class T>
SDOT_HD int plane_cut_apply(const PolyView<T> &p, int n, int cap, T ox, T oy, T nx, T ny, int cut_id,
                            const CutFacts &f);

template <class T>
SDOT_HD int plane_cut(const PolyView<T> &p, int n, int cap, T ox, T oy, T nx, T ny, int cut_id) {
    CutFacts f;
    for (int k = 0; k < n; ++k) {
        const T d = (ox - p.X(k)) * nx + (oy - p.Y(k)) * ny;
        f.add(k, n, d < T(0));
    }
    return plane_cut_apply(p, n, cap, ox, oy, nx, ny, cut_id, f);
}

// The cut itself, given the classification of the vertices.  The new
// vertices sit at the ratios s_a / (s_b - s_a) of the signed distances along
// their edges; the ratios do not depend on the scale of the normal, so the
// distances are left unnormalised, and both ratios come from one division
// (1 / (u v), u and v the two distance differences: products of coordinates, far
// from underflow).
template <class T>
SDOT_HD int plane_cut_apply(const PolyView<T> &p, int n, int cap, T ox, T oy, T nx, T ny, int cut_id,
                            const CutFacts &f) {
    const int nb_out = f.nb_out, first_out = f.first_out, first_in = f.first_in;
    const bool out_last = f.out_last;
    if (nb_out == 0) return n;
    if (nb_out == n) return 0;
    auto dist = [&](int k) -> T { return (ox - p.X(k)) * nx + (oy - p.Y(k)) * ny; };
    // the two edge ratios a / (b - a), c / (d - c)
    auto ratios = [](T a, T b, T c, T d, T &m1, T &m2) {
        const T u = b - a, v = d - c, r = T(1) / (u * v);
        m1 = a * v * r;
        m2 = c * u * r;
    };

    // One layout for every case.  The removed run is [i1, i2] (cyclic), the
    // kept run [i3, i0]; A (on edge i0 -> i1) takes the cut's id, B (on edge
    // i2 -> i3) the id of that edge.  Without wrap (the run does not hold
    // both vertex n - 1 and vertex 0): A at i1, B at i1 + 1, the kept tail
    // [i3, n) shifted by 2 - nb_out.  With wrap: B at 0, the kept run moved
    // to [1, nb_in], A after it.  These are the positions of the reference's
    // four cases (one vertex out, two, a wrapping run, a longer run).
    const int nb_in = n - nb_out;
    if (nb_out == 1 && n + 1 > cap) return -1;
    const bool wrap = out_last && first_out == 0;  // nb_out >= 2 here, as nb_out == 1 cannot be both
    const int i3 = wrap ? first_in : first_out + nb_out;  // may be n: vertex 0
    const int i1 = wrap ? first_in + nb_in : first_out;
    const int i0 = i1 == 0 ? n - 1 : i1 - 1;
    const int i2 = i3 == 0 ? n - 1 : i3 - 1;
    const int i3c = i3 == n ? 0 : i3;
    T p0x = p.X(i0), p0y = p.Y(i0), p1x = p.X(i1), p1y = p.Y(i1);
    T p2x = p.X(i2), p2y = p.Y(i2), p3x = p.X(i3c), p3y = p.Y(i3c);
    T s0 = dist(i0), s1 = dist(i1), s2 = dist(i2), s3 = dist(i3c);
    T m1, m2;
    ratios(s0, s1, s3, s2, m1, m2);
    const T ax = p0x - m1 * (p1x - p0x), ay = p0y - m1 * (p1y - p0y);
    const T bx = p3x - m2 * (p2x - p3x), by = p3y - m2 * (p2y - p3y);
    const int id2 = p.I(i2);
    if (wrap) {
        for (int k = 0; k < nb_in; ++k) p.copy(1 + k, i3 + k);
        p.X(0) = bx;
        p.Y(0) = by;
        p.I(0) = id2;
        p.X(nb_in + 1) = ax;
        p.Y(nb_in + 1) = ay;
        p.I(nb_in + 1) = cut_id;
    } else {
        if (nb_out == 1) {
            for (int i = n - 1; i >= i3; --i) p.copy(i + 1, i);
        } else {
            for (int i = i3; i < n; ++i) p.copy(i + 2 - nb_out, i);
        }
        p.X(i1) = ax;
        p.Y(i1) = ay;
        p.I(i1) = cut_id;
        p.X(i1 + 1) = bx;
        p.Y(i1 + 1) = by;
        p.I(i1 + 1) = id2;
    }
    return nb_in + 2;
}

#ifdef __CUDACC__
// plane_cut done by a whole warp on one polygon (all 32 lanes call it with the
// same arguments): the lanes classify 32 vertices at a time, the facts the
// scalar version gathers in its pass come from warp votes, and vertex moves
// are done 32 at a time, each chunk read before it is written, in the order
// that keeps the scalar loop's result.  Same cases, same new vertices, same
// vertex order as plane_cut.
template <class T>
__device__ int plane_cut_warp(const PolyView<T> &p, int n, int cap, T ox, T oy, T nx, T ny, int cut_id) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int nb_out = 0, first_out = -1, first_in = -1, runs = 0;
    bool out1 = false, out_last = false;
    auto dist = [&](int k) -> T { return (ox - p.X(k)) * nx + (oy - p.Y(k)) * ny; };
    for (int base = 0; base < n; base += 32) {
        const int k = base + lane;
        const bool valid = k < n;
        const bool o = valid && dist(k) < T(0);
        const unsigned mo = __ballot_sync(FULL, o), mi = __ballot_sync(FULL, valid && !o);
        nb_out += __popc(mo);
        runs += __popc(mo & ~(mo << 1 | unsigned(out_last)));  // out_last: of the vertices before
        out_last = mo >> 31;
        if (first_out < 0 && mo) first_out = base + __ffs(mo) - 1;
        if (first_in < 0 && mi) first_in = base + __ffs(mi) - 1;
        if (base == 0 && n > 1) out1 = (mo >> 1) & 1u;
        if (n - 1 < base + 32) out_last = (mo >> (n - 1 - base)) & 1u;
    }
    if (nb_out == 0) return n;
    if (nb_out == n) return 0;
    if (runs - (out_last && first_out == 0) > 1) {
        // (every lane alike; rare)
        int a, g;
        farthest_run(n, dist, a, g);
        nb_out = g;
        const bool wrap = a + g > n;
        first_out = wrap ? 0 : a;
        first_in = wrap ? a + g - n : a == 0 ? g : 0;
        out1 = wrap ? a + g - n > 1 || a == 1 : a <= 1 && a + g > 1;
        out_last = a + g >= n;
    }
    int i1 = first_out;
    if (nb_out == 1) {
        if (n + 1 > cap) return -1;
        const int i0 = (i1 + n - 1) % n, i2 = (i1 + 1) % n;
        const T p0x = p.X(i0), p0y = p.Y(i0), p1x = p.X(i1), p1y = p.Y(i1), p2x = p.X(i2), p2y = p.Y(i2);
        const T s0 = dist(i0), s1 = dist(i1), s2 = dist(i2);
        const T m0 = s0 / (s1 - s0), m1 = s2 / (s1 - s2);
        const int id1 = p.I(i1);
        __syncwarp();
        for (int hi = n; hi > i1 + 1; hi -= 32) {  // [i1 + 1, n) moves up by one, top chunk first
            const int lo = hi - 32 > i1 + 1 ? hi - 32 : i1 + 1;
            const int k = lo + lane;
            T vx = T(0), vy = T(0);
            int vi = 0;
            if (k < hi) {
                vx = p.X(k);
                vy = p.Y(k);
                vi = p.I(k);
            }
            __syncwarp();
            if (k < hi) {
                p.X(k + 1) = vx;
                p.Y(k + 1) = vy;
                p.I(k + 1) = vi;
            }
            __syncwarp();
        }
        if (lane == 0) {
            p.X(i1 + 1) = p2x - m1 * (p1x - p2x);
            p.Y(i1 + 1) = p2y - m1 * (p1y - p2y);
            p.I(i1 + 1) = id1;
            p.X(i1) = p0x - m0 * (p1x - p0x);
            p.Y(i1) = p0y - m0 * (p1y - p0y);
            p.I(i1) = cut_id;
        }
        __syncwarp();
        return n + 1;
    }
    if (nb_out == 2) {
        if (i1 == 0 && !out1) i1 = n - 1;
        const int i0 = (i1 + n - 1) % n, i2 = (i1 + 1) % n, i3 = (i1 + 2) % n;
        const T p0x = p.X(i0), p0y = p.Y(i0), p1x = p.X(i1), p1y = p.Y(i1);
        const T p2x = p.X(i2), p2y = p.Y(i2), p3x = p.X(i3), p3y = p.Y(i3);
        const T s0 = dist(i0), s1 = dist(i1), s2 = dist(i2), s3 = dist(i3);
        const T m1 = s0 / (s1 - s0), m2 = s3 / (s2 - s3);
        __syncwarp();
        if (lane == 0) {
            p.X(i1) = p0x - m1 * (p1x - p0x);
            p.Y(i1) = p0y - m1 * (p1y - p0y);
            p.I(i1) = cut_id;
            p.X(i2) = p3x - m2 * (p2x - p3x);
            p.Y(i2) = p3y - m2 * (p2y - p3y);
        }
        __syncwarp();
        return n;
    }
    // left move of [src0, src0 + cnt) to [src0 - by, ...), low chunk first
    auto move_down = [&](int src0, int cnt, int by) {
        for (int c = 0; c < cnt; c += 32) {
            const int k = src0 + c + lane;
            const bool v = c + lane < cnt;
            T vx = T(0), vy = T(0);
            int vi = 0;
            if (v) {
                vx = p.X(k);
                vy = p.Y(k);
                vi = p.I(k);
            }
            __syncwarp();
            if (v) {
                p.X(k - by) = vx;
                p.Y(k - by) = vy;
                p.I(k - by) = vi;
            }
            __syncwarp();
        }
    };
    if (i1 == 0 && out_last) {
        const int nb_in = n - nb_out;
        const int i3 = first_in;
        i1 = nb_in + i3;
        const int i0 = i1 - 1, i2 = i3 - 1;
        const T p0x = p.X(i0), p0y = p.Y(i0), p1x = p.X(i1), p1y = p.Y(i1);
        const T p2x = p.X(i2), p2y = p.Y(i2), p3x = p.X(i3), p3y = p.Y(i3);
        const T s0 = dist(i0), s1 = dist(i1), s2 = dist(i2), s3 = dist(i3);
        const T m1 = s0 / (s1 - s0), m2 = s3 / (s2 - s3);
        const int id2 = p.I(i2);
        __syncwarp();
        if (lane == 0) {
            p.X(0) = p3x - m2 * (p2x - p3x);
            p.Y(0) = p3y - m2 * (p2y - p3y);
            p.I(0) = id2;
        }
        __syncwarp();
        if (i2 > 0) move_down(i2 + 1, nb_in, i2);
        if (lane == 0) {
            p.X(nb_in + 1) = p0x - m1 * (p1x - p0x);
            p.Y(nb_in + 1) = p0y - m1 * (p1y - p0y);
            p.I(nb_in + 1) = cut_id;
        }
        __syncwarp();
        return nb_in + 2;
    }
    const int i0 = (i1 + n - 1) % n, i2 = (i1 + nb_out - 1) % n, i3 = (i1 + nb_out) % n;
    const T p0x = p.X(i0), p0y = p.Y(i0), p1x = p.X(i1), p1y = p.Y(i1);
    const T p2x = p.X(i2), p2y = p.Y(i2), p3x = p.X(i3), p3y = p.Y(i3);
    const T s0 = dist(i0), s1 = dist(i1), s2 = dist(i2), s3 = dist(i3);
    const T m1 = s0 / (s1 - s0), m2 = s3 / (s2 - s3);
    const int id2 = p.I(i2);
    __syncwarp();
    if (lane == 0) {
        p.X(i1) = p0x - m1 * (p1x - p0x);
        p.Y(i1) = p0y - m1 * (p1y - p0y);
        p.I(i1) = cut_id;
        p.X(i1 + 1) = p3x - m2 * (p2x - p3x);
        p.Y(i1 + 1) = p3y - m2 * (p2y - p3y);
        p.I(i1 + 1) = id2;
    }
    __syncwarp();
    const int nb_rem = nb_out - 2;
    if (i2 + 1 < n) move_down(i2 + 1, n - i2 - 1, nb_rem);
    return n - nb_rem;
}
#endif

// Weighted bisector of (c0, w0) and (c1, w1) as the reference's traversal
// builds it (src/sdot/PowerDiagram/Visitors/SpZGrid.tcc:506-522): origin
// c0 + x V, normal V = c1 - c0, x = 1/2 + 1/2 (w0 - w1) / |V|^2.
template <class T>
SDOT_HD void bisector(T c0x, T c0y, T w0, T c1x, T c1y, T w1, T &ox, T &oy, T &nx, T &ny) {
    nx = c1x - c0x;
    ny = c1y - c0y;
    T nn = nx * nx + ny * ny;
    T x = T(0.5) + T(0.5) * (w0 - w1) / nn;
    ox = c0x + x * nx;
    oy = c0y + x * ny;
}

// Cuts the polygon q (m vertices) in place to the half-plane s (coord - c) >= 0,
// coord = x if axis == 0 else y; the new edge along the line gets the id `own`.
// Returns the new count: m + 1 at most (there is room for it), or up to `room`
// where that is more.
// A run of vertices outside gives way to two on the line: A on the edge into the
// run, B on the edge out of it.  The run of the farthest vertex goes first.  A
// convex polygon has no other one but for rounding; where a side of the cell lies
// on a pixel's line and its corners are several vertices at one place (a lattice
// of Diracs over an image) there are some more, and each is cut in its turn, so
// that the pixels on both sides of the line share out the side's length.  (Taken
// edge by edge in one pass in place, the third crossing would be written over a
// vertex not read yet.)  A vertex outside by rounding for which there is no room
// stays.
// The vertices keep their order; the polygon starts at its vertex 0 or, where
// that one goes, at the B of its run.
template <class P>
SDOT_HD int axis_cut(const P &q, int m, int axis, double c, double s, int own, int room) {
    auto val = [&](int k) { return s * ((axis == 0 ? q.X(k) : q.Y(k)) - c); };
    for (bool first = true;; first = false) {
        // the run: gone vertices from i1 on (cyclic) of the out outside
        int i1 = -1, gone = 0, out = 0;
        if (m <= 32) {
            unsigned mask = 0;
            for (int k = 0; k < m; ++k) mask |= unsigned(val(k) < 0) << k;
            if (!mask) return m;
            const unsigned starts = mask & ~(mask << 1 | mask >> (m - 1));
            out = popcount(mask);
            if (!starts) return 0;
            if (!(starts & (starts - 1))) {
                i1 = first_bit(starts);
                gone = out;
            }
        }
        if (!gone) {
            out = 0;
            for (int k = 0; k < m; ++k) out += val(k) < 0;
            if (!out) return m;
            if (out == m) return 0;
            farthest_run(m, val, i1, gone);
        }
        // i0 the vertex before the run, [i1, i2] the run, i3 the one after
        const int i0 = i1 == 0 ? m - 1 : i1 - 1, i2 = i1 + gone - 1 < m ? i1 + gone - 1 : i1 + gone - 1 - m;
        const int i3 = i2 + 1 == m ? 0 : i2 + 1;
        const double v0 = val(i0), v1 = val(i1), v2 = val(i2), v3 = val(i3);
        if (gone == 1 && !first && m >= room) return m;
        auto on_line = [&](int k, double vk, int l, double vl, double &x, double &y) {
            const double px = q.X(k), py = q.Y(k), t = vk / (vk - vl);
            x = axis == 0 ? c : px + t * (q.X(l) - px);
            y = axis == 0 ? py + t * (q.Y(l) - py) : c;
        };
        double ax, ay, bx, by;
        on_line(i0, v0, i1, v1, ax, ay);
        on_line(i2, v2, i3, v3, bx, by);
        const int bt = q.I(i2);
        int ia, ib;  // their places
        if (i1 == 0 || i1 > i2) {  // vertex 0 goes: B, the kept run from i3 on, A
            ib = 0;
            ia = m - gone + 1;
            if (i3 > 1)
                for (int k = 1; k < ia; ++k) q.copy(k, i3 + k - 1);
        } else {
            ia = i1;
            ib = i1 + 1;
            if (gone == 1) {
                for (int k = m; k > ib; --k) q.copy(k, k - 1);
            } else if (gone > 2) {
                for (int k = i2 + 1; k < m; ++k) q.copy(k + 2 - gone, k);
            }
        }
        q.X(ia) = ax;
        q.Y(ia) = ay;
        q.I(ia) = own;
        q.X(ib) = bx;
        q.Y(ib) = by;
        q.I(ib) = bt;
        m += 2 - gone;
        if (gone == out) return m;
    }
}

#ifdef __CUDACC__
// Disc clipping restated from ConvexPolyhedron2::ball_cut
// (ConvexPolyhedron2.tcc:534-666): the edge a -> b of a polygon emits 0, 1 or 2
// vertices of the clipped one (x, y, and whether an arc leaves it; else its
// edge is the polygon's).  Returns their number.
struct DiscEdge {
    double x[2], y[2];
    bool arc[2];
};
__device__ __forceinline__ int disc_edge(double ax, double ay, double bx, double by, double cx, double cy, double r,
                                         DiscEdge &e) {
    const double ux = ax - cx, uy = ay - cy, vx = bx - cx, vy = by - cy;
    const double da = ux * ux + uy * uy - r * r, db = vx * vx + vy * vy - r * r;
    e.x[0] = ax;
    e.y[0] = ay;
    e.arc[0] = e.arc[1] = false;
    if (da <= 0 && db <= 0) return 1;
    // the two crossings of the line: a + t (b - a), t = (-h -+ sqrt(h^2 - q c)) / q,
    // taken from the end inside where one is
    const bool from_b = da > 0 && db <= 0;
    const double px = from_b ? bx : ax, py = from_b ? by : ay, dx = from_b ? ax - bx : bx - ax,
                 dy = from_b ? ay - by : by - ay;
    const double q = dx * dx + dy * dy;
    const double h = (px - cx) * dx + (py - cy) * dy;
    const double disc = h * h - q * (from_b ? db : da);
    if (da <= 0 || db <= 0) {  // one crossing
        const double d = sqrt(fmax(0.0, disc));
        const double u = (-h + d) / q, v = (-h - d) / q;
        double t = fabs(u - 0.5) <= fabs(v - 0.5) ? u : v;
        t = fmin(1.0, fmax(0.0, t));
        const int k = from_b ? 0 : 1;
        e.x[k] = px + t * dx;
        e.y[k] = py + t * dy;
        e.arc[1] = true;
        return k + 1;
    }
    if (q == 0 || disc <= 0) return 0;
    const double d = sqrt(disc);
    double u = (-h - d) / q, v = (-h + d) / q;
    if (u > 0 && u < 1)
        v = fmax(0.0, fmin(1.0, v));
    else if (v > 0 && v < 1)
        u = fmax(0.0, fmin(1.0, u));
    else
        return 0;
    e.x[0] = px + u * dx;
    e.y[0] = py + u * dy;
    e.x[1] = px + v * dx;
    e.y[1] = py + v * dy;
    e.arc[1] = true;
    return atan2(e.y[0] - cy, e.x[0] - cx) != atan2(e.y[1] - cy, e.x[1] - cx) ? 2 : 0;
}

// Pushes the vertices of a polygon (m vertices; tag(k): the tag of edge k) to
// sink.push(x, y, tag, closing), with BALL those of its intersection with the
// disc (c, r), arcs tagged ID_ARC; with CLOSE the first one once more at the end
// (closing).  One loop and one call of push, so that it is inlined once.
// Returns the radius of the result as the reference stores it: r, 0 if void;
// -1 without a disc.  A polygon that leaves no vertex is apart from the circle: it
// stands for the full disc where the centre lies inside it, which is where a ray
// from the centre to greater x crosses an odd number of edges.  (Its side of
// every edge says the same, but not of an edge between vertices at one place,
// whose direction is rounding; such an edge lies far from the centre, and on one
// side of it whatever its direction.)
template <bool BALL, bool CLOSE, class P, class Tag, class S>
__device__ __forceinline__ double stream_piece(const P &q, int m, const Tag &tag, double cx, double cy, double r, S &sink) {
    int nout = 0, ft = 0;
    bool inside = false;
    double fx = 0, fy = 0;
    double ax = m > 0 ? q.X(0) : 0, ay = m > 0 ? q.Y(0) : 0;
    const double qx = ax, qy = ay;
    const int turns = m + (CLOSE ? 1 : 0);
#pragma unroll 1
    for (int k = 0; k < turns; ++k) {
        DiscEdge e;
        int cnt = 1, t = ft;
        if (CLOSE && k == m) {
            e.x[0] = fx;
            e.y[0] = fy;
            e.arc[0] = false;
            if (!nout) cnt = 0;
        } else {
            const double bx = k + 1 < m ? q.X(k + 1) : qx, by = k + 1 < m ? q.Y(k + 1) : qy;
            t = tag(k);
            if (BALL) {
                if ((ay > cy) != (by > cy))
                    inside ^= ((bx - ax) * (cy - ay) - (cx - ax) * (by - ay) > 0) == (by > ay);
                cnt = disc_edge(ax, ay, bx, by, cx, cy, r, e);
            } else {
                e.x[0] = ax;
                e.y[0] = ay;
                e.arc[0] = false;
            }
            ax = bx;
            ay = by;
        }
#pragma unroll 1
        for (int o = 0; o < cnt; ++o) {
            const double x = o ? e.x[1] : e.x[0], y = o ? e.y[1] : e.y[0];
            const int g = (o ? e.arc[1] : e.arc[0]) ? ID_ARC : t;
            const bool closing = CLOSE && k == m;
            if (!nout) {
                fx = x;
                fy = y;
                ft = g;
            }
            sink.push(x, y, g, closing);
            ++nout;
        }
    }
    if (!BALL) return -1.0;
    return m == 0 || (nout == 0 && !inside) ? 0.0 : r;
}

// The segment of the disc (c, r) between the chord p0 -> p1 and the arc (area,
// moments about the origin, angle of the arc), restated from
// ConvexPolyhedron2::_arc_area / _centroid_arc / _arc_length
// (ConvexPolyhedron2.tcc:2296-2381), which each take the angles anew.
// Ends that meet to rounding may come in the wrong order (the sides of a sliver,
// an ulp apart, cut by the circle), and the arc would be all but a full turn: it
// is none if the rest is less than 1000 ulp of the coordinates, as seen from the
// centre.  (A chord that leaves an arc of all but a full turn spans 1e-8 at
// least, where its line touches the circle to rounding.)
struct Arc {
    double area, mx, my, angle;
};
__device__ __forceinline__ Arc arc_segment(double p0x, double p0y, double p1x, double p1y, double cx, double cy, double r) {
    p0x -= cx; p0y -= cy;
    p1x -= cx; p1y -= cy;
    const double a0 = atan2(p0y, p0x);
    double a1 = atan2(p1y, p1x);
    if (a1 < a0) a1 += 2 * kPi;
    if ((2 * kPi - (a1 - a0)) * r < 0x1p-42 * (fabs(cx) + fabs(cy) + r)) a1 = a0;
    const double ex = p0x - p1x, ey = p0y - p1y;
    const double d0 = sqrt(ex * ex + ey * ey) / 2;
    const double d1 = sqrt(fmax(0.0, r * r - d0 * d0));
    const double sg = a1 - a0 > kPi ? 1.0 : -1.0;  // the triangle joins the pie or leaves it
    const double tri = sg * d1 * d0, pie = r * r * (a1 - a0) / 2;
    double sm, cm;
    sincos((a1 + a0) / 2, &sm, &cm);
    const double f = 2.0 / 3.0 * (r * r * r) * sin((a1 - a0) / 2);
    Arc a;
    a.angle = a1 - a0;
    a.area = pie + tri;
    a.mx = f * cm + tri * ((1.0 / 3.0) * (p0x + p1x)) + a.area * cx;
    a.my = f * sm + tri * ((1.0 / 3.0) * (p0y + p1y)) + a.area * cy;
    return a;
}
#endif

}  // namespace sdot
