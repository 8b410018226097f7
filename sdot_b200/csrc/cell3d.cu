// 3D Laguerre-cell kernels (see cell3d.cuh).
//
// One warp builds one cell.  The cell is a simple convex polyhedron held by
// its vertices (every vertex on exactly three faces; a point where more faces
// meet is several vertices at one place), one vertex per lane and block of 32,
// in shared memory and in coordinates relative to the cell's Dirac.  A vertex
// keeps its three faces, counter-clockwise seen from outside, and opposite to
// each of them the vertex at the other end of its third edge.  Most of the
// walk asks on which side of a plane, or how near a box, the vertices lie:
// that is one evaluation per vertex, about 27 of them in 32 lanes, and a
// ballot.  (Held by its faces, each vertex was stored and tested three times
// in loops over the faces' polygons, 11.9 of 32 lanes active.)
//
// A plane cut marks the vertices outside; every edge from one of them to a
// vertex that stays gives a new vertex on the cut, found from its inside and
// outside ends, with the two faces of that edge and the cut as its faces.  Each
// face that is cut through has one new vertex where the cut enters it and one
// where it leaves: two tables over the faces link the new vertices.
// Faces live in numbered slots, a new face in the lowest one free, and the
// neighbour lists come out in slot order.
//
// Reference behaviour restated (ConvexPolyhedron3 and the 3D traversal):
//  * traversal and eviction test: SpZGrid::for_each_laguerre_cell, as in 2D
//    (SpZGrid.tcc:494-719, eviction :475-480), weighted bisector :506-522;
//  * volume: sum over faces of (O . N) area / 3 (ConvexPolyhedron3.tcc:1022-1057),
//    here with the cell's Dirac as the apex (O . N is the signed distance of the
//    face plane from it);
//  * centroid: pyramid centroids weighted by their volumes
//    (ConvexPolyhedron3::add_centroid_contrib, ConvexPolyhedron3.tcc:884-924);
//  * face area by a fan of triangles (ConvexPolyhedron3::area, :1367-1419);
//  * Hessian row: -1/2 coeff area / |x_i - x_j| per neighbour face, the
//    diagonal their sum; domain faces skipped (get_der_integrals_wrt_weights.h:43-88).
//
// Multilinear density (an extension: the reference's 3D densities are
// piecewise constant).  Relative to the cell's Dirac the density is
// sum_k g_k(u), g_k homogeneous of degree k <= 3, and by Euler's identity
// div(u g_k) = (k + 3) g_k, so the pyramid of a face at signed distance h
// holds h/(k+3) times the face integral of g_k (and u g_k, of degree k + 1,
// h/(k+4) times its face integral).  The face integrals use Dunavant's
// degree-4 rule on each fan triangle (6 points; D. A. Dunavant, "High degree
// efficient symmetrical Gaussian quadrature rules for the triangle", IJNME
// 21, 1985), exact for every term here.
#include "cell3d.cuh"

namespace sdot {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int STACK3 = 96;  // depth <= 10 levels (10 key bits per axis), <= 7 pending siblings each
constexpr int MAX_NEW = 128;  // vertices of a new face

// One warp's cell in shared memory: up to 32 VB vertices and MAXP faces.
template <int VB, int MAXP>
struct Cell3 {
    static constexpr int MAXV = 32 * VB, PW = MAXP / 32;
    static_assert(MAXV <= 1024 && PW <= 32, "vertex numbers of 10 bits, one word of the face mask per lane");
    double x[MAXV], y[MAXV], z[MAXV];
    double plane[MAXP][4];               // face: plane a . u <= b (a, b)
    int pid[MAXP];                       // face: its cut id
    unsigned alive[VB];                  // bit v & 31 of word v >> 5: vertex v is in use
    unsigned live[PW];                   // the same for the faces
    unsigned short fp[3][MAXV];          // vertex: its faces, counter-clockwise
    unsigned short nb[3][MAXV];          // vertex: the neighbour opposite to each face
};
// What a cut and the walk need beside the cell (not part of its copies).
template <int VB, int MAXP>
struct Work3 {
    unsigned out[VB];                    // the vertices outside a cut
    unsigned rm[MAXP / 32], hm[MAXP / 32];  // faces of the removed vertices, faces that are cut through
    int first[MAXP];                     // where the polygon of each face begins
    unsigned short ta[MAXP], tb[MAXP];   // new vertex with this face second, third
    unsigned short req[MAXP];            // edges to cut: vertex outside | edge << 10
    unsigned short list[MAXP];           // faces in slot order
    int stack[STACK3];
};

__device__ inline int next3(int i) { return i == 2 ? 0 : i + 1; }

// Loops over the blocks of vertices are unrolled where a cell has two.
template <int VB, class F>
__device__ __forceinline__ void each_block(int nr, F &&f) {
    if constexpr (VB <= 2) {
#pragma unroll
        for (int r = 0; r < VB; ++r)
            if (r < nr) f(r);
    } else {
        for (int r = 0; r < nr; ++r) f(r);
    }
}

// Cuts the cell by qx x + qy y + qz z <= qb.
// Outcome: 0 done (changed is set where a vertex was outside), 1 a capacity was
// exceeded, 2 degenerate geometry.
template <int VB, int MAXP>
__device__ __forceinline__ int cut3(Cell3<VB, MAXP> &C, Work3<VB, MAXP> &W, int &nr, double qx, double qy, double qz,
                                    double qb, int qid, bool &changed) {
    constexpr int PW = MAXP / 32;
    // the small cells keep the masks of faces in registers, and give the
    // places of removed vertices to new ones, so that most use one block
    constexpr bool SMALL = VB <= 2 && PW <= 2;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned any = 0, kept = 0;
    each_block<VB>(nr, [&](int r) {
        const unsigned al = C.alive[r];
        const int v = lane + 32 * r;
        const bool o = (al >> lane & 1u) && qb - (qx * C.x[v] + qy * C.y[v] + qz * C.z[v]) < 0.0;
        const unsigned om = __ballot_sync(FULL, o);
        if (lane == 0) W.out[r] = om;
        any |= om;
        kept |= al & ~om;
    });
    if (!any) return 0;
    changed = true;
    if (!SMALL && lane < PW) W.rm[lane] = W.hm[lane] = 0;
    __syncwarp();
    if (!kept) {  // nothing is left
        if (lane < PW) C.live[lane] = 0;
        nr = 0;
        __syncwarp();
        return 0;
    }
    // ---- the edges that cross the cut, and the faces touched
    unsigned long long rm = 0, hm = 0;  // SMALL: faces of the removed vertices, faces cut through
    int m = 0;
    each_block<VB>(nr, [&](int r) {
        const unsigned om = W.out[r];
        if (!om) return;
        const int v = lane + 32 * r;
        unsigned hz = 0;
        int f[3] = {0, 0, 0};
        if (om >> lane & 1u) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int u = C.nb[i][v];
                f[i] = C.fp[i][v];
                hz |= unsigned(!(W.out[u >> 5] >> (u & 31) & 1u)) << i;
                if (SMALL)
                    rm |= 1ull << f[i];
                else
                    atomicOr(&W.rm[f[i] >> 5], 1u << (f[i] & 31));
            }
        }
        const int c = __popc(hz);
        const unsigned b0 = __ballot_sync(FULL, c & 1), b1 = __ballot_sync(FULL, c & 2);
        int k = m + __popc(b0 & below) + 2 * __popc(b1 & below);
        m += __popc(b0) + 2 * __popc(b1);
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (hz >> i & 1u) {
                if (k < MAXP) W.req[k] = (unsigned short)(v | i << 10);
                const int a = f[i == 2 ? 0 : i + 1];
                if (SMALL)
                    hm |= 1ull << a;
                else
                    atomicOr(&W.hm[a >> 5], 1u << (a & 31));
                ++k;
            }
    });
    if (m < 3) return 2;
    if (m > MAX_NEW || m > MAXP) return 1;
    // ---- the new face's slot: the lowest one free once the faces that lost
    // every vertex (touched, not cut through) are gone
    int slot;
    if constexpr (SMALL) {
        unsigned long long live = C.live[0];
        if (PW == 2) live |= (unsigned long long)C.live[PW - 1] << 32;
        const unsigned g0 = __reduce_or_sync(FULL, unsigned(rm)), h0 = __reduce_or_sync(FULL, unsigned(hm));
        unsigned g1 = 0, h1 = 0;
        if (PW == 2 && live >> 32) {
            g1 = __reduce_or_sync(FULL, unsigned(rm >> 32));
            h1 = __reduce_or_sync(FULL, unsigned(hm >> 32));
        }
        live &= ~(((unsigned long long)g1 << 32 | g0) & ~((unsigned long long)h1 << 32 | h0));
        slot = __ffsll((long long)~live) - 1;
        if (slot < 0 || slot >= MAXP) return 1;
        live |= 1ull << slot;
        __syncwarp();
        if (lane < PW) C.live[lane] = unsigned(live >> (32 * lane));
    } else {
        __syncwarp();
        unsigned lw = FULL;
        if (lane < PW) lw = C.live[lane] & ~(W.rm[lane] & ~W.hm[lane]);
        const unsigned room = __ballot_sync(FULL, lw != FULL);
        if (!room) return 1;
        const int word = __ffs(int(room)) - 1;
        slot = 32 * word + __ffs(int(~__shfl_sync(FULL, lw, word))) - 1;
        if (lane == word) lw |= 1u << (slot & 31);
        if (lane < PW) C.live[lane] = lw;
    }
    // ---- the new vertices
    struct New {
        double x, y, z;
        int a, b, n;
    };
    // request q: the edge from a removed vertex t to the kept vertex n
    auto compute = [&](int q) {
        New w;
        const int t = q & 1023, i = q >> 10;
        const int ia = next3(i), ib = next3(ia);
        w.a = C.fp[ia][t];
        w.b = C.fp[ib][t];
        w.n = C.nb[i][t];
        const double tx = C.x[t], ty = C.y[t], tz = C.z[t], ux = C.x[w.n], uy = C.y[w.n], uz = C.z[w.n];
        const double din = qb - (qx * ux + qy * uy + qz * uz), dout = qb - (qx * tx + qy * ty + qz * tz);
        const double s = din / (din - dout);
        w.x = ux + s * (tx - ux);
        w.y = uy + s * (ty - uy);
        w.z = uz + s * (tz - uz);
        return w;
    };
    auto store = [&](int v, const New &w) {
        C.x[v] = w.x;
        C.y[v] = w.y;
        C.z[v] = w.z;
        C.fp[0][v] = (unsigned short)slot;
        C.fp[1][v] = (unsigned short)w.a;
        C.fp[2][v] = (unsigned short)w.b;
        C.nb[0][v] = (unsigned short)w.n;
        W.ta[w.a] = W.tb[w.b] = (unsigned short)v;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int f = C.fp[j][w.n];
            if (f != w.a && f != w.b) C.nb[j][w.n] = (unsigned short)v;
        }
    };
    unsigned mine = 0;  // bit r: this lane's vertex of block r is new
    int base = 0, top = 0;
    if constexpr (SMALL) {
        New w[VB];
        unsigned now[VB];
#pragma unroll
        for (int r = 0; r < VB; ++r) {
            now[r] = r < nr ? C.alive[r] & ~W.out[r] : 0u;
            if (base < m) {
                const int rank = base + __popc(~now[r] & below);
                if (!(now[r] >> lane & 1u) && rank < m) {
                    mine |= 1u << r;
                    w[r] = compute(W.req[rank]);
                }
                base += 32 - __popc(now[r]);
                now[r] |= __ballot_sync(FULL, mine >> r & 1u);
            }
            if (now[r]) top = r + 1;
        }
        if (base < m) return 1;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < VB; ++r) {
            if (mine >> r & 1u) store(lane + 32 * r, w[r]);
            if (lane == 0) C.alive[r] = now[r];
        }
    } else {
        // in places that were free before the cut: a removed vertex is read
        // until the last new one is made
        for (int r = 0; r < VB && (r < nr || base < m); ++r) {
            const unsigned al = r < nr ? C.alive[r] : 0u;
            const int rank = base + __popc(~al & below);
            const bool make = !(al >> lane & 1u) && rank < m;
            if (make) {
                store(lane + 32 * r, compute(W.req[rank]));
                mine |= 1u << r;
            }
            base += __popc(~al);
            const unsigned now = (r < nr ? al & ~W.out[r] : 0u) | __ballot_sync(FULL, make);
            __syncwarp();
            if (lane == 0) C.alive[r] = now;
            if (now) top = r + 1;
        }
        if (base < m) return 1;
    }
    nr = top;
    if (lane == 0) {
        C.pid[slot] = qid;
        C.plane[slot][0] = qx;
        C.plane[slot][1] = qy;
        C.plane[slot][2] = qz;
        C.plane[slot][3] = qb;
    }
    __syncwarp();
    // ---- link them around the new face: across the edge of the cut and face
    // b lies the new vertex that has b second, and so on.  Where a face was
    // entered twice, or entered and not left (the outside vertices are not one
    // patch), the tables do not agree
    bool bad = false;
    each_block<VB>(nr, [&](int r) {
        if (!(mine >> r & 1u)) return;
        const int v = lane + 32 * r, a = C.fp[1][v], b = C.fp[2][v];
        const int p = W.ta[b], q = W.tb[a];
        bad |= W.ta[a] != v || W.tb[b] != v;
        bad |= p >= 32 * VB || !(C.alive[p >> 5] >> (p & 31) & 1u) || C.fp[0][p] != slot || C.fp[1][p] != b;
        bad |= q >= 32 * VB || !(C.alive[q >> 5] >> (q & 31) & 1u) || C.fp[0][q] != slot || C.fp[2][q] != a;
        C.nb[1][v] = (unsigned short)p;
        C.nb[2][v] = (unsigned short)q;
    });
    if (__any_sync(FULL, bad)) return 2;
    __syncwarp();
    return 0;
}

// A multilinear density rewritten about the cell's Dirac c: coefficients of
// 1, u_x, u_y, u_z, u_x u_y, u_x u_z, u_y u_z, u_x u_y u_z for u = x - c.
struct PolyRel {
    double b1, bx, by, bz, bxy, bxz, byz, bxyz;
    __device__ PolyRel(const double *a, double cx, double cy, double cz) {
        bxyz = a[7];
        bxy = a[4] + a[7] * cz;
        bxz = a[5] + a[7] * cy;
        byz = a[6] + a[7] * cx;
        bx = a[1] + a[4] * cy + a[5] * cz + a[7] * cy * cz;
        by = a[2] + a[4] * cx + a[6] * cz + a[7] * cx * cz;
        bz = a[3] + a[5] * cx + a[6] * cy + a[7] * cx * cy;
        b1 = a[0] + a[1] * cx + a[2] * cy + a[3] * cz + a[4] * cx * cy + a[5] * cx * cz + a[6] * cy * cz +
             a[7] * cx * cy * cz;
    }
    // One point q (relative coordinates) of a face rule with weight wt:
    // pm += wt * sum_k g_k(q)/(k+3), pd += wt * q * sum_k g_k(q)/(k+4),
    // pf += wt * sum_k g_k(q).
    __device__ void add(double qx, double qy, double qz, double wt, double &pm, double &pdx, double &pdy, double &pdz,
                        double &pf) const {
        const double g0 = b1;
        const double g1 = bx * qx + by * qy + bz * qz;
        const double g2 = bxy * qx * qy + bxz * qx * qz + byz * qy * qz;
        const double g3 = bxyz * qx * qy * qz;
        pm += wt * (g0 * (1.0 / 3) + g1 * 0.25 + g2 * 0.2 + g3 * (1.0 / 6));
        const double gd = wt * (g0 * 0.25 + g1 * 0.2 + g2 * (1.0 / 6) + g3 * (1.0 / 7));
        pdx += gd * qx;
        pdy += gd * qy;
        pdz += gd * qz;
        pf += wt * (g0 + g1 + g2 + g3);
    }
    // Dunavant's degree-4 rule on the triangle p0, p0 + e1, p0 + e2 of area ta.
    __device__ void triangle(double x0, double y0, double z0, double e1x, double e1y, double e1z, double e2x,
                             double e2y, double e2z, double ta, double &pm, double &pdx, double &pdy, double &pdz,
                             double &pf) const {
        constexpr double A[2] = {0.4459484909159648863, 0.0915762135097707435};
        constexpr double W[2] = {0.2233815896780114657, 0.1099517436553218676};
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const double a = A[g], b = 1.0 - 2.0 * A[g], wt = W[g] * ta;
            add(x0 + a * (e1x + e2x), y0 + a * (e1y + e2y), z0 + a * (e1z + e2z), wt, pm, pdx, pdy, pdz, pf);
            add(x0 + b * e1x + a * e2x, y0 + b * e1y + a * e2y, z0 + b * e1z + a * e2z, wt, pm, pdx, pdy, pdz, pf);
            add(x0 + a * e1x + b * e2x, y0 + a * e1y + b * e2y, z0 + a * e1z + b * e2z, wt, pm, pdx, pdy, pdz, pf);
        }
    }
};

// The domain box as six faces (slots 0..5: x-lo, x-hi, y-lo, ...) and eight
// vertices (vertex v at corner bits x, y, z = 0, 1, 2 of v: 0 lo, 1 hi).
template <int VB, int MAXP>
__device__ __forceinline__ void init_box(Cell3<VB, MAXP> &C, int &nr, const Cell3DArgs &A, double c0x, double c0y,
                                         double c0z) {
    const int lane = threadIdx.x & 31;
    if (lane < 8) {
        const int bx = lane & 1, by = lane >> 1 & 1, bz = lane >> 2 & 1;
        C.x[lane] = (bx ? A.box_hi[0] : A.box_lo[0]) - c0x;
        C.y[lane] = (by ? A.box_hi[1] : A.box_lo[1]) - c0y;
        C.z[lane] = (bz ? A.box_hi[2] : A.box_lo[2]) - c0z;
        // faces x, y, z run counter-clockwise at the corner (hi, hi, hi), and
        // the other way round where an odd number of coordinates is lo
        const bool odd = !((bx + by + bz) & 1);
        C.fp[0][lane] = (unsigned short)bx;
        C.nb[0][lane] = (unsigned short)(lane ^ 1);
        C.fp[odd ? 2 : 1][lane] = (unsigned short)(2 + by);
        C.nb[odd ? 2 : 1][lane] = (unsigned short)(lane ^ 2);
        C.fp[odd ? 1 : 2][lane] = (unsigned short)(4 + bz);
        C.nb[odd ? 1 : 2][lane] = (unsigned short)(lane ^ 4);
    }
    if (lane < 6) {
        const int ax = lane >> 1, side = lane & 1;
        const double c = ax == 0 ? c0x : ax == 1 ? c0y : c0z;
        for (int d = 0; d < 3; ++d) C.plane[lane][d] = d == ax ? (side ? 1.0 : -1.0) : 0.0;
        C.plane[lane][3] = side ? A.box_hi[ax] - c : -(A.box_lo[ax] - c);
        C.pid[lane] = domain_id(lane);
    }
    for (int r = lane; r < VB; r += 32) C.alive[r] = r == 0 ? 0xffu : 0u;
    if (lane < MAXP / 32) C.live[lane] = lane == 0 ? 0x3fu : 0u;
    nr = 1;
    __syncwarp();
}

// First failed guard of a 3D cell (the 2D kernels' guard_fail).
__device__ void guard_fail3(const Cell3DArgs &A, int code, long long s, long long value) {
    if (A.guard && atomicCAS(&A.guard[0], 0, code) == 0) {
        A.guard[1] = int(s);
        A.guard[2] = int(value);
    }
    flag_error(A.err, DE_GUARD);
}

// The outputs of a cell that could not be built.
__device__ void fail_cell(const Cell3DArgs &A, long long s) {
    if (A.mass) A.mass[s] = nan("");
    if (A.ctd) A.ctd[3 * s] = A.ctd[3 * s + 1] = A.ctd[3 * s + 2] = nan("");
    if (A.rows.cnt) {
        A.rows.cnt[s] = 1;
        A.rows.col[s] = int(s);
        A.rows.val[s] = 0.0;
    }
    if (A.nb.cnt) A.nb.cnt[s] = 0;
}

// The faces of the cell in slot order into W.list, and for each the vertex its
// polygon is taken from into W.first (below the vertex, the slot of the face
// after it: the one with the lowest such slot, which does not depend on where
// the pass keeps its vertices, so that every pass sums alike); returns the
// number of faces, or -1 where the numbers of faces and vertices are not those
// of a polyhedron (V = 2 F - 4).
template <int VB, int MAXP>
__device__ __forceinline__ int list_faces(const Cell3<VB, MAXP> &C, Work3<VB, MAXP> &W, int nr) {
    const int lane = threadIdx.x & 31;
    int nf = 0, nv = 0;
#pragma unroll
    for (int w = 0; w < MAXP / 32; ++w) {
        const unsigned lw = C.live[w];
        W.first[32 * w + lane] = 1 << 30;
        if (lw >> lane & 1u) W.list[nf + __popc(lw & ((1u << lane) - 1u))] = (unsigned short)(32 * w + lane);
        nf += __popc(lw);
    }
    __syncwarp();
    for (int r = 0; r < nr; ++r) {
        const unsigned al = C.alive[r];
        nv += __popc(al);
        if (al >> lane & 1u)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int v = lane + 32 * r;
                atomicMin(&W.first[C.fp[i][v]], int(C.fp[i == 2 ? 0 : i + 1][v]) << 10 | v);
            }
    }
    __syncwarp();
    return nv == (nf ? 2 * nf - 4 : 0) ? nf : -1;
}

// Walks the polygon of face f counter-clockwise and calls tri(x0, y0, z0, e1,
// e2) for the triangles of its fan from its first vertex (e1, e2 from that
// vertex).  At most 32 VB steps; false where the walk does not close.
template <int VB, int MAXP, class F>
__device__ __forceinline__ bool walk_face(const Cell3<VB, MAXP> &C, const Work3<VB, MAXP> &W, int f, F &&tri) {
    if (W.first[f] >= 1 << 30) return false;
    const int v0 = W.first[f] & 1023;
    const double x0 = C.x[v0], y0 = C.y[v0], z0 = C.z[v0];
    auto step = [&](int v) { return int(C.fp[0][v] == f ? C.nb[1][v] : C.fp[1][v] == f ? C.nb[2][v] : C.nb[0][v]); };
    int v = step(v0);
    double ax = C.x[v] - x0, ay = C.y[v] - y0, az = C.z[v] - z0;
    for (int k = 0; k < 32 * VB; ++k) {
        v = step(v);
        if (v == v0) return true;
        const double bx = C.x[v] - x0, by = C.y[v] - y0, bz = C.z[v] - z0;
        tri(x0, y0, z0, ax, ay, az, bx, by, bz);
        ax = bx;
        ay = by;
        az = bz;
    }
    return false;
}

// Integrals of one face at constant density: its area and the sum over its
// fan of (triangle area) x 3 (triangle centroid).
template <int VB, int MAXP>
__device__ __forceinline__ bool face_area(const Cell3<VB, MAXP> &C, const Work3<VB, MAXP> &W, int f, double ux, double uy,
                                          double uz, double &area, double &fx, double &fy, double &fz) {
    return walk_face(C, W, f, [&](double x0, double y0, double z0, double e1x, double e1y, double e1z, double e2x,
                                  double e2y, double e2z) {
        const double ta =
            0.5 * ((e1y * e2z - e1z * e2y) * ux + (e1z * e2x - e1x * e2z) * uy + (e1x * e2y - e1y * e2x) * uz);
        area += ta;
        fx += ta * (3 * x0 + e1x + e2x);
        fy += ta * (3 * y0 + e1y + e2y);
        fz += ta * (3 * z0 + e1z + e2z);
    });
}

// Adds a face's pyramid of apex c0 (area, moments as face_area gives them, h
// the signed distance of its plane from c0): the centroid of a pyramid lies 3/4
// of the way from the apex to that of the face.
__device__ __forceinline__ void add_pyramid(double h, double area, double fx, double fy, double fz, double &vol,
                                            double &mx, double &my, double &mz) {
    const double v = h * area / 3;
    vol += v;
    if (area != 0) {
        const double k = v * 0.75 / (3 * area);
        mx += k * fx;
        my += k * fy;
        mz += k * fz;
    }
}

template <class T>
__device__ __forceinline__ void copy_cell(T &dst, const T &src) {
    static_assert(sizeof(T) % 8 == 0, "copied by 8 bytes");
    const double *s = reinterpret_cast<const double *>(&src);
    double *d = reinterpret_cast<double *>(&dst);
    for (int i = threadIdx.x & 31; i < int(sizeof(T) / 8); i += 32) d[i] = s[i];
    __syncwarp();
}

// The cell integrated voxel by voxel (ScaledImage::for_each_intersection,
// ScaledImage.tcc:98-149: each voxel box intersected with the cell and
// integrated with the voxel's value): for every voxel that the cell's bounding
// box meets a copy of the cell is cut by the voxel's six planes and
// integrated.  Sums (this lane's faces) into vol, m*, and per face slot of the
// cell the value-weighted area into wa.  Leaves the cell in C.  Returns 0, or
// 1 / 2 as cut3 (capacity, degenerate).
template <int VB, int MAXP>
__device__ int voxel_integrals(const Cell3DArgs &A, Cell3<VB, MAXP> &C, Work3<VB, MAXP> &W, Cell3<VB, MAXP> &B, double *wa,
                               int &nr, double c0x, double c0y, double c0z, double &vol, double &mx, double &my,
                               double &mz) {
    const int lane = threadIdx.x & 31;
    for (int f = lane; f < MAXP; f += 32) wa[f] = 0;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int r = 0; r < nr; ++r)
        if (C.alive[r] >> lane & 1u) {
            const int v = lane + 32 * r;
            lo[0] = fmin(lo[0], C.x[v]); hi[0] = fmax(hi[0], C.x[v]);
            lo[1] = fmin(lo[1], C.y[v]); hi[1] = fmax(hi[1], C.y[v]);
            lo[2] = fmin(lo[2], C.z[v]); hi[2] = fmax(hi[2], C.z[v]);
        }
    for (int d = 0; d < 3; ++d)
        for (int o = 16; o > 0; o >>= 1) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(FULL, lo[d], o));
            hi[d] = fmax(hi[d], __shfl_xor_sync(FULL, hi[d], o));
        }
    if (!(lo[0] <= hi[0])) return 0;  // an empty cell
    const double c0[3] = {c0x, c0y, c0z};
    int i0[3], i1[3];
    double ps[3];
    for (int d = 0; d < 3; ++d) {
        ps[d] = (A.img_hi[d] - A.img_lo[d]) / A.img_n[d];
        i0[d] = max(0, int(floor((lo[d] + c0[d] - A.img_lo[d]) / ps[d])));
        i1[d] = min(A.img_n[d] - 1, int(floor((hi[d] + c0[d] - A.img_lo[d]) / ps[d])));
    }
    const int nr0 = nr;
    __syncwarp();
    copy_cell(B, C);
    for (int iz = i0[2]; iz <= i1[2]; ++iz)
        for (int iy = i0[1]; iy <= i1[1]; ++iy)
            for (int ix = i0[0]; ix <= i1[0]; ++ix) {
                const double val = A.img[((long long)iz * A.img_n[1] + iy) * A.img_n[0] + ix];
                copy_cell(C, B);
                nr = nr0;
                // the voxel's six planes, relative to c0
                const int ii[3] = {ix, iy, iz};
                bool cut = false;
                for (int d = 0; d < 3; ++d) {
                    const double vlo = A.img_lo[d] + ps[d] * ii[d] - c0[d];
                    const double vhi = A.img_lo[d] + ps[d] * (ii[d] + 1) - c0[d];
                    double a[3] = {0, 0, 0};
                    a[d] = -1.0;
                    int st = cut3(C, W, nr, a[0], a[1], a[2], -vlo, domain_id(200 + 2 * d), cut);
                    if (st) return st;
                    a[d] = 1.0;
                    st = cut3(C, W, nr, a[0], a[1], a[2], vhi, domain_id(201 + 2 * d), cut);
                    if (st) return st;
                }
                const int nf = list_faces(C, W, nr);
                if (nf < 0) return 2;
                bool closed = true;
                for (int k = lane; k < nf; k += 32) {
                    const int f = W.list[k];
                    const double *q = C.plane[f];
                    const double na = sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2]);
                    double area = 0, fx = 0, fy = 0, fz = 0, v = 0, px = 0, py = 0, pz = 0;
                    closed &= face_area(C, W, f, q[0] / na, q[1] / na, q[2] / na, area, fx, fy, fz);
                    add_pyramid(q[3] / na, area, fx, fy, fz, v, px, py, pz);
                    vol += val * v;
                    mx += val * px;
                    my += val * py;
                    mz += val * pz;
                    // a face of the cell keeps its slot while it lives
                    if (C.pid[f] >= 0) wa[f] += val * area;
                }
                if (!__all_sync(FULL, closed)) return 2;
                __syncwarp();
            }
    copy_cell(C, B);
    nr = nr0;
    return 0;
}

// The squared distance from c0 of the farthest vertex, rounded up to 20 bits
// (more than a relative 4e-7 above it), so that what is ruled out by it is so
// by a margin beyond the rounding of the exact tests.
template <int VB, class C3>
__device__ __forceinline__ int farthest(const C3 &C, int nr) {
    const int lane = threadIdx.x & 31;
    double m = 0;
    each_block<VB>(nr, [&](int r) {
        if (!(C.alive[r] >> lane & 1u)) return;
        const int v = lane + 32 * r;
        const double d = C.x[v] * C.x[v] + C.y[v] * C.y[v] + C.z[v] * C.z[v];
        m = d > m ? d : m;
    });
    return int(__reduce_max_sync(FULL, unsigned(__double2hiint(m)))) + 2;
}

// Squares outside (TINY, HUGE_SQ) are not compared: they may have lost their
// digits.
constexpr double TINY = 1e-290, HUGE_SQ = 1e300;
// Boxes waiting beyond which a sweep is worth its loads.
constexpr int SWEEP_MIN = 2;

// A box is evicted if every vertex u has |u|^2 - w0 <= d(u)^2 - maxw, d its
// distance from the box.  With D the box's distance from c0 and every |u| <= R
// <= D, d(u) >= D - |u|, and that holds if 2 D R <= D^2 + w0 - maxw.
__device__ __forceinline__ bool beyond(const TreeNode<3> &nd, double c0x, double c0y, double c0z, double w0, double r2) {
    const double gx = gap(nd.lo[0], nd.hi[0], c0x), gy = gap(nd.lo[1], nd.hi[1], c0y), gz = gap(nd.lo[2], nd.hi[2], c0z);
    const double d2 = gx * gx + gy * gy + gz * gz, t = d2 + (w0 - nd.maxw), q = t * t;
    return t > 0 && d2 >= r2 && q >= 4 * (r2 * d2) && q > TINY && q < HUGE_SQ;
}

// Builds and integrates the cell of sorted Dirac s.  Returns 0 (outputs
// written), 1 (a capacity was exceeded: retry in the next pass), 2 (failed:
// outputs written as NaN / empty row, error flagged).
enum Density3 : int { D_CONST = 0, D_POLY = 1, D_IMAGE = 2 };
template <int VB, int MAXP, int DENS, int PASS>
__device__ __forceinline__ int cell3d(const Cell3DArgs &A, long long s, Cell3<VB, MAXP> &C, Work3<VB, MAXP> &W,
                                      Cell3<VB, MAXP> *B, double *wa) {
    const int lane = threadIdx.x & 31;
    const double c0x = A.pos[3 * s], c0y = A.pos[3 * s + 1], c0z = A.pos[3 * s + 2], w0 = A.w[s];
    int nr;
    init_box(C, nr, A, c0x, c0y, c0z);
    int status = 0;
    bool changed = true;  // since r2 was taken
    int r2h = 0;          // high word of a bound of their squared distance from c0
    // a convex shape: its half-spaces cut the box first (relative to c0:
    // a . u <= b - a . c0), as ConvexPolyhedronAssembly::add_convex_polyhedron
    // cuts its box (ConvexPolyhedronAssembly.tcc:7-33)
    for (int k = 0; k < A.nplanes && status == 0; ++k) {
        const double ax = A.planes[4 * k], ay = A.planes[4 * k + 1], az = A.planes[4 * k + 2];
        const double b = A.planes[4 * k + 3] - (ax * c0x + ay * c0y + az * c0z);
        status = cut3(C, W, nr, ax, ay, az, b, domain_id(6 + k), changed);
    }
    if (lane == 0) W.stack[0] = 0;
    __syncwarp();
    int sp = 1;
    for (int visits = 0; sp > 0 && status == 0; ++visits) {
        if (visits > A.max_nodes) {
            if (lane == 0) flag_error(A.err, DE_ITER);
            status = 2;
            break;
        }
        // After a cut the boxes waiting are tried against the ball that holds
        // the cell, one per lane (the 32 nearest): most of those that would
        // fail the vertex test when popped go here, many at a time
        if (changed) {
            changed = false;
            r2h = farthest<VB>(C, nr);
            if (sp > SWEEP_MIN) {
                const int base = max(sp - 32, 0);
                bool keep = false;
                int mine = 0;
                if (base + lane < sp) {
                    mine = W.stack[base + lane];
                    const TreeNode<3> nd = A.nodes[mine];
                    keep = !beyond(nd, c0x, c0y, c0z, w0, __hiloint2double(r2h, 0));
                }
                const unsigned km = __ballot_sync(FULL, keep);
                __syncwarp();
                if (keep) W.stack[base + __popc(km & ((1u << lane) - 1u))] = mine;
                __syncwarp();
                sp = base + __popc(km);
                if (sp == 0) break;
            }
        }
        const int node = W.stack[--sp];
        __syncwarp();
        const TreeNode<3> nd = A.nodes[node];
        // eviction test (SpZGrid.tcc:475-480) on every vertex
        const double lo0 = nd.lo[0] - c0x, lo1 = nd.lo[1] - c0y, lo2 = nd.lo[2] - c0z;
        const double hi0 = nd.hi[0] - c0x, hi1 = nd.hi[1] - c0y, hi2 = nd.hi[2] - c0z;
        bool need = false;
        each_block<VB>(nr, [&](int r) {
            if (need) return;
            bool fail = false;
            if (C.alive[r] >> lane & 1u) {
                const int v = lane + 32 * r;
                const double px = C.x[v], py = C.y[v], pz = C.z[v];
                const double qx = gap(lo0, hi0, px), qy = gap(lo1, hi1, py), qz = gap(lo2, hi2, pz);
                const double lhs = px * px + py * py + pz * pz - w0;
                const double rhs = qx * qx + qy * qy + qz * qz - nd.maxw;
                fail = !(lhs <= rhs);
            }
            need = __any_sync(FULL, fail);
        });
        if (!need) continue;
        if (nd.b < 0) {
            const int first = nd.a, nch = -nd.b;
            if (nch < 2 || nch > 8 || first < 1 || first + nch > A.max_nodes) {
                if (lane == 0) guard_fail3(A, 1, s, node);
                status = 2;
                break;
            }
            if (sp + nch > STACK3) {
                if (lane == 0) flag_error(A.err, DE_STACK);
                status = 2;
                break;
            }
            // children farthest first (nearest popped first): lane c keys child
            // c and writes it at its rank among the keys (larger keys first,
            // equal keys in child order, as a stable sort would place them)
            float key = 0;
            if (lane < nch) {
                const TreeNode<3> &cn = A.nodes[first + lane];
                const double mx = 0.5 * (cn.lo[0] + cn.hi[0]) - c0x, my = 0.5 * (cn.lo[1] + cn.hi[1]) - c0y,
                             mz = 0.5 * (cn.lo[2] + cn.hi[2]) - c0z;
                key = float(mx * mx + my * my + mz * mz);
                if (beyond(cn, c0x, c0y, c0z, w0, __hiloint2double(r2h, 0))) key = -1.f;  // not pushed
            }
            int rank = 0;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float kc = __shfl_sync(FULL, key, c);
                rank += c < nch && (kc > key || (kc == key && c < lane));
            }
            const unsigned pm = __ballot_sync(FULL, lane < nch && !(key < 0));
            if (pm >> lane & 1u) W.stack[sp + rank] = first + lane;
            __syncwarp();
            sp += __popc(pm);
        } else {
            if (nd.a < 0 || nd.b > A.n) {
                if (lane == 0) guard_fail3(A, 2, s, node);
                status = 2;
                break;
            }
            for (int j0 = nd.a; j0 < nd.b && status == 0; j0 += 32) {
                // weighted bisectors, one per lane, relative to c0: V . u <=
                // 1/2 |V|^2 + 1/2 (w0 - w1); those that miss the ball cut
                // nothing, the others are tried in index order
                bool near = false;
                double vx = 0, vy = 0, vz = 0, qb = 0;
                if (j0 + lane < nd.b && j0 + lane != s) {
                    const int j = j0 + lane;
                    vx = A.pos[3 * j] - c0x, vy = A.pos[3 * j + 1] - c0y, vz = A.pos[3 * j + 2] - c0z;
                    const double v2 = vx * vx + vy * vy + vz * vz;
                    qb = 0.5 * v2 + 0.5 * (w0 - A.w[j]);
                    const double q = qb * qb;
                    near = !(qb > 0 && q >= __hiloint2double(r2h, 0) * v2 && q > TINY && q < HUGE_SQ);
                }
                for (unsigned todo = __ballot_sync(FULL, near); todo && status == 0; todo &= todo - 1) {
                    const int l = __ffs(int(todo)) - 1;
                    status = cut3(C, W, nr, __shfl_sync(FULL, vx, l), __shfl_sync(FULL, vy, l), __shfl_sync(FULL, vz, l),
                                  __shfl_sync(FULL, qb, l), j0 + l, changed);
                }
            }
        }
    }
    if (status == 1) return 1;
    // ---- integrals over the faces (pyramids with apex c0)
    double vol = 0, mx = 0, my = 0, mz = 0, der0 = 0;
    if (DENS == D_IMAGE && status == 0) {
        status = voxel_integrals(A, C, W, *B, wa, nr, c0x, c0y, c0z, vol, mx, my, mz);
        if (status == 1) return 1;
    }
    int nf = 0, nrow = 0;
    if (status == 0) {
        nf = list_faces(C, W, nr);
        if (nf < 0) status = 2;
    }
    bool ok = true;  // the rows fit the side buffer
    if (status == 0) {
        for (int k0 = 0; k0 < nf; k0 += 32)
            nrow += __popc(__ballot_sync(FULL, k0 + lane < nf && C.pid[W.list[min(k0 + lane, nf - 1)]] >= 0));
        RowPut row(A.rows, s, nrow + 1), nbr(A.nb, s, nf);
        ok = row.ok && nbr.ok;
        bool closed = true;
        int at = 0;
        for (int k0 = 0; k0 < nf; k0 += 32) {
            const int k = k0 + lane;
            const bool has = k < nf;
            const int f = has ? W.list[k] : 0;
            const int id = has ? C.pid[f] : -1;
            const unsigned rm = __ballot_sync(FULL, id >= 0);
            if (has) {
                const double qa = C.plane[f][0], qc = C.plane[f][1], qd = C.plane[f][2];
                const double na = sqrt(qa * qa + qc * qc + qd * qd);
                const double ux = qa / na, uy = qc / na, uz = qd / na;
                const double h = C.plane[f][3] / na;  // signed distance of the face plane from c0
                double area = 0;
                if (DENS == D_IMAGE) {
                    area = wa[f];  // integrated voxel by voxel above
                } else if (DENS == D_POLY) {
                    const PolyRel pr(A.poly, c0x, c0y, c0z);
                    double pm = 0, pdx = 0, pdy = 0, pdz = 0;  // density-weighted
                    closed &= walk_face(C, W, f, [&](double x0, double y0, double z0, double e1x, double e1y, double e1z,
                                                     double e2x, double e2y, double e2z) {
                        const double ta = 0.5 * ((e1y * e2z - e1z * e2y) * ux + (e1z * e2x - e1x * e2z) * uy +
                                                 (e1x * e2y - e1y * e2x) * uz);
                        pr.triangle(x0, y0, z0, e1x, e1y, e1z, e2x, e2y, e2z, ta, pm, pdx, pdy, pdz, area);
                    });
                    vol += h * pm;
                    mx += h * pdx;
                    my += h * pdy;
                    mz += h * pdz;
                } else {
                    double fx = 0, fy = 0, fz = 0;
                    closed &= face_area(C, W, f, ux, uy, uz, area, fx, fy, fz);
                    add_pyramid(h, area, fx, fy, fz, vol, mx, my, mz);
                }
                if (id >= 0) {
                    const double bd = 0.5 * A.coeff * area / na;  // |x_i - x_j| = |a|
                    row.put(at + __popc(rm & ((1u << lane) - 1u)), id, -bd);
                    der0 += bd;
                }
                nbr.put(k, id, 0.0);
            }
            at += __popc(rm);
        }
        if (!__all_sync(FULL, closed)) status = 2;
        for (int o = 16; o > 0; o >>= 1) {
            vol += __shfl_xor_sync(FULL, vol, o);
            mx += __shfl_xor_sync(FULL, mx, o);
            my += __shfl_xor_sync(FULL, my, o);
            mz += __shfl_xor_sync(FULL, mz, o);
            der0 += __shfl_xor_sync(FULL, der0, o);
        }
        if (status == 0 && ok && lane == 0) {
            row.put(nrow, int(s), der0);
            row.finish();
            nbr.finish();
            if (A.mass) A.mass[s] = A.coeff * vol;
            if (A.ctd) {
                const bool empty = vol == 0;
                A.ctd[3 * s] = empty ? 0.0 : c0x + mx / vol;
                A.ctd[3 * s + 1] = empty ? 0.0 : c0y + my / vol;
                A.ctd[3 * s + 2] = empty ? 0.0 : c0z + mz / vol;
            }
            if (A.hint) {
                // polyhedra grow larger during the build than at its end, so
                // the hint is the pass that held this build, lowered by one
                // level at most when the final polyhedron is much smaller (a
                // cell that then overflows moves on to the next pass again)
                const int level = 2 * nf - 4 <= 40 ? 0 : 2 * nf - 4 <= 128 ? 1 : 2;
                A.hint[s] = (unsigned char)(level >= PASS ? PASS : PASS - 1);
            }
        }
    }
    if (status == 2 || !ok) {
        if (lane == 0) {
            flag_error(A.err, status == 2 ? DE_DEGEN : DE_SIDE);
            fail_cell(A, s);
        }
        return 2;
    }
    return 0;
}

// Shared memory of one warp of a pass: the cell, its working space and, for
// voxel images, the copy of the cell and the weighted areas.
template <int VB, int MAXP, int DENS>
constexpr size_t warp_smem_bytes() {
    const size_t b = sizeof(Cell3<VB, MAXP>) + sizeof(Work3<VB, MAXP>) +
                     (DENS == D_IMAGE ? sizeof(Cell3<VB, MAXP>) + MAXP * sizeof(double) : 0);
    return (b + 15) / 16 * 16;
}

// The passes.  The first takes every cell, with room for 64 vertices (a
// uniform cell has 27, and about 36 at most while it is built).  Cells that
// outgrow it run again with 192 vertices and 128 faces, then with 640 vertices
// and 256 faces (508 vertices): every pass in shared memory.
//
// Bound by instruction issue and by the latency of FP64 and shared memory
// between the instructions (28 effective cuts per uniform cell), so the first
// pass takes the occupancy of 80 registers (20, 24, 28, 32 blocks at constant
// density: 0.81, 0.74, 0.77, 0.81 ms for 20,000 uniform Diracs; 18, 24, 26, 20
// of the multilinear kernel 7.9, 7.3, 7.6, 7.9 ms for 200,000).  One warp a
// block: with two the block waited for the longer cell (9.5 -> 8.5 ms).
// The tests against the ball took the place of most of the 98 box tests and 50
// ineffective cuts of a cell that the vertices were tried for before: with the
// blocks chosen anew, 200,000 Diracs of the 3D mix 10.2 -> 7.3 ms, 20,000
// uniform ones 1.13 -> 0.74.  The larger passes fetch their cells (with a fixed
// share each, 20,000 clustered Diracs took 2.7 instead of 2.2 ms).
// Against the faces held as polygons, four passes, the last two in global
// memory: 30.9 -> 7.3 ms and 13.1 -> 2.2 ms, whole evaluations 31.7 -> 7.9 and
// 13.9 -> 2.7 ms.
struct Pass0 { static constexpr int VB = 2, MAXP = 64, BLOCKS = 24, POLY_BLOCKS = 24; };
struct Pass1 { static constexpr int VB = 6, MAXP = 128, BLOCKS = 16, POLY_BLOCKS = 10; };
struct Pass2 { static constexpr int VB = 20, MAXP = 256, BLOCKS = 5, POLY_BLOCKS = 5; };

template <class P, int PASS, int DENS>
__global__ void __launch_bounds__(32, DENS == D_IMAGE ? 1 : DENS == D_POLY ? P::POLY_BLOCKS : P::BLOCKS)
    k_cells3d(const Cell3DArgs A, const int *list, const int *list_cnt, int *cursor, int *next_list, int *next_cnt) {
    extern __shared__ double smem3[];
    constexpr int VB = P::VB, MAXP = P::MAXP;
    const int lane = threadIdx.x;
    char *base = reinterpret_cast<char *>(smem3);
    using C3 = Cell3<VB, MAXP>;
    using W3 = Work3<VB, MAXP>;
    C3 &C = *reinterpret_cast<C3 *>(base);
    W3 &W = *reinterpret_cast<W3 *>(base + sizeof(C3));
    C3 *B = reinterpret_cast<C3 *>(base + sizeof(C3) + sizeof(W3));
    double *wa = reinterpret_cast<double *>(base + 2 * sizeof(C3) + sizeof(W3));
    // the first pass has a block per cell; the others' blocks fetch the next
    // entry of their list until it is used up (fewer than n of them, so the
    // cursor stays an int)
    const long long cnt = PASS == 0 ? A.n : *list_cnt;
    auto fetch = [&] {
        int k = 0;
        if (lane == 0) k = atomicAdd(cursor, 1);
        return (long long)__shfl_sync(FULL, k, 0);
    };
    for (long long i = PASS == 0 ? blockIdx.x : fetch(); i < cnt; i = PASS == 0 ? cnt : fetch()) {
        const long long s = PASS == 0 ? i : list[i];
        if (PASS == 0 && A.use_hint && A.hint) {
            // a cell that needed a larger pass last time goes straight there
            const int h = A.hint[s];
            if (h == 1 || h == 2) {
                if (lane == 0) {
                    if (h == 1)
                        next_list[atomicAdd(next_cnt, 1)] = int(s);
                    else
                        A.ovf_list2[atomicAdd(A.ovf_cnt2, 1)] = int(s);
                }
                return;
            }
        }
        const int r = cell3d<VB, MAXP, DENS, PASS>(A, s, C, W, B, wa);
        if (r == 1 && lane == 0) {
            if (next_list) {
                next_list[atomicAdd(next_cnt, 1)] = int(s);
            } else {
                flag_error(A.err, DE_CAPACITY);
                fail_cell(A, s);
            }
        }
        __syncwarp();
    }
}

template <class P, int PASS, int DENS>
void launch3(const Cell3DArgs &a, const int *list, const int *list_cnt, int *cursor, int *next_list, int *next_cnt,
             long long blocks, cudaStream_t st) {
    const size_t smem = warp_smem_bytes<P::VB, P::MAXP, DENS>();
    static PerDevice<int> attr;
    attr.once([&] {
        SDOT_CUDA(cudaFuncSetAttribute(k_cells3d<P, PASS, DENS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    });
    k_cells3d<P, PASS, DENS><<<int(blocks), 32, smem, st>>>(a, list, list_cnt, cursor, next_list, next_cnt);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

template <int DENS>
void launch_passes(const Cell3DArgs &a, cudaStream_t st) {
    // one block per cell: the hardware hands them out as blocks end
    launch3<Pass0, 0, DENS>(a, nullptr, nullptr, nullptr, a.ovf_list, a.ovf_cnt, a.n, st);
    // the larger passes take the overflow lists (their lengths are on the
    // device): as many blocks as fit the device, or one per cell
    launch3<Pass1, 1, DENS>(a, a.ovf_list, a.ovf_cnt, a.ovf_cnt2 + 1, a.ovf_list2, a.ovf_cnt2,
                            std::min<long long>(a.n, 148LL * Pass1::BLOCKS), st);
    launch3<Pass2, 2, DENS>(a, a.ovf_list2, a.ovf_cnt2, a.ovf_cnt2 + 2, nullptr, nullptr,
                            std::min<long long>(a.n, 148LL * Pass2::BLOCKS), st);
}

}  // namespace

void cells3d_launch(const Cell3DArgs &a, cudaStream_t st) {
    if (a.n == 0) return;
    SDOT_CUDA(cudaMemsetAsync(a.ovf_cnt, 0, sizeof(int), st));
    SDOT_CUDA(cudaMemsetAsync(a.ovf_cnt2, 0, 3 * sizeof(int), st));  // and the cursors
    if (a.rows.side_used) SDOT_CUDA(cudaMemsetAsync(a.rows.side_used, 0, sizeof(unsigned long long), st));
    if (a.nb.side_used) SDOT_CUDA(cudaMemsetAsync(a.nb.side_used, 0, sizeof(unsigned long long), st));
    if (a.img)
        launch_passes<D_IMAGE>(a, st);
    else if (a.has_poly)
        launch_passes<D_POLY>(a, st);
    else
        launch_passes<D_CONST>(a, st);
}

}  // namespace sdot
