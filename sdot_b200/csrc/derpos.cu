// Derivatives of the cell centroids and masses with respect to the weights
// and the positions (2D): get_der_centroids_and_integrals_wrt_weight_and_positions
// (src/sdot/PowerDiagram/get_der_centroids_and_integrals_wrt_weight_and_positions.h:17-216).
//
// The cells come from the neighbour pass (one row per cell in sorted order:
// the cut id of the edge leaving each vertex, domain edges included); each
// vertex is rebuilt in FP64 as the intersection of the lines of its two edges
// (a weighted bisector, or a domain edge), in coordinates relative to the
// cell's Dirac.  Per edge with a Dirac on the other side the reference's
// boundary item gives the measure (coeff * length), the position integral
// 1/2 l (p0 + p1) and the second moments l/6 (2 (p0 p0' + p1 p1') + p0 p1'
// + p1 p0') (ConvexPolyhedron2.tcc:437-478); the row items are the reference's
// 3 x 3 blocks (rows: centroid x, centroid y, mass; columns: position x,
// position y, weight), corrected by the centroid and divided by
// mass + (mass == 1) as the reference divides (.h:178-182), sorted by column
// and merged.  Eight lanes per cell, an edge each; cells of more than DP_CAP
// vertices report a capacity error.
#include "derpos.cuh"

#include <climits>

namespace sdot {

namespace {

constexpr int DP_CAP = 64;   // vertices of a cell
constexpr int DP_ROW = 65;   // blocks of a row (one per edge and the diagonal)
constexpr int LANES = 8;     // lanes per cell: an edge each up to 8 edges (a cell has 6 on average)
constexpr int TB = 64;
constexpr int CELLS = TB / LANES;

struct DpArgs {
    Rows nb;
    long long n;
    const double *pos, *w;
    const int *idx;
    int start_n;
    const double *start_xy;
    double coeff;
    int ntrans;
    const double *trans;
};

// position of the Dirac (or periodic image) on the other side of an edge with this id
__device__ void other_site(const DpArgs &A, int id, double &x, double &y, double &w, int &j) {
    const unsigned n = unsigned(A.n), t = A.ntrans ? unsigned(id) / n : 0;
    j = int(unsigned(id) - t * n);
    x = A.pos[2 * j];
    y = A.pos[2 * j + 1];
    if (t) {
        x += A.trans[2 * (t - 1)];
        y += A.trans[2 * (t - 1) + 1];
    }
    w = A.w[j];
}

// line a . u = b of the edge with this id, u relative to c0
__device__ void edge_line(const DpArgs &A, int id, double c0x, double c0y, double w0, double &ax, double &ay,
                          double &b) {
    if (id >= 0) {
        double x, y, w1;
        int j;
        other_site(A, id, x, y, w1, j);
        const double dx = x - c0x, dy = y - c0y;
        ax = dx;
        ay = dy;
        b = 0.5 * (dx * dx + dy * dy) + 0.5 * (w0 - w1);
    } else {
        const int e = domain_edge(id), e1 = e + 1 < A.start_n ? e + 1 : 0;
        const double p0x = A.start_xy[2 * e] - c0x, p0y = A.start_xy[2 * e + 1] - c0y;
        const double p1x = A.start_xy[2 * e1] - c0x, p1y = A.start_xy[2 * e1 + 1] - c0y;
        ax = p0y - p1y;
        ay = p1x - p0x;
        b = ax * p0x + ay * p0y;
    }
}

// The edges of a cell in shared memory.
struct RowIds {
    int id[DP_CAP];
    int col[DP_ROW];   // caller column of every item (edge k, or m for the diagonal); -1: a domain edge
    int head[DP_ROW];  // the same where no item before it has this column, else INT_MAX
};

// The cell rebuilt from them: its vertices; and where it lies.
struct CellGeo {
    int m;
    const int *id;
    double c0x, c0y, w0;
    const double *vx, *vy;
    double cx, cy, mass;
};

// Lanes of one cell: the group's place in the warp.
struct Group {
    int lane;       // in the group
    unsigned mask;  // of its lanes
    __device__ Group() : lane(threadIdx.x & (LANES - 1)), mask(0xffu << (threadIdx.x & 24)) {}
    template <class T>
    __device__ T sum(T v) const {
#pragma unroll
        for (int o = LANES / 2; o; o >>= 1) v += __shfl_xor_sync(mask, v, o);
        return v;
    }
};

// Edges and columns of cell s (sorted order), and the number of distinct
// columns; -1 past the capacity (or for an edge id that this pass does not
// handle).  Columns are unique but for periodic images.
__device__ int load_row(const DpArgs &A, long long s, const Group &g, RowIds &r, int &m) {
    m = A.nb.cnt[s];
    if (m > DP_CAP) return -1;
    const long long nid = (A.ntrans + 1LL) * A.n;
    bool ok = true;
    for (int k = g.lane; k < m; k += LANES) {
        const int id = *A.nb.colp(s, k);
        // a Dirac (or an image) or a domain edge; anything else (an arc) is not handled
        const bool known = id >= 0 ? id < nid : id <= ID_DOMAIN0 && domain_edge(id) < A.start_n;
        ok = ok && known;
        r.id[k] = id;
        r.col[k] = known && id >= 0 ? A.idx[A.ntrans ? int(unsigned(id) % unsigned(A.n)) : id] : -1;
    }
    if (g.lane == 0) r.col[m] = A.idx[s];
    if (__any_sync(g.mask, !ok)) return -1;
    __syncwarp(g.mask);
    int heads = 0;
    for (int k = g.lane; k <= m; k += LANES) {
        const int c = r.col[k];
        bool head = c >= 0;
        for (int q = 0; q < k; ++q) head = head && r.col[q] != c;
        r.head[k] = head ? c : INT_MAX;
        heads += head;
    }
    heads = g.sum(heads);
    __syncwarp(g.mask);
    return heads;
}

// The block of the edge leaving vertex i0 (a Dirac on the other side): t
// receives the off-diagonal block (row-major, rows centroid x, centroid y,
// mass; columns x, y, weight), d0 (if not null) accumulates the diagonal's
// share.
__device__ void edge_block(const DpArgs &A, const CellGeo &g, int i0, double *t, double *d0) {
    const int i1 = i0 + 1 < g.m ? i0 + 1 : 0;
    double x1, y1, w1;
    int j;
    other_site(A, g.id[i0], x1, y1, w1, j);
    const double p0[2] = {g.vx[i0], g.vy[i0]}, p1[2] = {g.vx[i1], g.vy[i1]};
    const double l = sqrt((p1[0] - p0[0]) * (p1[0] - p0[0]) + (p1[1] - p0[1]) * (p1[1] - p0[1]));
    const double meas = A.coeff * l;
    const double P[2] = {0.5 * l * (p0[0] + p1[0]), 0.5 * l * (p0[1] + p1[1])};
    double M[2][2];
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b)
            M[a][b] = l / 6 * (2 * (p0[a] * p0[b] + p1[a] * p1[b]) + p0[a] * p1[b] + p1[a] * p0[b]);
    const double c0[2] = {g.c0x, g.c0y}, c1[2] = {x1, y1};
    const double dist = sqrt((x1 - g.c0x) * (x1 - g.c0x) + (y1 - g.c0y) * (y1 - g.c0y));
    const double bd = 0.5 * meas / dist;
    for (int k = 0; k < 9; ++k) t[k] = 0;
    if (d0) d0[8] += bd;
    t[8] = -bd;
    for (int q = 0; q < 2; ++q) {
        const double value = 0.5 * P[q] / dist;
        if (d0) d0[3 * q + 2] += value;
        t[3 * q + 2] = -value;
    }
    for (int d = 0; d < 2; ++d) {
        if (d0) d0[6 + d] += (P[d] - meas * c0[d]) / dist;
        t[6 + d] = (meas * c1[d] - P[d]) / dist;
    }
    for (int d = 0; d < 2; ++d)
        for (int q = 0; q < 2; ++q) {
            if (d0) d0[3 * q + d] += (M[d][q] - P[q] * c0[d]) / dist;
            t[3 * q + d] = (P[q] * c1[d] - M[d][q]) / dist;
        }
}

// centroid correction, as the reference divides (.h:178-182)
__device__ void correct(const CellGeo &g, double *t) {
    const double div = g.mass + (g.mass == 1);
    const double c[2] = {g.cx, g.cy};
    for (int r = 0; r < 2; ++r)
        for (int e = 0; e < 3; ++e) t[3 * r + e] = (t[3 * r + e] - t[6 + e] * c[r]) / div;
}

__global__ void __launch_bounds__(TB) k_dp_count(DpArgs A, long long *nblocks, unsigned *err) {
    __shared__ RowIds rows[CELLS];
    const Group g;
    const long long s = blockIdx.x * (long long)CELLS + threadIdx.x / LANES;
    if (s >= A.n) return;
    int m;
    const int cnt = load_row(A, s, g, rows[threadIdx.x / LANES], m);
    if (g.lane) return;
    if (cnt < 0) atomicOr(err, unsigned(DE_CAPACITY));
    nblocks[A.idx[s]] = cnt < 0 ? 0 : cnt;
}

// block offsets boff (caller order, exclusive scan of the counts) -> CSR of
// 3 n rows: row 3 i + d holds, for every block of Dirac i, its row d; the
// items of one column are corrected, then added in index order (the diagonal
// last).
// Bound by its loads of neighbours and its stores (54 entries of 16 bytes a
// cell).  Lanes of a cell share its lines and vertices through shared memory
// and store blocks that lie side by side; a thread per cell kept 2 KB of local
// memory each and stored 72 bytes apart.  100,000 Diracs, the whole call with
// the count: 1035 -> 862 us.
__global__ void __launch_bounds__(TB) k_dp_write(DpArgs A, const long long *boff, long long *off, long long *cols,
                                                 double *vals, double *v) {
    struct Cell {
        RowIds r;
        double ax[DP_CAP], ay[DP_CAP], b[DP_CAP], vx[DP_CAP], vy[DP_CAP];
    };
    __shared__ Cell cells[CELLS];
    Cell &C = cells[threadIdx.x / LANES];
    const Group gr;
    const long long s = blockIdx.x * (long long)CELLS + threadIdx.x / LANES;
    if (s >= A.n) return;
    const long long i = A.idx[s];
    const long long base = 9 * boff[i];
    if (s == 0 && gr.lane == 0) off[3 * A.n] = 9 * boff[A.n];
    CellGeo g;
    const int cnt = load_row(A, s, gr, C.r, g.m);
    if (cnt < 0) {
        if (gr.lane < 3) {
            off[3 * i + gr.lane] = base;
            v[3 * i + gr.lane] = 0;
        }
        return;
    }
    const int m = g.m;
    g.id = C.r.id;
    g.vx = C.vx;
    g.vy = C.vy;
    g.c0x = A.pos[2 * s];
    g.c0y = A.pos[2 * s + 1];
    g.w0 = A.w[s];
    for (int k = gr.lane; k < m; k += LANES)
        edge_line(A, C.r.id[k], g.c0x, g.c0y, g.w0, C.ax[k], C.ay[k], C.b[k]);
    __syncwarp(gr.mask);
    // vertex k: the intersection of edges k - 1 and k
    for (int k = gr.lane; k < m; k += LANES) {
        const int q = k == 0 ? m - 1 : k - 1;
        const double a1x = C.ax[q], a1y = C.ay[q], b1 = C.b[q], a2x = C.ax[k], a2y = C.ay[k], b2 = C.b[k];
        const double det = a1x * a2y - a1y * a2x;
        C.vx[k] = g.c0x + (b1 * a2y - b2 * a1y) / det;
        C.vy[k] = g.c0y + (a1x * b2 - a2x * b1) / det;
    }
    __syncwarp(gr.mask);
    // mass and centroid: fan from vertex 0 (add_centroid_contrib, ConvexPolyhedron2.tcc:1047-1074)
    double mass = 0, mx = 0, my = 0;
    for (int k = 2 + gr.lane; k < m; k += LANES) {
        const double ax = C.vx[0], ay = C.vy[0], bx = C.vx[k - 1], by = C.vy[k - 1], cx = C.vx[k], cy = C.vy[k];
        const double lea = 0.5 * (ax * (by - cy) + bx * (cy - ay) + cx * (ay - by)) * A.coeff;
        mx += lea * (1.0 / 3.0) * (ax + bx + cx);
        my += lea * (1.0 / 3.0) * (ay + by + cy);
        mass += lea;
    }
    mass = gr.sum(mass);
    mx = gr.sum(mx);
    my = gr.sum(my);
    g.mass = mass;
    g.cx = mass != 0 ? mx / mass : 0.0;
    g.cy = mass != 0 ? my / mass : 0.0;
    if (gr.lane < 3) {
        v[3 * i + gr.lane] = gr.lane == 0 ? g.cx : gr.lane == 1 ? g.cy : g.mass;
        off[3 * i + gr.lane] = base + 3LL * cnt * gr.lane;
    }
    // the diagonal: every edge's share
    double d0[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, t[9];
    for (int k = gr.lane; k < m; k += LANES)
        if (C.r.id[k] >= 0) edge_block(A, g, k, t, d0);
#pragma unroll
    for (int q = 0; q < 9; ++q) d0[q] = gr.sum(d0[q]);
    correct(g, d0);
    for (int k = gr.lane; k <= m; k += LANES) {
        const int c = C.r.head[k];
        if (c == INT_MAX) continue;
        double acc[9];
        if (k == m) {
            for (int q = 0; q < 9; ++q) acc[q] = d0[q];
        } else {
            edge_block(A, g, k, acc, nullptr);
            correct(g, acc);
        }
        int b = 0;  // its place: the columns before it
        for (int e = 0; e <= m; ++e) {
            b += C.r.head[e] < c;
            if (e <= k || C.r.col[e] != c) continue;
            if (e == m) {
                for (int q = 0; q < 9; ++q) t[q] = d0[q];
            } else {
                edge_block(A, g, e, t, nullptr);
                correct(g, t);
            }
            for (int q = 0; q < 9; ++q) acc[q] += t[q];
        }
        for (int d = 0; d < 3; ++d)
            for (int e = 0; e < 3; ++e) {
                const long long o = base + 3LL * cnt * d + 3 * b + e;
                cols[o] = 3LL * c + e;
                vals[o] = acc[3 * d + e];
            }
    }
}

}  // namespace

void derpos_count(const Rows &nb, long long n, const double *pos, const double *w, const int *idx, int start_n,
                  const double *start_xy, double coeff, int ntrans, const double *trans, long long *nblocks,
                  unsigned *err, cudaStream_t st) {
    if (n <= 0) return;
    const DpArgs A{nb, n, pos, w, idx, start_n, start_xy, coeff, ntrans, trans};
    k_dp_count<<<ceil_div(n, CELLS), TB, 0, st>>>(A, nblocks, err);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

void derpos_write(const Rows &nb, long long n, const double *pos, const double *w, const int *idx, int start_n,
                  const double *start_xy, double coeff, int ntrans, const double *trans, const long long *boff,
                  long long *off, long long *cols, double *vals, double *v, cudaStream_t st) {
    if (n <= 0) return;
    const DpArgs A{nb, n, pos, w, idx, start_n, start_xy, coeff, ntrans, trans};
    k_dp_write<<<ceil_div(n, CELLS), TB, 0, st>>>(A, boff, off, cols, vals, v);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

}  // namespace sdot
