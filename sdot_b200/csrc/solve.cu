// Preconditioned conjugate gradients on the device (see solve.cuh).
//
// Every reduction is two-stage with a fixed order (per-block partials, then
// one block sums them), so a solve is bitwise reproducible run to run.  The
// scalars of the iteration (alpha, beta, |r|^2) stay on the device; the host
// only reads |r|^2 every `check` iterations to decide to stop.
#include "solve.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace sdot {

namespace {

constexpr int TB = 256;
enum { S_RZ = 0, S_RR = 1, S_RR0 = 2, S_PQ = 3, S_ALPHA = 4, S_BETA = 5, S_GDIAG = 6, S_BAD = 7, S_NSCAL = 8 };
constexpr int S_ITER = S_PQ;  // the multilevel solve keeps p . q in registers and its iteration count here

__device__ double block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double r = 0;
    if (warp == 0) {
        r = lane < (blockDim.x >> 5) ? sh[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    __syncthreads();
    return r;  // valid in thread 0
}

// sum_k val_k f(col_k) over an ELL row, in order.  U entries are read at once,
// so that their latencies overlap (entry by entry a row is a chain of m loads
// of the column and then of the vector); the first U slots (the row has at
// least U, used or not) without waiting for the row's length.
template <int U, class V, class F>
__device__ __forceinline__ double ell_sum(const V *val, const int *col, long long stride, long long s, const int *cnt,
                                          int m, const F &f) {
    double acc = 0;
    int c[U];
    V v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (cnt || u < m) {
            c[u] = col[u * stride + s];
            v[u] = val[u * stride + s];
        }
    if (cnt) m = cnt[s];
#pragma unroll 1
    for (int k0 = 0; k0 < m; k0 += U) {
        if (k0 > 0) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k0 + u < m) {
                    c[u] = col[(k0 + u) * stride + s];
                    v[u] = val[(k0 + u) * stride + s];
                }
        }
        double x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k0 + u < m) x[u] = f(c[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k0 + u < m) acc += double(v[u]) * x[u];
    }
    return acc;
}

// Matrix views for the PCG kernels: row s times x, and the diagonal entry
// (sums in double whatever the precision of the values and vectors).
// RowsMatT: the Hessian rows (ELL + side buffer) with values of type V
// (rows.val itself, or an FP32 copy in the same layout).
template <class V>
struct RowsMatT {
    Rows R;
    const V *val;
    const V *side_val;
    template <class X>
    __device__ double row_dot(long long s, const X *x) const {
        const int m = R.cnt[s];
        double acc = 0;
        if (m <= R.cap) {
            for (int k = 0; k < m; ++k) acc += double(val[k * R.stride + s]) * double(x[R.col[k * R.stride + s]]);
        } else {
            const long long o = R.side[s];
            for (int k = 0; k < m; ++k) acc += double(side_val[o + k]) * double(x[R.side_col[o + k]]);
        }
        return acc;
    }
    __device__ int len(long long s) const { return R.cnt[s]; }
    __device__ long long colk(long long s, int k) const { return *R.colp(s, k); }
    __device__ double valk(long long s, int k) const {
        return R.cnt[s] > R.cap ? double(side_val[R.side[s] + k]) : double(val[k * R.stride + s]);
    }
    __device__ double diag(long long s) const {
        double d = 0;
        for (int k = 0, m = R.cnt[s]; k < m; ++k)
            if (colk(s, k) == s) d += valk(s, k);
        return d;
    }
    // sum_k a_sk f(col_sk)
    template <class F>
    __device__ double row_sum(long long s, const F &f) const {
        const int m = R.cnt[s];
        if (m <= R.cap) return ell_sum<4>(val, R.col, R.stride, s, R.cnt, m, f);
        const long long o = R.side[s];
        return ell_sum<2>(side_val + o, R.side_col + o, 1, 0, nullptr, m, f);
    }
};
using RowsMat = RowsMatT<double>;
inline RowsMat rows_mat(const Rows &R) { return RowsMat{R, R.val, R.side_val}; }

// The FP32 copy of the Hessian rows in Laplacian form: an off-diagonal entry
// holds the edge weight w_sj = -a_sj, the diagonal entry the row sum r_s (the
// part of the diagonal that is not the sum of the edge weights: disc arcs),
// so that (A x)_s = r_s x_s + sum_j w_sj (x_s - x_j).  Rounding the weights to
// FP32 then perturbs each edge by a relative 6e-8, which bounds the FP32
// operator between (1 -+ 6e-8) times the exact one; rounding the entries
// themselves would break the zero row sums by 6e-8 of the diagonal, far
// above the smallest eigenvalues of these systems.  Sums in double.
struct RowsLap32 {
    Rows R;
    const float *val;
    const float *side_val;
    __device__ int len(long long s) const { return R.cnt[s]; }
    __device__ long long colk(long long s, int k) const { return *R.colp(s, k); }
    __device__ double raw(long long s, int k) const {
        return R.cnt[s] > R.cap ? double(side_val[R.side[s] + k]) : double(val[k * R.stride + s]);
    }
    template <class F>
    __device__ double row_sum(long long s, const F &f) const {
        const int m = R.cnt[s];
        const double fs = f(s);
        double acc = 0;
        for (int k = 0; k < m; ++k) {
            const long long c = colk(s, k);
            acc += c == s ? raw(s, k) * fs : raw(s, k) * (fs - f(c));
        }
        return acc;
    }
    template <class X>
    __device__ double row_dot(long long s, const X *x) const {
        return row_sum(s, [&](long long j) { return double(x[j]); });
    }
    __device__ double diag(long long s) const {
        double d = 0;
        for (int k = 0, m = R.cnt[s]; k < m; ++k) d += raw(s, k);  // r_s + sum of the weights
        return d;
    }
    __device__ double valk(long long s, int k) const { return colk(s, k) == s ? diag(s) : -raw(s, k); }
};

struct CsrView {
    CsrMat M;
    template <class X>
    __device__ double row_dot(long long s, const X *x) const {
        double acc = 0;
        for (long long k = M.off[s], e = M.off[s + 1]; k < e; ++k) acc += M.val[k] * double(x[M.col[k]]);
        return acc;
    }
    __device__ double diag(long long s) const {
        double d = 0;
        for (long long k = M.off[s], e = M.off[s + 1]; k < e; ++k)
            if (M.col[k] == s) d += M.val[k];
        return d;
    }
    __device__ int len(long long s) const { return int(M.off[s + 1] - M.off[s]); }
    __device__ long long colk(long long s, int k) const { return M.col[M.off[s] + k]; }
    __device__ double valk(long long s, int k) const { return M.val[M.off[s] + k]; }
    template <class F>
    __device__ double row_sum(long long s, const F &f) const {
        double acc = 0;
        for (long long k = M.off[s], e = M.off[s + 1]; k < e; ++k) acc += M.val[k] * f(M.col[k]);
        return acc;
    }
};

// ---- multilevel preconditioner (one V-cycle per application) ------------
// Aggregates: consecutive rows (the rows are in Morton order, so an aggregate
// is a compact patch of cells), 4 of the finest level, MG_B of the others.
// Coarse matrices P^T A P / MG_SCALE with P piecewise constant on the
// aggregates, stored as ELL (width mg_cap); damped-Jacobi smoothing (MG_OMEGA)
// before and after the coarse correction; the coarsest level (<= MG_COARSE
// rows) is applied as its dense inverse.  Same smoother on both sides and
// symmetric coarse operators: the cycle is a symmetric positive operator (the
// smoother converges for MG_OMEGA < 1, the matrices being weighted graph
// Laplacians plus a diagonal), a valid CG preconditioner.
//
// Piecewise constant P makes the coarse matrices too stiff for smooth errors
// (over-correction: D. Braess, "Towards algebraic multigrid for elliptic
// problems of second order", Computing 55, 1995); 1.4 is the best of 1 to 2.2
// with 0.8 of 0.67 to 0.9.  CG iterations to 1e-12 on Voronoi Laplacians,
// 10,000 uniform / 30,000 clustered / 8,000 3D points: aggregates of 8, omega
// 0.67, no scaling 135 / 195 / 59; omega 0.8 and 1.4: 113 / 149 / 51; 4 at the
// finest level: 99 / 136 / 45; 4 at every level: 87 / 110 / 41, but twice the
// levels, each with two barriers of the grid.
constexpr int MG_BF = 4;         // rows of an aggregate of the finest level
constexpr int MG_B = 8;          // and of the coarse levels
constexpr int MG_CAP_MAX = 128;  // coarse ELL width: w.mg_cap (64 in 2D, 128 in 3D)
constexpr int MG_COARSE = 48;  // dense coarsest level: two 48 x 49 doubles in shared memory
constexpr double MG_OMEGA = 0.8;
constexpr double MG_SCALE = 1.4;

template <class V>
struct EllViewT {
    const int *cnt;
    const int *col;
    const V *val;
    long long stride;
    __device__ int len(long long s) const { return cnt[s]; }
    __device__ long long colk(long long s, int k) const { return col[k * stride + s]; }
    __device__ double valk(long long s, int k) const { return double(val[k * stride + s]); }
    template <class F>
    __device__ double row_sum(long long s, const F &f) const {
        return ell_sum<4>(val, col, stride, s, cnt, 0, f);
    }
};

template <class M, class T>
__global__ void k_diag_inv(M A, long long n, long long g, T *dinv, double *scal) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        double d = A.diag(s);
        if (s == g) {
            scal[S_GDIAG] = d;
            d *= 2;
        }
        dinv[s] = T(d != 0 ? 1.0 / d : 0.0);
    }
}

template <class T>
__global__ void k_init(const T *b, T *x, T *r, T *z, T *p, const T *dinv, double *partial, long long n) {
    __shared__ double sh[32];
    double rz = 0, rr = 0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        const T rv = b[s];
        const T zv = dinv[s] * rv;
        x[s] = 0;
        r[s] = rv;
        z[s] = zv;
        p[s] = zv;
        rz += double(rv) * double(zv);
        rr += double(rv) * double(rv);
    }
    rz = block_sum(rz, sh);
    rr = block_sum(rr, sh);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = rz;
        partial[gridDim.x + blockIdx.x] = rr;
    }
}

// mode 0: after init (rz, rr, rr0); 1: after spmv (pq -> alpha); 2: after update (rz_new, rr -> beta)
__global__ void k_final(const double *partial, int nb, double *scal, int mode) {
    __shared__ double sh[32];
    double a = 0, b = 0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        a += partial[i];
        b += partial[nb + i];
    }
    a = block_sum(a, sh);
    b = block_sum(b, sh);
    if (threadIdx.x == 0) {
        if (mode == 0) {
            scal[S_RZ] = a;
            scal[S_RR] = b;
            scal[S_RR0] = b;
            scal[S_BAD] = 0;
        } else if (mode == 1) {
            scal[S_PQ] = a;
            const double alpha = scal[S_RZ] / a;
            if (!(a > 0) || !isfinite(alpha)) scal[S_BAD] = 1;
            scal[S_ALPHA] = scal[S_BAD] != 0 ? 0.0 : alpha;
        } else {
            const double beta = a / scal[S_RZ];
            scal[S_BETA] = isfinite(beta) ? beta : 0.0;
            scal[S_RZ] = a;
            scal[S_RR] = b;
        }
    }
}

template <class M, class T>
__global__ void k_spmv(M A, long long n, long long g, const T *p, T *q, const double *scal, double *partial) {
    __shared__ double sh[32];
    double pq = 0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        double v = A.row_dot(s, p);
        if (s == g) v += scal[S_GDIAG] * double(p[s]);
        const T qv = T(v);
        q[s] = qv;
        pq += double(p[s]) * double(qv);
    }
    pq = block_sum(pq, sh);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = pq;
        partial[gridDim.x + blockIdx.x] = 0;
    }
}

template <class T>
__global__ void k_update(T *x, T *r, T *z, const T *p, const T *q, const T *dinv, const double *scal, double *partial,
                         long long n) {
    __shared__ double sh[32];
    const T alpha = T(scal[S_ALPHA]);
    double rz = 0, rr = 0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        x[s] += alpha * p[s];
        const T rv = r[s] - alpha * q[s];
        r[s] = rv;
        const T zv = dinv[s] * rv;
        z[s] = zv;
        rz += double(rv) * double(zv);
        rr += double(rv) * double(rv);
    }
    rz = block_sum(rz, sh);
    rr = block_sum(rr, sh);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = rz;
        partial[gridDim.x + blockIdx.x] = rr;
    }
}

template <class T>
__global__ void k_pupdate(const T *z, T *p, const double *scal, long long n) {
    const T beta = T(scal[S_BETA]);
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x)
        p[s] = z[s] + beta * p[s];
}

__global__ void k_mass_partial(const double *m, const double *t, long long n, double *partial) {
    __shared__ double sh[32];
    __shared__ double shmax[32], shmin[32];
    double mx = 0, mn = 1.0 / 0.0, ss = 0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        const double d = m[s] - t[s];
        mx = fmax(mx, fabs(d) / t[s]);
        mn = fmin(mn, m[s]);
        ss += d * d;
    }
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
        mn = fmin(mn, __shfl_down_sync(0xffffffffu, mn, o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        shmax[warp] = mx;
        shmin[warp] = mn;
    }
    ss = block_sum(ss, sh);
    if (threadIdx.x == 0) {
        for (int w = 1; w < (blockDim.x >> 5); ++w) {
            mx = fmax(mx, shmax[w]);
            mn = fmin(mn, shmin[w]);
        }
        partial[3 * blockIdx.x] = mx;
        partial[3 * blockIdx.x + 1] = mn;
        partial[3 * blockIdx.x + 2] = ss;
    }
}

__global__ void k_mass_final(const double *partial, int nb, double *out) {
    if (threadIdx.x != 0) return;
    double mx = 0, mn = 1.0 / 0.0, ss = 0;
    for (int b = 0; b < nb; ++b) {
        mx = fmax(mx, partial[3 * b]);
        mn = fmin(mn, partial[3 * b + 1]);
        ss += partial[3 * b + 2];
    }
    out[0] = mx;
    out[1] = mn;
    out[2] = ss;
}

__global__ void k_axpby(const double *a, const double *b, double *out, double alpha, double beta, long long n) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x)
        out[s] = alpha * a[s] + beta * b[s];
}

__global__ void k_apply_step(const double *w_base, const double *d, const int *idx, double tau, double *w_out,
                             long long n) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        const int i = idx[s];
        w_out[i] = w_base[i] - tau * d[s];
    }
}

__global__ void k_gather_sorted(const double *t, const int *idx, double *out, long long n) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x)
        out[s] = t[idx[s]];
}

// One warp per coarse row c: the entries of fine rows c*B .. c*B+B-1, in
// row order then stored order, are merged by coarse column into a table of
// 32 SLOTS entries (SLOTS per lane), so the sums have a fixed order.  The
// gauge term of the fine level joins the coarse diagonal.  A row with more
// than 32 SLOTS coarse columns sets *flag (the solve falls back to Jacobi).
template <class M, int SLOTS, int B, class T>
__global__ void k_mg_coarsen(M A, long long nf, long long gauge, const double *scal, MgLevelT<T> out, int *flag) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long c = warp; c < out.n; c += nwarps) {
        int key[SLOTS], count = 0;
        double v[SLOTS];
#pragma unroll
        for (int q = 0; q < SLOTS; ++q) {
            key[q] = -1;
            v[q] = 0;
        }
        bool over = false;
        auto insert = [&](int cc, double x) {
            bool found = false;
#pragma unroll
            for (int q = 0; q < SLOTS; ++q) {
                const unsigned m = __ballot_sync(FULL, key[q] == cc);
                if (!found && m) {
                    if (lane == __ffs(int(m)) - 1) v[q] += x;
                    found = true;
                }
            }
            if (found) return;
            if (count < 32 * SLOTS) {
                if (lane == (count & 31)) {
#pragma unroll
                    for (int q = 0; q < SLOTS; ++q)
                        if (q == (count >> 5)) {
                            key[q] = cc;
                            v[q] = x;
                        }
                }
                ++count;
            } else {
                over = true;
            }
        };
        for (int r = 0; r < B; ++r) {
            const long long s = c * B + r;
            if (s >= nf) break;
            const int len = A.len(s);
            for (int k = 0; k < len; ++k) insert(int(A.colk(s, k) / B), A.valk(s, k));
            if (s == gauge) insert(int(c), scal[S_GDIAG]);
        }
        double diag = 0;
#pragma unroll
        for (int q = 0; q < SLOTS; ++q)
            if (lane + 32 * q < count) {
                out.col[(lane + 32 * q) * out.n + c] = key[q];
                v[q] *= 1.0 / MG_SCALE;
                out.val[(lane + 32 * q) * out.n + c] = T(v[q]);
                if (key[q] == c) diag = v[q];
            }
        for (int o = 16; o > 0; o >>= 1) diag += __shfl_xor_sync(FULL, diag, o);
        if (lane == 0) {
            out.cnt[c] = count;
            out.dinv[c] = T(diag > 0 ? 1.0 / diag : 0.0);
            if (over) atomicExch(flag, 1);
        }
    }
}

// Dense inverse of the coarsest level (nc <= MG_COARSE rows, one block of
// MG_COARSE threads, thread t owns row t).  Gauss-Jordan without pivoting
// (the matrix is symmetric positive semi-definite); a pivot below 1e-13 of
// the largest diagonal entry marks a null direction, left out of the inverse.
template <class V>
__global__ void k_mg_coarsest_setup(EllViewT<V> A, int nc, double *cinv) {
    __shared__ double M[MG_COARSE][MG_COARSE + 1], I[MG_COARSE][MG_COARSE + 1];
    __shared__ double dmax;
    const int t = threadIdx.x;
    if (t < nc) {
        for (int c = 0; c < nc; ++c) {
            M[t][c] = 0;
            I[t][c] = c == t ? 1.0 : 0.0;
        }
        for (int k = 0, m = A.cnt[t]; k < m; ++k) M[t][A.col[k * A.stride + t]] += double(A.val[k * A.stride + t]);
    }
    __syncthreads();
    if (t == 0) {
        double d = 0;
        for (int c = 0; c < nc; ++c) d = fmax(d, M[c][c]);
        dmax = d;
    }
    __syncthreads();
    for (int k = 0; k < nc; ++k) {
        const double piv = M[k][k];
        const bool ok = piv > 1e-13 * dmax;
        __syncthreads();
        if (t == k) {
            const double inv = ok ? 1.0 / piv : 0.0;
            for (int c = 0; c < nc; ++c) {
                M[k][c] *= inv;
                I[k][c] *= inv;
            }
        }
        __syncthreads();
        if (t < nc && t != k && ok) {
            const double f = M[t][k];
            for (int c = 0; c < nc; ++c) {
                M[t][c] -= f * M[k][c];
                I[t][c] -= f * I[k][c];
            }
        }
        __syncthreads();
    }
    if (t < nc)
        for (int c = 0; c < nc; ++c) cinv[t * nc + c] = I[t][c];
}

// CG start for the multilevel preconditioner: x = 0, r = b, s = omega D^-1 r;
// the vectors of a previous iteration are zero.
template <class T>
__global__ void k_init_mg(const T *b, T *x, T *r, T *s, const T *dinv, T *p, T *q, T *qs, T *z, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const T rv = b[i];
        x[i] = p[i] = q[i] = qs[i] = z[i] = 0;
        r[i] = rv;
        s[i] = T(MG_OMEGA * double(dinv[i]) * double(rv));
    }
}

int grid_of(long long n) {
    long long g = (n + TB - 1) / TB;
    return int(g < PCG_BLOCKS ? (g < 1 ? 1 : g) : PCG_BLOCKS);
}

}  // namespace

size_t pcg_work_doubles(long long n) { return size_t(5) * (n + 32) + 6 * PCG_BLOCKS + S_NSCAL + 64; }

namespace {

constexpr int MG_MAX_LEV = 16;

template <class T>
struct MgPlan {
    int L = 0;                        // coarse levels 1..L (level L is the coarsest)
    MgLevelT<double> lev[MG_MAX_LEV + 1];  // lev[0]: the fine level (n only); coarse levels in FP64
    double *cinv = nullptr;           // coarsest dense inverse
    int *flag = nullptr;              // coarse-row overflow
    unsigned *sync = nullptr;         // the solve's grid barrier: arrivals, given up
    T *s0 = nullptr, *s1 = nullptr, *qs = nullptr, *p1 = nullptr;  // vectors beside PcgWorkT's
};

// Carves the levels of an n-row solve out of `base` (null: sizes only);
// returns the doubles used.
template <class T>
size_t mg_plan(long long n, int cap, double *base, MgPlan<T> &pl) {
    auto pad = [](size_t k) { return (k + 31) & ~size_t(31); };
    size_t used = 0;
    // room for `count` elements of type E, in doubles
    auto take = [&](size_t count, auto *type) {
        using E = std::remove_pointer_t<decltype(type)>;
        E *p = base ? reinterpret_cast<E *>(base + used) : nullptr;
        used += pad((count * sizeof(E) + sizeof(double) - 1) / sizeof(double));
        return p;
    };
    pl = MgPlan<T>{};
    pl.lev[0].n = n;
    long long m = n;
    while (m > MG_COARSE && pl.L < MG_MAX_LEV) {
        const int ag = pl.L == 0 ? MG_BF : MG_B;
        m = (m + ag - 1) / ag;
        MgLevelT<double> &v = pl.lev[++pl.L];
        v.n = m;
        v.val = take(size_t(cap) * m, (double *)nullptr);
        v.dinv = take(m, (double *)nullptr);
        v.r = take(m, (double *)nullptr);
        v.zo = take(m, (double *)nullptr);
        v.cnt = take(m, (int *)nullptr);
        v.col = take(size_t(cap) * m, (int *)nullptr);
    }
    if (pl.L > 0) {
        pl.cinv = take(size_t(MG_COARSE) * MG_COARSE, (double *)nullptr);
        pl.flag = take(1, (int *)nullptr);
        pl.sync = take(2, (unsigned *)nullptr);
        pl.s0 = take(n, (T *)nullptr);
        pl.s1 = take(n, (T *)nullptr);
        pl.qs = take(n, (T *)nullptr);
        pl.p1 = take(n, (T *)nullptr);
    }
    return used;
}

int coarse_grid(long long n) {
    long long g = (n + TB - 1) / TB;
    return int(g < 148 * 8 ? (g < 1 ? 1 : g) : 148 * 8);
}

inline EllViewT<double> ell(const MgLevelT<double> &v) { return EllViewT<double>{v.cnt, v.col, v.val, v.n}; }

// Builds the coarse levels of A; false when a coarse row outgrew MG_CAP.
template <class M, int SLOTS, class T>
void mg_coarsen_all(const M &A, long long gauge, const double *scal, const MgPlan<T> &pl, cudaStream_t st) {
    for (int l = 1; l <= pl.L; ++l) {
        const int g = coarse_grid(32 * pl.lev[l].n);  // one warp per coarse row
        if (l == 1)
            k_mg_coarsen<M, SLOTS, MG_BF, double><<<g, TB, 0, st>>>(A, pl.lev[0].n, gauge, scal, pl.lev[1], pl.flag);
        else
            k_mg_coarsen<EllViewT<double>, SLOTS, MG_B, double><<<g, TB, 0, st>>>(ell(pl.lev[l - 1]), pl.lev[l - 1].n, -1, scal,
                                                                  pl.lev[l], pl.flag);
        note_launch();
    }
}

template <class M, class T>
bool mg_setup(const M &A, long long gauge, const double *scal, const MgPlan<T> &pl, int cap, cudaStream_t st) {
    SDOT_CUDA(cudaMemsetAsync(pl.flag, 0, sizeof(int), st));
    if (cap > 64)
        mg_coarsen_all<M, 4>(A, gauge, scal, pl, st);
    else
        mg_coarsen_all<M, 2>(A, gauge, scal, pl, st);
    k_mg_coarsest_setup<double><<<1, MG_COARSE, 0, st>>>(ell(pl.lev[pl.L]), int(pl.lev[pl.L].n), pl.cinv);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
    int flag = 0;
    SDOT_CUDA(cudaMemcpyAsync(&flag, pl.flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    SDOT_CUDA(cudaStreamSynchronize(st));
    return flag == 0;
}

}  // namespace

size_t mg_work_doubles(long long n, int cap) {
    MgPlan<double> pl;
    return mg_plan(n, cap, nullptr, pl);
}

template <class T>
void pcg_bind(PcgWorkT<T> &w, double *base, long long n) {
    const long long m = n + 32;
    T *v = reinterpret_cast<T *>(base);
    w.r = v;
    w.z = v + m;
    w.p = v + 2 * m;
    w.q = v + 3 * m;
    w.dinv = v + 4 * m;
    w.partial = base + (5 * m * (long long)sizeof(T) + 7) / 8;
    w.scal = w.partial + 6 * PCG_BLOCKS;
}
template void pcg_bind<double>(PcgWorkT<double> &, double *, long long);
template void pcg_bind<float>(PcgWorkT<float> &, double *, long long);

namespace {

// ---- the whole solve in one kernel -----------------------------------------
// As launches, an iteration of multilevel CG is 13 to 16 kernels of 3 to 20 us
// at 10,000 to 60,000 rows, most of it their latency.  Here the blocks
// stay for up to `iters` iterations (a cooperative launch: every block is
// resident) and meet at grid barriers:
//   A  p = z + beta p_old; q = A p, qs = omega D^-1 q; p . q       | barrier
//   B  x += alpha p; r -= alpha q; s = s_old - alpha qs (= omega D^-1 r);
//      |r|^2; coarse right-hand side sum (r - A s)                 | barrier
//   C  coarse levels above SOLO rows: one barrier a level and direction; the
//      rest by one block, its vectors in shared memory             | barrier
//   D  z' = s + P zc, z = z' + omega D^-1 (r - A z'); r . z        | barrier
// The vector updates are folded into the passes over the matrix: what a row
// needs of its neighbours' new values it computes from the old ones (hence two
// copies of p and s).  Sums go by block partials that every block adds in one
// order, so that all blocks take the same decisions and a solve repeats bit
// for bit.  The barrier gives up after a bounded wait (the solve then ends as
// not converged).
//
// One thread per row.  Measured per iteration (launches of the phases in a CUDA
// graph -> this kernel): 10,000 rows 45 -> 29 us, 60,000 70 -> 45, 20,000 3D
// rows 80 -> 51; about 2 us of each are a barrier, 1 to 4 us a phase (two
// dependent reads of the L2 and the block's sum).  Blocks of 128, 256, 512
// threads: 32 / 29 / 35 us and 59 / 45 / 52 us.  A hardware cluster of 16
// blocks has a barrier of 0.7 us, but its 16 SMs take 8 us for a phase of 10,000
// rows.  From several 100,000 rows on the passes are bound by the loads in flight
// and blocks of 512 pay (Newton at 300,000 / 500,000 / 1M rows, 1M clamped
// clusters: 0.142 / 0.255 / 1.53 / 1.86 s; with 256 0.132 / 0.280 / 1.85 / 2.17;
// two blocks of 256 per SM - / 0.278 / 1.61 / 2.16; more of them spill).
constexpr int MGT = 256;
constexpr int MGT_MANY = 512;
constexpr long long MANY_ROWS = 400000;
constexpr int SOLO = 512;       // rows of the largest level one block does alone
constexpr int SOLO_ALL = 640;   // rows of all such levels together (512 + 64 + 8, and a margin)

template <class M, class T>
struct PcgArgs {
    M A;
    long long n, gauge;
    MgPlan<T> pl;
    const T *dinv;
    T *x, *r, *s[2], *q, *qs, *p[2], *z;
    double *scal, *partial;
    double rel2;  // square of the relative tolerance
    int iters;
    int first;    // 1: starts a solve; 0: goes on from scal
};

// Sum of the blocks' partials, the same in every thread of every block.
__device__ double grid_sum(const double *partial, double *sh) {
    double a = 0;
    for (int i = threadIdx.x; i < int(gridDim.x); i += blockDim.x) a += partial[i];
    a = block_sum(a, sh);
    if (threadIdx.x == 0) sh[0] = a;
    __syncthreads();
    a = sh[0];
    __syncthreads();
    return a;
}

// r - A z of row i with z_j = f(j); the aggregate's sum of it to rc (whole
// warps call this: rows past n give 0)
template <int B>
__device__ void restrict_row(double t, long long i, long long n, double *rc) {
    for (int o = B / 2; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o, B);
    if ((threadIdx.x & (B - 1)) == 0 && i < n) rc[i / B] = t;
}

// The phases.  Each is a function of its own: in one body the compiler keeps
// the addresses of all of them in registers and spills inside the loops (1.6 KB
// a thread; the barriers empty the L1 cache that would hold them), and they take
// the block's size at run time: compiled for each size, with more registers for
// the smaller, they took 4% longer at 10,000 rows.
template <class M, class T>
__device__ __noinline__ double phase_a(const PcgArgs<M, T> &a, const T *pold, T *pnew, double beta, double gd) {
    const int nt = blockDim.x;
    const long long step = (long long)gridDim.x * nt;
    auto pv = [&](long long j) { return double(T(double(a.z[j]) + beta * double(pold[j]))); };
    double pq = 0;
    for (long long i = blockIdx.x * (long long)nt + threadIdx.x; i < a.n; i += step) {
        const double pi = pv(i);
        double v = a.A.row_sum(i, pv);
        if (i == a.gauge) v += gd * pi;
        const T qv = T(v);
        pnew[i] = T(pi);
        a.q[i] = qv;
        a.qs[i] = T(MG_OMEGA * double(a.dinv[i]) * double(qv));
        pq += pi * double(qv);
    }
    return pq;
}

template <class M, class T>
__device__ __noinline__ double phase_b(const PcgArgs<M, T> &a, const T *p, const T *sold, T *snew, double alpha,
                                       double gd, bool update) {
    const int nt = blockDim.x;
    const long long step = (long long)gridDim.x * nt;
    auto sv = [&](long long j) { return double(T(double(sold[j]) - alpha * double(a.qs[j]))); };
    double rs = 0;
    for (long long i0 = blockIdx.x * (long long)nt; i0 < a.n; i0 += step) {
        const long long i = i0 + threadIdx.x;
        double t = 0;
        if (i < a.n) {
            T rv = a.r[i];
            if (update) {
                a.x[i] += T(alpha) * p[i];
                rv = T(double(rv) - alpha * double(a.q[i]));
                a.r[i] = rv;
            }
            const double si = sv(i);
            snew[i] = T(si);
            double v = a.A.row_sum(i, sv);
            if (i == a.gauge) v += gd * si;
            t = double(rv) - v;
            rs += double(rv) * double(rv);
        }
        restrict_row<MG_BF>(t, i, a.n, a.pl.lev[1].r);
    }
    return rs;
}

template <class M, class T>
__device__ __noinline__ double phase_d(const PcgArgs<M, T> &a, const T *s, double gd) {
    const int nt = blockDim.x;
    const long long step = (long long)gridDim.x * nt;
    const double *zc = a.pl.lev[1].zo;
    auto zv = [&](long long j) { return double(s[j]) + zc[j / MG_BF]; };
    double rs = 0;
    for (long long i = blockIdx.x * (long long)nt + threadIdx.x; i < a.n; i += step) {
        const double zi = zv(i), ri = double(a.r[i]);
        double v = a.A.row_sum(i, zv);
        if (i == a.gauge) v += gd * zi;
        const T zo = T(zi + MG_OMEGA * double(a.dinv[i]) * (ri - v));
        a.z[i] = zo;
        rs += ri * double(zo);
    }
    return rs;
}

// Smoothing and restriction of a coarse level (right-hand side r, the sums to
// rc), rows i0 + threadIdx.x of every step-th block of rows from i0
__device__ __noinline__ void coarse_down(const EllViewT<double> A, int n, const double *dinv, const double *r, double *rc,
                                         int i0, int step) {
    for (; i0 < n; i0 += step) {
        const int i = i0 + threadIdx.x;
        double t = 0;
        if (i < n) t = r[i] - A.row_sum(i, [&](long long j) { return MG_OMEGA * dinv[j] * r[j]; });
        restrict_row<MG_B>(t, i, n, rc);
    }
}

// Coarse correction zc and smoothing of a coarse level, into zo
__device__ __noinline__ void coarse_up(const EllViewT<double> A, int n, const double *dinv, const double *r,
                                       const double *zc, double *zo, int i0, int step) {
    auto zv = [&](long long j) { return MG_OMEGA * dinv[j] * r[j] + zc[j / MG_B]; };
    for (int i = i0 + threadIdx.x; i < n; i += step)
        zo[i] = zv(i) + MG_OMEGA * dinv[i] * (r[i] - A.row_sum(i, zv));
}

// Levels [solo, L] by one block, their vectors in shared memory.
struct SoloMem {
    double r[SOLO_ALL], z[SOLO_ALL], dinv[SOLO_ALL];
    double cinv[MG_COARSE * MG_COARSE];
};
template <class T>
__device__ __noinline__ void coarse_solo(const MgPlan<T> &pl, int solo, SoloMem &S) {
    double *sr = S.r, *sz = S.z;
    const int tid = threadIdx.x, nt = blockDim.x, L = pl.L;
    const int n0 = int(pl.lev[solo].n);
    for (int i = tid; i < n0; i += nt) sr[i] = pl.lev[solo].r[i];
    __syncthreads();
    int at = 0;
    for (int l = solo; l < L; ++l) {
        const MgLevelT<double> &v = pl.lev[l];
        const double *r = sr + at, *dinv = S.dinv + at;
        const int nl = int(v.n);
        const EllViewT<double> A{v.cnt, v.col, v.val, v.n};
        at += nl;
        for (int i0 = 0; i0 < nl; i0 += nt) {
            const int i = i0 + tid;
            double t = 0;
            if (i < nl) t = r[i] - A.row_sum(i, [&](long long j) { return MG_OMEGA * dinv[j] * r[j]; });
            restrict_row<MG_B>(t, i, nl, sr + at);
        }
        __syncthreads();
    }
    const int nc = int(pl.lev[L].n);
    if (tid < nc) {
        double acc = 0;
        for (int c = 0; c < nc; ++c) acc += S.cinv[c * nc + tid] * sr[at + c];
        sz[at + tid] = acc;
    }
    __syncthreads();
    for (int l = L - 1; l >= solo; --l) {
        const MgLevelT<double> &v = pl.lev[l];
        const int nl = int(v.n);
        const double *zc = sz + at;
        at -= nl;
        const double *r = sr + at, *dinv = S.dinv + at;
        const EllViewT<double> A{v.cnt, v.col, v.val, v.n};
        auto zv = [&](long long j) { return MG_OMEGA * dinv[j] * r[j] + zc[j / MG_B]; };
        for (int i = tid; i < nl; i += nt) sz[at + i] = zv(i) + MG_OMEGA * dinv[i] * (r[i] - A.row_sum(i, zv));
        __syncthreads();
    }
    for (int i = tid; i < n0; i += nt) pl.lev[solo].zo[i] = sz[i];
}

template <class M, class T, int NT>
__global__ void __launch_bounds__(NT, 1) k_pcg_mg(const __grid_constant__ PcgArgs<M, T> param) {
    __shared__ double sh[33];
    __shared__ SoloMem solo_mem;
    // the arguments in shared memory: read through the L1 cache, which the
    // barriers empty, each use of a pointer would wait for the L2 first
    using Args = PcgArgs<M, T>;
    static_assert(sizeof(Args) % 8 == 0, "copied by 8 bytes");
    __shared__ double arg_mem[sizeof(Args) / 8];
    for (int i = threadIdx.x; i < int(sizeof(Args) / 8); i += NT)
        arg_mem[i] = reinterpret_cast<const double *>(&param)[i];
    const Args &a = *reinterpret_cast<const Args *>(arg_mem);
    __syncthreads();
    const int tid = threadIdx.x, L = a.pl.L, t0 = blockIdx.x * NT, step = gridDim.x * NT;
    const double gd = a.gauge >= 0 ? a.scal[S_GDIAG] : 0.0;
    double *p_pq = a.partial, *p_rr = a.partial + gridDim.x, *p_rz = a.partial + 2 * gridDim.x;
    // the levels [solo, L] are one block's
    int solo = L;
    while (solo > 1 && a.pl.lev[solo - 1].n <= SOLO) --solo;
    if (blockIdx.x == 0) {
        const int nc = int(a.pl.lev[L].n);
        for (int i = tid; i < nc * nc; i += NT) solo_mem.cinv[i] = a.pl.cinv[i];
        int at = 0;
        for (int l = solo; l < L; at += int(a.pl.lev[l].n), ++l)
            for (int i = tid; i < int(a.pl.lev[l].n); i += NT) solo_mem.dinv[at + i] = a.pl.lev[l].dinv[i];
        __syncthreads();
    }
    unsigned target = 0;
    bool first = a.first != 0, bad = false;
    double rz = first ? 0 : a.scal[S_RZ], beta = first ? 0 : a.scal[S_BETA], rr0 = first ? 0 : a.scal[S_RR0];
    double rr = 0, alpha = 0;
    int done = first ? 0 : int(a.scal[S_ITER]);
    const int last = done + a.iters;
    int cur = first ? 0 : (done + 1) & 1;  // the copy of s that holds the current one (and of p, the last one)
    // the block's share of a sum to every block's total; false: waits given up
    auto total = [&](double &v, double *partial) {
        v = block_sum(v, sh);
        if (tid == 0) partial[blockIdx.x] = v;
        if (!grid_barrier(a.pl.sync, target)) return false;
        v = grid_sum(partial, sh);
        return true;
    };
    while (true) {
        bad = true;
        if (!first) {
            if (done >= last) {
                bad = false;
                break;
            }
            double pq = phase_a(a, a.p[cur], a.p[cur ^ 1], beta, gd);
            if (!total(pq, p_pq)) break;
            alpha = rz / pq;
            if (!(pq > 0) || !isfinite(alpha)) break;
        }
        rr = phase_b(a, a.p[cur ^ 1], a.s[cur], a.s[cur ^ 1], alpha, gd, !first);
        if (!total(rr, p_rr)) break;
        cur ^= 1;
        if (first)
            rr0 = rr;
        else
            ++done;
        if (!(rr > a.rel2 * rr0)) {  // reached, or not a number
            bad = false;
            break;
        }
        bool lost = false;
        for (int l = 1; l < solo && !lost; ++l) {
            const MgLevelT<double> &v = a.pl.lev[l];
            coarse_down(EllViewT<double>{v.cnt, v.col, v.val, v.n}, int(v.n), v.dinv, v.r, a.pl.lev[l + 1].r, t0, step);
            lost = !grid_barrier(a.pl.sync, target);
        }
        if (lost) break;
        if (blockIdx.x == 0) coarse_solo(a.pl, solo, solo_mem);
        lost = !grid_barrier(a.pl.sync, target);
        for (int l = solo - 1; l >= 1 && !lost; --l) {
            const MgLevelT<double> &v = a.pl.lev[l];
            coarse_up(EllViewT<double>{v.cnt, v.col, v.val, v.n}, int(v.n), v.dinv, v.r, a.pl.lev[l + 1].zo, v.zo, t0, step);
            lost = !grid_barrier(a.pl.sync, target);
        }
        if (lost) break;
        double rzn = phase_d(a, a.s[cur], gd);
        if (!total(rzn, p_rz)) break;
        beta = first ? 0.0 : rzn / rz;
        if (!isfinite(beta)) beta = 0;
        rz = rzn;
        first = false;
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.scal[S_RZ] = rz;
        a.scal[S_BETA] = beta;
        a.scal[S_RR] = rr;
        a.scal[S_RR0] = rr0;
        a.scal[S_ITER] = done;
        a.scal[S_BAD] = bad ? 1.0 : 0.0;
    }
}

template <class M, class T>
PcgResult pcg_run_mg(const M &A, long long n, long long gauge_row, const T *b, T *x, double rel_tol, int max_iter,
                     const PcgWorkT<T> &w, const MgPlan<T> &pl, cudaStream_t st, int check, int stall_checks) {
    PcgResult res;
    res.levels = pl.L;
    int sms = 0, dev = 0;
    SDOT_CUDA(cudaGetDevice(&dev));
    SDOT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool many = n > MANY_ROWS;
    const int nt = many ? MGT_MANY : MGT;
    void (*const kernel)(PcgArgs<M, T>) = many ? k_pcg_mg<M, T, MGT_MANY> : k_pcg_mg<M, T, MGT>;
    // all blocks are resident: one per SM
    const int g = int(std::min<long long>((n + nt - 1) / nt, std::min(sms, 2 * PCG_BLOCKS)));
    k_init_mg<T><<<grid_of(n), TB, 0, st>>>(b, x, w.r, pl.s0, w.dinv, pl.p1, w.q, pl.qs, w.z, n);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
    PcgArgs<M, T> a{A, n, gauge_row, pl, w.dinv, x, w.r, {pl.s0, pl.s1}, w.q, pl.qs, {w.p, pl.p1}, w.z, w.scal, w.partial,
                    rel_tol * rel_tol, 0, 1};
    double hs[S_NSCAL] = {0}, hist[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int nchecks = 0;
    // a launch runs until the tolerance is met or for this many iterations, so
    // that no kernel holds the device for long
    const int chunk = stall_checks > 0 ? check : 256;
    for (int it = 0;;) {
        a.iters = std::min(chunk, max_iter - it);
        SDOT_CUDA(cudaMemsetAsync(pl.sync, 0, 2 * sizeof(unsigned), st));
        void *args[] = {&a};
        SDOT_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(kernel), dim3(g), dim3(nt), args, 0, st));
        note_launch();
        SDOT_CUDA(cudaMemcpyAsync(hs, w.scal, sizeof(hs), cudaMemcpyDeviceToHost, st));
        SDOT_CUDA(cudaStreamSynchronize(st));
        a.first = 0;
        it = int(hs[S_ITER]);
        if (hs[S_BAD] != 0 || !(hs[S_RR] == hs[S_RR])) break;
        if (hs[S_RR] <= a.rel2 * hs[S_RR0]) {
            res.converged = true;
            break;
        }
        if (it >= max_iter) break;
        if (stall_checks > 0) {
            const int k = stall_checks < 8 ? stall_checks : 8;
            if (nchecks >= k && !(hs[S_RR] <= 0.5 * hist[(nchecks - k) % 8])) break;
            hist[nchecks % 8] = hs[S_RR];
            ++nchecks;
        }
    }
    res.iterations = int(hs[S_ITER]);
    if (hs[S_RR0] == 0) {
        res.converged = true;
        return res;
    }
    res.rel_residual = std::sqrt(hs[S_RR] / hs[S_RR0]);
    if (res.rel_residual <= rel_tol) res.converged = true;
    return res;
}

// stall_checks > 0: also stop once |r|^2 has not halved over the last
// stall_checks checks (the inner FP32 solves, whose attainable accuracy ends
// above the tolerance on ill-conditioned systems).
template <class M, class T>
PcgResult pcg_run(const M &A, long long n, long long gauge_row, const T *b, T *x, double rel_tol, int max_iter,
                  const PcgWorkT<T> &w, cudaStream_t st, int check, bool graph, bool multilevel,
                  int stall_checks = 0) {
    PcgResult res;
    if (n <= 0) {
        res.converged = true;
        return res;
    }
    const int g = grid_of(n);
    k_diag_inv<M, T><<<g, TB, 0, st>>>(A, n, gauge_row, w.dinv, w.scal);
    note_launch();
    MgPlan<T> pl;
    const int cap = w.mg_cap > 64 ? MG_CAP_MAX : 64;
    const bool mg = multilevel && n > MG_COARSE && w.mg && mg_plan(n, cap, nullptr, pl) <= w.mg_doubles;
    if (mg) {
        mg_plan(n, cap, w.mg, pl);
        if constexpr (!std::is_same_v<M, CsrView>)  // CSR solves are Jacobi's
            if (mg_setup(A, gauge_row, w.scal, pl, cap, st))
                return pcg_run_mg(A, n, gauge_row, b, x, rel_tol, max_iter, w, pl, st, check, stall_checks);
    }
    k_init<T><<<g, TB, 0, st>>>(b, x, w.r, w.z, w.p, w.dinv, w.partial, n);
    note_launch();
    k_final<<<1, TB, 0, st>>>(w.partial, g, w.scal, 0);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
    double hs[S_NSCAL];
    SDOT_CUDA(cudaMemcpyAsync(hs, w.scal, sizeof(hs), cudaMemcpyDeviceToHost, st));
    SDOT_CUDA(cudaStreamSynchronize(st));
    const double rr0 = hs[S_RR0];
    if (rr0 == 0) {
        res.converged = true;
        return res;
    }
    const double target = rel_tol * rel_tol * rr0;
    auto launch_chunk = [&](int chunk) {
        for (int c = 0; c < chunk; ++c) {
            k_spmv<M, T><<<g, TB, 0, st>>>(A, n, gauge_row, w.p, w.q, w.scal, w.partial);
            k_final<<<1, TB, 0, st>>>(w.partial, g, w.scal, 1);
            k_update<T><<<g, TB, 0, st>>>(x, w.r, w.z, w.p, w.q, w.dinv, w.scal, w.partial, n);
            k_final<<<1, TB, 0, st>>>(w.partial, g, w.scal, 2);
            k_pupdate<T><<<g, TB, 0, st>>>(w.z, w.p, w.scal, n);
        }
    };
    const int per_iter = 5;
    // With `graph`, a full chunk of iterations is captured once as a CUDA
    // graph and replayed: one launch instead of 5 * check.
    cudaGraphExec_t exec = nullptr;
    struct ExecGuard {
        cudaGraphExec_t &e;
        ~ExecGuard() {
            if (e) cudaGraphExecDestroy(e);
        }
    } exec_guard{exec};
    if (graph && max_iter >= check) {
        cudaGraph_t gr = nullptr;
        SDOT_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        launch_chunk(check);
        const cudaError_t le = cudaGetLastError();
        const cudaError_t ce = cudaStreamEndCapture(st, &gr);
        SDOT_CUDA(le);
        SDOT_CUDA(ce);
        const cudaError_t ie = cudaGraphInstantiate(&exec, gr, 0);
        cudaGraphDestroy(gr);
        SDOT_CUDA(ie);
    }
    int it = 0;
    double hist[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int nchecks = 0;
    while (it < max_iter) {
        const int chunk = check < max_iter - it ? check : max_iter - it;
        if (exec && chunk == check)
            SDOT_CUDA(cudaGraphLaunch(exec, st));
        else
            launch_chunk(chunk);
        for (int c = 0; c < per_iter * chunk; ++c) note_launch();
        SDOT_CUDA(cudaGetLastError());
        it += chunk;
        SDOT_CUDA(cudaMemcpyAsync(hs, w.scal, sizeof(hs), cudaMemcpyDeviceToHost, st));
        SDOT_CUDA(cudaStreamSynchronize(st));
        if (hs[S_BAD] != 0 || !(hs[S_RR] == hs[S_RR])) break;
        if (hs[S_RR] <= target) {
            res.converged = true;
            break;
        }
        if (stall_checks > 0) {
            const int k = stall_checks < 8 ? stall_checks : 8;
            if (nchecks >= k && !(hs[S_RR] <= 0.5 * hist[(nchecks - k) % 8])) break;
            hist[nchecks % 8] = hs[S_RR];
            ++nchecks;
        }
    }
    res.iterations = it;
    res.rel_residual = std::sqrt(hs[S_RR] / rr0);
    if (res.rel_residual <= rel_tol) res.converged = true;
    return res;
}

}  // namespace

PcgResult pcg_solve(const Rows &rows, long long n, long long gauge_row, const double *b, double *x, double rel_tol,
                    int max_iter, const PcgWork &w, cudaStream_t st, int check, bool graph, bool multilevel) {
    return pcg_run(rows_mat(rows), n, gauge_row, b, x, rel_tol, max_iter, w, st, check, graph, multilevel);
}

PcgResult pcg_solve_csr(const CsrMat &A, long long n, long long gauge_row, const double *b, double *x, double rel_tol,
                        int max_iter, const PcgWork &w, cudaStream_t st, int check) {
    return pcg_run(CsrView{A}, n, gauge_row, b, x, rel_tol, max_iter, w, st, check, false, false);
}

void mass_errors(const double *m, const double *t, long long n, double *partial, double *out, cudaStream_t st) {
    const int g = grid_of(n);
    k_mass_partial<<<g, TB, 0, st>>>(m, t, n, partial);
    note_launch();
    k_mass_final<<<1, 32, 0, st>>>(partial, g, out);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

void axpby(const double *a, const double *b, double *out, double alpha, double beta, long long n, cudaStream_t st) {
    k_axpby<<<grid_of(n), TB, 0, st>>>(a, b, out, alpha, beta, n);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

void apply_step(const double *w_base, const double *d_sorted, const int *idx, double tau, double *w_out, long long n,
                cudaStream_t st) {
    k_apply_step<<<grid_of(n), TB, 0, st>>>(w_base, d_sorted, idx, tau, w_out, n);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

void gather_sorted(const double *t_orig, const int *idx, double *t_sorted, long long n, cudaStream_t st) {
    k_gather_sorted<<<grid_of(n), TB, 0, st>>>(t_orig, idx, t_sorted, n);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

// ---- FP32 solves with FP64 iterative refinement ---------------------------
namespace {

// the Laplacian form of RowsLap32, one thread per row
__global__ void k_rows_to_float(Rows R, long long n, float *val32, float *side32) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        const int m = R.cnt[s];
        double rs = 0;
        for (int k = 0; k < m; ++k) rs += *R.valp(s, k);
        const bool side = m > R.cap;
        for (int k = 0; k < m; ++k) {
            const float v = float(*R.colp(s, k) == s ? rs : -*R.valp(s, k));
            if (side)
                side32[R.side[s] + k] = v;
            else
                val32[k * R.stride + s] = v;
        }
    }
}

// partial[block] = sum of v^2 over the block's entries
__global__ void k_sumsq(const double *v, long long n, double *partial) {
    __shared__ double sh[32];
    double a = 0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x)
        a += v[s] * v[s];
    a = block_sum(a, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = a;
}
__global__ void k_sum_partials(const double *partial, int nb, double *out) {
    __shared__ double sh[32];
    double a = 0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) a += partial[i];
    a = block_sum(a, sh);
    if (threadIdx.x == 0) *out = a;
}
// out32 = scale * r (rounded to float)
__global__ void k_to_float(const double *r, double scale, float *out32, long long n) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x)
        out32[s] = float(scale * r[s]);
}
// x += scale * d (d in float or double)
template <class T>
__global__ void k_add_scaled(double *x, const T *d, double scale, long long n) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x)
        x[s] += scale * double(d[s]);
}
// r = b - (H + gauge term) x, in FP64
template <class M>
__global__ void k_residual(M A, long long n, long long g, const double *scal, const double *b, const double *x,
                           double *r) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        double v = A.row_dot(s, x);
        if (s == g) v += scal[S_GDIAG] * x[s];
        r[s] = b[s] - v;
    }
}

double sumsq(const double *v, long long n, double *partial, double *dev_out, cudaStream_t st) {
    const int g = grid_of(n);
    k_sumsq<<<g, TB, 0, st>>>(v, n, partial);
    k_sum_partials<<<1, TB, 0, st>>>(partial, g, dev_out);
    note_launch();
    note_launch();
    double h = 0;
    SDOT_CUDA(cudaMemcpyAsync(&h, dev_out, sizeof(double), cudaMemcpyDeviceToHost, st));
    SDOT_CUDA(cudaStreamSynchronize(st));
    return h;
}

}  // namespace

void rows_to_float(const Rows &rows, long long n, float *val32, float *side_val32, cudaStream_t st) {
    if (n <= 0) return;
    k_rows_to_float<<<PCG_BLOCKS, TB, 0, st>>>(rows, n, val32, side_val32);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

PcgResult pcg_solve_refined(const Rows &rows, const float *val32, const float *side_val32, long long n,
                            long long gauge_row, const double *b, double *x, double rel_tol, int max_iter,
                            const PcgWork &w64, const PcgWorkT<float> &w32, double *res64, cudaStream_t st,
                            double inner_tol, int check, bool multilevel) {
    PcgResult res;
    if (n <= 0) {
        res.converged = true;
        return res;
    }
    const RowsMat A64 = rows_mat(rows);
    const RowsLap32 A32{rows, val32, side_val32};
    const int g = grid_of(n);
    double *r64 = res64;                                        // n doubles: the FP64 residual
    float *b32 = reinterpret_cast<float *>(res64 + n);          // n floats: the scaled residual
    float *d32 = b32 + n;                                       // n floats: the FP32 correction
    double *e64 = res64 + n;                                    // n doubles (FP64 fallback, reuses b32 / d32)
    double *dev_sum = w64.scal + S_NSCAL;                       // a spare device scalar
    // the FP64 gauge term (scal[S_GDIAG]) for the residuals
    k_diag_inv<RowsMat, double><<<g, TB, 0, st>>>(A64, n, gauge_row, w64.dinv, w64.scal);
    note_launch();
    SDOT_CUDA(cudaMemsetAsync(x, 0, size_t(n) * sizeof(double), st));
    SDOT_CUDA(cudaMemcpyAsync(r64, b, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, st));
    const double bb = sumsq(b, n, w64.partial, dev_sum, st);
    if (!(bb > 0)) {
        res.converged = bb == 0;
        return res;
    }
    const double target = rel_tol * rel_tol * bb;
    double rr = bb;
    int it = 0;
    bool fp32_ok = true;
    for (int outer = 0; outer < 60 && it < max_iter; ++outer) {
        if (rr <= target) break;
        const double nr = std::sqrt(rr);
        if (fp32_ok) {
            // the correction for the current residual, solved in FP32
            k_to_float<<<g, TB, 0, st>>>(r64, 1.0 / nr, b32, n);
            note_launch();
            const PcgResult in = pcg_run(A32, n, gauge_row, b32, d32, inner_tol, std::min(max_iter - it, 4000), w32,
                                         st, check, st != nullptr, multilevel, 4);
            it += in.iterations;
            res.levels = in.levels;
            k_add_scaled<float><<<g, TB, 0, st>>>(x, d32, nr, n);
        } else {
            // the rest in FP64: solve H e = r, x += e
            const PcgResult in = pcg_run(A64, n, gauge_row, r64, e64, std::sqrt(target / rr), max_iter - it, w64,
                                         st, check, st != nullptr, multilevel);
            it += in.iterations;
            res.levels = in.levels;
            k_add_scaled<double><<<g, TB, 0, st>>>(x, e64, 1.0, n);
        }
        note_launch();
        k_residual<RowsMat><<<g, TB, 0, st>>>(A64, n, gauge_row, w64.scal, b, x, r64);
        note_launch();
        SDOT_CUDA(cudaGetLastError());
        const double rr_new = sumsq(r64, n, w64.partial, dev_sum, st);
        if (!(rr_new == rr_new)) break;
        // an outer step that does not halve |r|: the FP32 matrix is too far
        // from H for this system
        if (fp32_ok && !(rr_new <= 0.25 * rr)) fp32_ok = false;
        rr = rr_new;
    }
    res.iterations = it;
    res.rel_residual = std::sqrt(rr / bb);
    res.converged = rr <= target;
    return res;
}

}  // namespace sdot
