// Hessian row assembly (see csr.cuh).
#include "csr.cuh"

#include <climits>

namespace sdot {

namespace {

constexpr int TB = 256;

// Rows are sorted by counting: an entry's place is the number of smaller
// columns in its row, so every entry finds it for itself from the row's keys
// (original columns) in shared memory.  L lanes take a row of up to L E entries
// (8 lanes in 2D, where a row has 7 on average, 16 in 3D, where it has 16);
// rows longer than that a whole warp, one after another, up to SM_LONG entries,
// and longer ones one lane by insertion in place.
// Bound by the latency of two dependent gathers at small n and by their
// sectors at large n.  In 3D against insertion in global memory by a thread a
// row (with what follows it): 200,000 Diracs 300 -> 132 us, 20,000 clustered
// ones (rows of up to 200 entries) 190 -> 36, 20,000 uniform ones 103 -> 34.
constexpr int SM_TB = 128;
constexpr int SM_E = 4;
constexpr int SM_LONG = 256;
constexpr int SM_ROW = 16;
// 2D diagrams of more Diracs have a thread per row instead (k_sort_merge_staged):
// 10,000 Diracs 26 us by lanes and 34 us by threads with what follows, 147,000
// 58 and 56, 1M 286 and 212.
constexpr long long SM_LANES_2D = 131072;

// Sorts and merges row s of m <= L E entries with the L lanes of `mask`; key:
// room for m.  Merging never lengthens a row; a side-buffer row whose merged
// count fits the ELL width is moved to its ELL slots, so that Rows::colp (which
// picks the storage from the count) stays consistent.
template <int L, int E>
__device__ __forceinline__ void sort_row(const Rows &R, long long s, int m, const int *idx, long long *cnt_orig, int lane,
                                         unsigned mask, int *key) {
    int c[E], place[E];
    double v[E];
    bool head[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int k = lane + L * q;
        if (k >= m) continue;
        c[q] = *R.colp(s, k);
        v[q] = *R.valp(s, k);
        key[k] = idx[c[q]];
    }
    __syncwarp(mask);
    int gone = 0;
    auto count = [&](bool first) {
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int k = lane + L * q;
            if (k >= m || (!first && !head[q])) continue;
            const int mine = key[k];
            int p = 0;
            bool again = false;
            if (first) head[q] = true;
            for (int e = 0; e < m; ++e) {
                const int ke = key[e];
                p += ke < mine;
                if (first && ke == mine) {
                    if (e < k) head[q] = false;
                    again |= e > k;
                }
            }
            place[q] = p;
            if (first && !head[q]) ++gone;
            if (!first || !again || !head[q]) continue;
            // the sum of the equal columns' values, smallest first
            double sum = 0, last = 0;
            int at = -1;
            bool number = true;
            for (int done = 0;; ++done) {
                double best = 0;
                int b = -1;
                for (int e = 0; e < m; ++e) {
                    if (key[e] != mine) continue;
                    const double x = *R.valp(s, e);
                    number &= x == x;
                    const bool left = !done || x > last || (x == last && e > at);
                    if (left && (b < 0 || x < best)) {
                        best = x;
                        b = e;
                    }
                }
                if (b < 0 || !number) break;
                sum = done ? sum + best : best;
                last = best;
                at = b;
            }
            v[q] = number ? sum : nan("");
        }
    };
    count(true);
    if (__any_sync(mask, gone)) {
        // without the merged ones
#pragma unroll
        for (int q = 0; q < E; ++q)
            if (lane + L * q < m && !head[q]) key[lane + L * q] = INT_MAX;
        __syncwarp(mask);
        count(false);
#pragma unroll
        for (int o = L / 2; o; o >>= 1) gone += __shfl_xor_sync(mask, gone, o);
    }
    __syncwarp(mask);
    const int o = m - gone;
    const bool side = o > R.cap;
#pragma unroll
    for (int q = 0; q < E; ++q) {
        if (lane + L * q >= m || !head[q]) continue;
        const long long to = side ? R.side[s] + place[q] : place[q] * R.stride + s;
        (side ? R.side_col : R.col)[to] = c[q];
        (side ? R.side_val : R.val)[to] = v[q];
    }
    if (lane == 0) {
        R.cnt[s] = o;
        cnt_orig[idx[s]] = o;
    }
}

// The same in place by one lane (a row of any length).
__device__ void sort_row_serial(const Rows &R, long long s, int m, const int *idx, long long *cnt_orig) {
    for (int i = 1; i < m; ++i) {
        const int c = *R.colp(s, i);
        const double v = *R.valp(s, i);
        const int oc = idx[c];
        int j = i - 1;
        while (j >= 0) {
            const int cj = *R.colp(s, j);
            const int ocj = idx[cj];
            const double vj = *R.valp(s, j);
            if (ocj < oc || (ocj == oc && !(vj > v))) break;
            *R.colp(s, j + 1) = cj;
            *R.valp(s, j + 1) = vj;
            --j;
        }
        *R.colp(s, j + 1) = c;
        *R.valp(s, j + 1) = v;
    }
    // merge equal columns
    int o = 0;
    for (int i = 0; i < m; ++i) {
        const int c = *R.colp(s, i);
        const double v = *R.valp(s, i);
        if (i + 1 < m && *R.colp(s, i + 1) == c) {
            *R.valp(s, i + 1) += v;
            continue;
        }
        *R.colp(s, o) = c;
        *R.valp(s, o) = v;
        ++o;
    }
    if (m > R.cap && o <= R.cap) {
        for (int k = 0; k < o; ++k) {
            const int c = *R.colp(s, k);
            const double v = *R.valp(s, k);
            R.col[k * R.stride + s] = c;
            R.val[k * R.stride + s] = v;
        }
    }
    R.cnt[s] = o;
    cnt_orig[idx[s]] = o;
}

#ifdef SDOT_CHECKS
// Row s checked by lane `lane` of `lanes`: its length (0 if it cannot be), columns out of range replaced.
__device__ int check_row(const Rows &R, long long s, long long n, int m, int lane, int lanes) {
    if (m < 0 || m > 4096 || (m > R.cap && (R.side[s] < 0 || R.side[s] + m > R.side_cap))) {
        if (lane == 0) check_fail(20, __LINE__, m);
        return 0;
    }
    for (int i = lane; i < m; i += lanes) {
        const int c = *R.colp(s, i);
        if (c < 0 || c >= n) {
            check_fail(21, __LINE__, c);
            *R.colp(s, i) = int(s);
        }
    }
    return m;
}
#endif

template <int L>
__global__ void __launch_bounds__(SM_TB) k_sort_merge(Rows R, long long n, const int *idx, long long *cnt_orig) {
    __shared__ int keys[SM_TB / 32][SM_LONG];
    const int lane = threadIdx.x & (L - 1), wl = threadIdx.x & 31;
    const unsigned mask = (L == 32 ? ~0u : (1u << L) - 1u) << (wl - lane);
    const long long s = (blockIdx.x * (long long)SM_TB + threadIdx.x) / L;
    int m = s < n ? R.cnt[s] : 0;
#ifdef SDOT_CHECKS
    if (s < n) m = check_row(R, s, n, m, lane, L);
    __syncwarp(mask);
#endif
    int *key = keys[threadIdx.x / 32];
    const bool fits = m <= L * SM_E;
    if (s < n && fits) sort_row<L, SM_E>(R, s, m, idx, cnt_orig, lane, mask, key + (wl - lane) * SM_E);
    __syncwarp();
    unsigned longer = __ballot_sync(0xffffffffu, lane == 0 && s < n && !fits);
    for (; longer; longer &= longer - 1) {
        const int from = __ffs(int(longer)) - 1;
        const long long sl = __shfl_sync(0xffffffffu, s, from);
        const int ml = __shfl_sync(0xffffffffu, m, from);
        if (ml <= SM_LONG)
            sort_row<32, SM_LONG / 32>(R, sl, ml, idx, cnt_orig, wl, 0xffffffffu, key);
        else if (wl == 0)
            sort_row_serial(R, sl, ml, idx, cnt_orig);
        __syncwarp();
    }
}

// The rows of a large 2D diagram, a thread each: rows of at most SM_ROW entries
// (every row of the fast tier) by insertion in shared memory, longer ones in
// place.  Neighbouring threads read and write neighbouring entries, which the
// lanes of a row do not.
__global__ void __launch_bounds__(SM_TB) k_sort_merge_staged(Rows R, long long n, const int *idx, long long *cnt_orig) {
    __shared__ int s_key[SM_ROW * SM_TB], s_col[SM_ROW * SM_TB];
    __shared__ double s_val[SM_ROW * SM_TB];
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    int m = R.cnt[s];
#ifdef SDOT_CHECKS
    m = check_row(R, s, n, m, 0, 1);
#endif
    if (m > SM_ROW) {
        sort_row_serial(R, s, m, idx, cnt_orig);
        return;
    }
    int o = 0;
    // entry i of this thread at [i * SM_TB + t]: no bank conflicts
    const int t = threadIdx.x;
    for (int i = 0; i < m; ++i) {
        const int c = *R.colp(s, i);
        s_col[i * SM_TB + t] = c;
        s_val[i * SM_TB + t] = *R.valp(s, i);
        s_key[i * SM_TB + t] = idx[c];
    }
    // insertion sort by (original column, value)
    for (int i = 1; i < m; ++i) {
        const int oc = s_key[i * SM_TB + t], c = s_col[i * SM_TB + t];
        const double v = s_val[i * SM_TB + t];
        int j = i - 1;
        while (j >= 0) {
            const int ocj = s_key[j * SM_TB + t];
            const double vj = s_val[j * SM_TB + t];
            if (ocj < oc || (ocj == oc && !(vj > v))) break;
            s_key[(j + 1) * SM_TB + t] = ocj;
            s_col[(j + 1) * SM_TB + t] = s_col[j * SM_TB + t];
            s_val[(j + 1) * SM_TB + t] = vj;
            --j;
        }
        s_key[(j + 1) * SM_TB + t] = oc;
        s_col[(j + 1) * SM_TB + t] = c;
        s_val[(j + 1) * SM_TB + t] = v;
    }
    // merge equal columns (each into the next) and write back
    for (int i = 0; i < m; ++i) {
        const int c = s_col[i * SM_TB + t];
        const double v = s_val[i * SM_TB + t];
        if (i + 1 < m && s_col[(i + 1) * SM_TB + t] == c) {
            s_val[(i + 1) * SM_TB + t] += v;
            continue;
        }
        *R.colp(s, o) = c;
        *R.valp(s, o) = v;
        ++o;
    }
    R.cnt[s] = o;
    cnt_orig[idx[s]] = o;
}

// WL lanes per row: the entries of a row are read and written side by side (one
// thread per row was a chain of dependent reads and scattered writes: 18 us at
// 1,000 rows, 146 us at 1M).
constexpr int WL = 8;
__global__ void k_write(Rows R, long long n, const int *idx, const long long *offsets, long long *cols, double *vals) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, s = t / WL;
    if (s >= n) return;
    const int m = R.cnt[s];
    const long long o = offsets[idx[s]];
    for (int i = int(t % WL); i < m; i += WL) {
        cols[o + i] = idx[*R.colp(s, i)];
        vals[o + i] = *R.valp(s, i);
    }
}

__global__ void k_nb_counts(Rows NB, long long n, const int *idx, long long *cnt_orig) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    cnt_orig[idx[s]] = NB.cnt[s];
}

__global__ void k_nb_write(Rows NB, long long n, const int *idx, const long long *offsets, long long *ids) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int m = NB.cnt[s];
    const long long o = offsets[idx[s]];
    for (int i = 0; i < m; ++i) {
        const int id = *NB.colp(s, i);
        // periodic images: id j + (k + 1) n keeps its translation k
        ids[o + i] = id >= 0 ? (long long)idx[id % n] + (long long)(id / n) * n : (id == ID_ARC ? -2 : -1);
    }
}

// Masses and centroids to caller order, the number of empty cells added to
// *n_void, the last CSR offset to *nnz, and the tree's status to *err.
__global__ void k_unpermute(const double *m, double *om, const double *mc, double *omc, const double *c, double *oc,
                            long long n, int d, const int *idx, const long long *offsets, long long *nnz,
                            unsigned long long *n_void, const unsigned *tree_sync, unsigned *err) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const bool in = s < n;
    const double ms = in ? m[s] : 1.0;
    if (in) {
        const long long i = idx[s];
        om[i] = ms;
        omc[i] = mc[s];
        for (int k = 0; k < d; ++k) oc[i * d + k] = c[s * d + k];
    }
    const int z = __syncthreads_count(ms == 0.0);  // one atomic per block
    if (threadIdx.x == 0 && z) atomicAdd(n_void, (unsigned long long)z);
    if (s == 0) {
        *nnz = offsets[n];
        if (tree_sync[1] | tree_sync[3]) atomicOr(err, unsigned(DE_TREE));
    }
}

// ---- domains of several shapes: one cell pass per shape, summed here
__global__ void k_rows_clear(Rows R, long long n) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s < n) R.cnt[s] = 0;
}

// dst row s += src row s (entries appended; a row that outgrows the ELL
// width moves, with the new entries, to a fresh place in the side buffer)
__global__ void k_rows_append(Rows dst, Rows src, long long n, unsigned *err) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int m0 = dst.cnt[s], m1 = src.cnt[s], m = m0 + m1;
    if (m1 == 0) return;
    if (m <= dst.cap) {
        for (int k = 0; k < m1; ++k) {
            dst.col[(m0 + k) * dst.stride + s] = *src.colp(s, k);
            if (dst.val) dst.val[(m0 + k) * dst.stride + s] = *src.valp(s, k);
        }
        dst.cnt[s] = m;
        return;
    }
    const unsigned long long off = atomicAdd(dst.side_used, (unsigned long long)m);
    if ((long long)(off + m) > dst.side_cap) {
        atomicOr(err, unsigned(DE_SIDE));
        return;
    }
    for (int k = 0; k < m0; ++k) {
        dst.side_col[off + k] = *dst.colp(s, k);
        if (dst.side_val) dst.side_val[off + k] = *dst.valp(s, k);
    }
    for (int k = 0; k < m1; ++k) {
        dst.side_col[off + m0 + k] = *src.colp(s, k);
        if (dst.side_val) dst.side_val[off + m0 + k] = *src.valp(s, k);
    }
    dst.side[s] = (long long)off;
    dst.cnt[s] = m;
}

// mass += t_mass, mass_c += t_mass_c, mom += t_ctd * t_mass_c (dim 2 or 3)
__global__ void k_accum(double *mass, double *mass_c, double *mom, const double *t_mass, const double *t_mass_c,
                        const double *t_ctd, long long n, int dim) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    mass[s] += t_mass[s];
    mass_c[s] += t_mass_c[s];
    for (int d = 0; d < dim; ++d) mom[dim * s + d] += t_ctd[dim * s + d] * t_mass_c[s];
}

// centroid = moment / (mass + (mass == 0)), as get_centroids divides
__global__ void k_ctd_final(double *ctd, const double *mom, const double *mass_c, long long n, int dim) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double d = mass_c[s] + (mass_c[s] == 0);
    for (int k = 0; k < dim; ++k) ctd[dim * s + k] = mom[dim * s + k] / d;
}

}  // namespace

void csr_read_checks(unsigned long long out[3]) {
#ifdef SDOT_CHECKS
    SDOT_CUDA(cudaMemcpyFromSymbol(out, sdot_dbg_word, 3 * sizeof(unsigned long long)));
#else
    out[0] = out[1] = out[2] = 0;
#endif
}

void csr_sort_merge(const Rows &R, long long n, const int *idx, long long *cnt_orig, bool short_rows, cudaStream_t st) {
    if (n <= 0) return;
    if (short_rows && n > SM_LANES_2D)
        k_sort_merge_staged<<<ceil_div(n, SM_TB), SM_TB, 0, st>>>(R, n, idx, cnt_orig);
    else if (short_rows)
        k_sort_merge<8><<<ceil_div(n * 8, SM_TB), SM_TB, 0, st>>>(R, n, idx, cnt_orig);
    else
        k_sort_merge<16><<<ceil_div(n * 16, SM_TB), SM_TB, 0, st>>>(R, n, idx, cnt_orig);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

void csr_write(const Rows &R, long long n, const int *idx, const long long *offsets, long long *cols, double *vals,
               cudaStream_t st) {
    if (n <= 0) return;
    k_write<<<ceil_div(n * WL, TB), TB, 0, st>>>(R, n, idx, offsets, cols, vals);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}
void nb_counts(const Rows &NB, long long n, const int *idx, long long *cnt_orig, cudaStream_t st) {
    if (n <= 0) return;
    k_nb_counts<<<ceil_div(n, TB), TB, 0, st>>>(NB, n, idx, cnt_orig);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}
void nb_write(const Rows &NB, long long n, const int *idx, const long long *offsets, long long *ids, cudaStream_t st) {
    if (n <= 0) return;
    k_nb_write<<<ceil_div(n, TB), TB, 0, st>>>(NB, n, idx, offsets, ids);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}
void unpermute(const double *m, double *om, const double *mc, double *omc, const double *c, double *oc, long long n, int d,
               const int *idx, const long long *offsets, long long *nnz, unsigned long long *n_void,
               const unsigned *tree_sync, unsigned *err, cudaStream_t st) {
    if (n <= 0) return;
    k_unpermute<<<ceil_div(n, TB), TB, 0, st>>>(m, om, mc, omc, c, oc, n, d, idx, offsets, nnz, n_void, tree_sync, err);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

void rows_clear(const Rows &R, long long n, cudaStream_t st) {
    if (n <= 0) return;
    k_rows_clear<<<ceil_div(n, TB), TB, 0, st>>>(R, n);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}
void rows_append(const Rows &dst, const Rows &src, long long n, unsigned *err, cudaStream_t st) {
    if (n <= 0) return;
    k_rows_append<<<ceil_div(n, TB), TB, 0, st>>>(dst, src, n, err);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}
void accum_pass(double *mass, double *mass_c, double *mom, const double *t_mass, const double *t_mass_c,
                const double *t_ctd, long long n, int dim, cudaStream_t st) {
    if (n <= 0) return;
    k_accum<<<ceil_div(n, TB), TB, 0, st>>>(mass, mass_c, mom, t_mass, t_mass_c, t_ctd, n, dim);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}
void centroids_final(double *ctd, const double *mom, const double *mass_c, long long n, int dim, cudaStream_t st) {
    if (n <= 0) return;
    k_ctd_final<<<ceil_div(n, TB), TB, 0, st>>>(ctd, mom, mass_c, n, dim);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

}  // namespace sdot
