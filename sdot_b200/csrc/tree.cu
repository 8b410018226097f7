// Device Z-order tree (see tree.cuh).
#include "prims.cuh"
#include "tree.cuh"

namespace sdot {

namespace {

constexpr int TB = 256;

__device__ __forceinline__ unsigned long long ord_bits(double v) {
    unsigned long long b = __double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double from_ord_bits(unsigned long long b) {
    return __longlong_as_double((b >> 63) ? (b & 0x7fffffffffffffffull) : ~b);
}

template <int D>
__global__ void k_bbox(const double *pos, long long n, unsigned long long *bits) {
    __shared__ unsigned long long smin[D], smax[D];
    if (threadIdx.x < D) {
        smin[threadIdx.x] = ~0ull;
        smax[threadIdx.x] = 0ull;
    }
    __syncthreads();
    unsigned long long lmin[D], lmax[D];
    for (int d = 0; d < D; ++d) { lmin[d] = ~0ull; lmax[d] = 0ull; }
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        for (int d = 0; d < D; ++d) {
            unsigned long long o = ord_bits(pos[D * i + d]);
            lmin[d] = o < lmin[d] ? o : lmin[d];
            lmax[d] = o > lmax[d] ? o : lmax[d];
        }
    }
    for (int d = 0; d < D; ++d) {
        atomicMin(&smin[d], lmin[d]);
        atomicMax(&smax[d], lmax[d]);
    }
    __syncthreads();
    if (threadIdx.x < D) {
        atomicMin(&bits[threadIdx.x], smin[threadIdx.x]);
        atomicMax(&bits[D + threadIdx.x], smax[threadIdx.x]);
    }
}

__device__ __forceinline__ unsigned spread2(unsigned v) {  // 16 bits -> even bits
    v &= 0xffffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}
__device__ __forceinline__ unsigned spread3(unsigned v) {  // 10 bits -> every third bit
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

template <int D>
__global__ void k_morton(const double *pos, long long n, const unsigned long long *bbox, int bits, unsigned *keys,
                         unsigned *vals) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double top = double((1u << bits) - 1u);
    unsigned q[D];
    for (int d = 0; d < D; ++d) {
        const double lo = from_ord_bits(bbox[d]), hi = from_ord_bits(bbox[D + d]);
        double ext = hi - lo;
        double t = ext > 0 ? (pos[D * i + d] - lo) / ext * double(1u << bits) : 0.0;
        t = fmin(fmax(t, 0.0), top);
        q[d] = unsigned(t);
    }
    unsigned k;
    if (D == 2)
        k = spread2(q[0]) | (spread2(q[1]) << 1);
    else
        k = spread3(q[0]) | (spread3(q[1]) << 1) | (spread3(q[2 % D]) << 2);
    keys[i] = k;
    vals[i] = unsigned(i);
}

// (A sort that was given up has left no order: any permutation keeps the indexes
// in range, and the level kernel marks the tree.)
template <int D>
__global__ void k_gather(const double *pos, const double *w, const unsigned *order, const unsigned *lost, long long n,
                         double *pos_s, double *w_s, int *idx, int *inv) {
    long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const unsigned i = *lost ? unsigned(s) : order[s];
    for (int d = 0; d < D; ++d) pos_s[D * s + d] = pos[D * (long long)i + d];
    w_s[s] = w[i];
    idx[s] = int(i);
    inv[i] = int(s);
}

// First indices of [a, b) whose keys are >= v + (c << shift), c = 1 .. C - 1,
// into st[c] (st[0] = a, st[C] = b), found by the 32 lanes of a warp together
// (every lane gets them): each round probes 32 evenly spaced keys of every
// stretch and keeps the part between the last one below and the next, so a range
// of r keys takes about log32(r) dependent reads, those of the C - 1 searches at
// once.
template <int C>
__device__ __forceinline__ void warp_bounds(const unsigned *keys, int a, int b, unsigned long long v, int shift, int *st) {
    const int lane = threadIdx.x & 31;
    int lo[C], hi[C];
#pragma unroll
    for (int c = 1; c < C; ++c) {
        lo[c] = a;
        hi[c] = b;
    }
    for (bool last = false; !last;) {
        last = true;
        unsigned k[C];
        int step[C];
#pragma unroll
        for (int c = 1; c < C; ++c) {
            step[c] = hi[c] - lo[c] > 32 ? (hi[c] - lo[c] + 31) / 32 : 1;
            last &= step[c] == 1;
            const int i = lo[c] + lane * step[c];
            k[c] = i < hi[c] ? keys[i] : 0u;
        }
#pragma unroll
        for (int c = 1; c < C; ++c) {
            const int i = lo[c] + lane * step[c];
            const bool below = i < hi[c] && (unsigned long long)k[c] < v + ((unsigned long long)c << shift);
            const int cnt = __popc(__ballot_sync(0xffffffffu, below));  // probes 0 .. cnt - 1 are below
            if (step[c] == 1) {
                lo[c] += cnt;
                hi[c] = lo[c];
            } else if (cnt == 0) {
                hi[c] = lo[c];
            } else {
                const int nhi = lo[c] + cnt * step[c];
                lo[c] += (cnt - 1) * step[c] + 1;
                if (nhi < hi[c]) hi[c] = nhi;
            }
        }
    }
    st[0] = a;
    st[C] = b;
#pragma unroll
    for (int c = 1; c < C; ++c) st[c] = lo[c];
}

// A tree that cannot be used: every walk that starts with a vertex opens the
// root, and its guard ends it there.
template <int D>
__device__ void lose_tree(TreeNode<D> *nodes) {
    nodes[0].a = -1;
    nodes[0].b = 1;
    for (int d = 0; d < D; ++d) nodes[0].lo[d] = nodes[0].hi[d] = 0;
    nodes[0].maxw = 1.0 / 0.0;
}

// err |= DE_TREE where a wait of the tree's kernels was given up.
__global__ void k_tree_status(const unsigned *sync, unsigned *err) {
    if (sync[1] | sync[3]) atomicOr(err, unsigned(DE_TREE));
}

template <int D>
struct TreeArgs {
    TreeNode<D> *nodes;
    int *level, *counters;   // counters: see DeviceTree
    const unsigned *keys;
    const double *pos;
    double *w;
    const double *w_orig;    // refresh: the new weights, caller order
    const int *idx;
    long long n;
    int bits, max_per_leaf, max_nodes, npass;
    unsigned *sync;
};

// Levels of the tree, in one cooperative kernel of blocks of 1024.  BUILD: the
// top-down split, level by level, one warp per node: its key range is cut at the
// 2^D child prefixes of its next Morton level (single-child levels skipped), the
// children are appended to the next level; then boxes and maximum weights
// bottom-up, the leaves of all levels at once.  Otherwise (new weights): the
// weights gathered, and the maximum weights bottom-up.
// As launches, a level was one kernel to split, one to note the count and one to
// reduce, for the 17 levels a key has and not the 6 to 11 of a tree: 51 launches,
// 170 us of the 230 of a build of 10,000 Diracs and 345 of 450 us at 1M; the
// refresh 17 launches, 54 us.
constexpr int TREE_TB = 1024;
template <int D, bool BUILD>
__global__ void __launch_bounds__(TREE_TB, 1) k_tree(const TreeArgs<D> A) {
    constexpr int C = 1 << D;
    const int lane = threadIdx.x & 31;
    const int warp = int((blockIdx.x * TREE_TB + threadIdx.x) >> 5), nwarps = int(gridDim.x * TREE_TB >> 5);
    const int thread = blockIdx.x * TREE_TB + threadIdx.x, nthreads = gridDim.x * TREE_TB;
    int *const start = A.counters + 1, *const added = A.counters + A.npass + 4;
    unsigned target = 0;
    int depth = 0;  // levels in use
    if (BUILD && A.sync[3]) {  // the sort's wait was given up: its keys are in no order
        if (thread == 0) lose_tree(A.nodes);
        return;
    }
    if (BUILD) {
        // nodes [beg, end) are the level's; added[p]: how many it gives the next
        int beg = 0, end = 1;
        for (int p = 0; p < A.npass && beg < end; ++p) {
            for (int node = beg + warp; node < end; node += nwarps) {
                const int a = A.nodes[node].a, b = A.nodes[node].b;
                int L = A.level[node];
                while (b - a > A.max_per_leaf && L < A.bits) {
                    const int shift = D * (A.bits - L - 1);
                    const unsigned long long prefix = (unsigned long long)A.keys[a] >> (shift + D);
                    int st[C + 1];
                    warp_bounds<C>(A.keys, a, b, (prefix << D) << shift, shift, st);
                    int ne = 0;
#pragma unroll
                    for (int c = 0; c < C; ++c) ne += st[c + 1] > st[c];
                    ++L;
                    if (ne == 1) continue;
                    int first = 0;
                    if (lane == 0) first = end + atomicAdd(&added[p], ne);
                    first = __shfl_sync(0xffffffffu, first, 0);
                    if (first + ne > A.max_nodes) break;  // cannot happen: nodes <= 2n
                    if (lane == 0) {
                        int k = first;
#pragma unroll
                        for (int c = 0; c < C; ++c)
                            if (st[c + 1] > st[c]) {
                                A.nodes[k].a = st[c];
                                A.nodes[k].b = st[c + 1];
                                A.level[k] = L;
                                ++k;
                            }
                        A.nodes[node].a = first;
                        A.nodes[node].b = -ne;
                    }
                    break;
                }
            }
            if (!grid_barrier(A.sync, target)) {
                lose_tree(A.nodes);
                return;
            }
            depth = p + 1;
            beg = end;
            end += added[p];
            if (thread == 0) start[p + 1] = beg;
        }
        if (thread == 0)
            for (int p = depth; p <= A.npass; ++p) start[p] = p == 0 ? 0 : beg;
    } else {
        while (depth < A.npass && start[depth] < start[depth + 1]) ++depth;
        for (long long s = thread; s < A.n; s += nthreads) A.w[s] = A.w_orig[A.idx[s]];
        if (!grid_barrier(A.sync, target)) {
            lose_tree(A.nodes);
            return;
        }
    }
    // ---- bottom-up.  The ranges of the levels, from the level counts or starts
    auto range = [&](int p, int &beg, int &end) {
        if (BUILD) {
            beg = 0;
            end = 1;
            for (int q = 0; q < p; ++q) {
                beg = end;
                end += added[q];
            }
        } else {
            beg = start[p];
            end = start[p + 1];
        }
    };
    int beg, total;
    range(depth - 1, beg, total);
    for (int node = thread; node < total; node += nthreads) {
        const int a = A.nodes[node].a, b = A.nodes[node].b;
        if (b <= 0) continue;
        double lo[D], hi[D], mw = -1.0 / 0.0;
        for (int d = 0; d < D; ++d) {
            lo[d] = 1.0 / 0.0;
            hi[d] = -1.0 / 0.0;
        }
        for (int s = a; s < b; ++s) {
            mw = fmax(mw, A.w[s]);
            if (BUILD)
                for (int d = 0; d < D; ++d) {
                    const double v = A.pos[D * (long long)s + d];
                    lo[d] = fmin(lo[d], v);
                    hi[d] = fmax(hi[d], v);
                }
        }
        A.nodes[node].maxw = mw;
        if (BUILD)
            for (int d = 0; d < D; ++d) {
                A.nodes[node].lo[d] = lo[d];
                A.nodes[node].hi[d] = hi[d];
            }
    }
    for (int p = depth - 2; p >= 0; --p) {  // the last level holds leaves only
        if (!grid_barrier(A.sync, target)) {
            lose_tree(A.nodes);
            return;
        }
        int end;
        range(p, beg, end);
        for (int node = beg + thread; node < end; node += nthreads) {
            const int a = A.nodes[node].a, nch = -A.nodes[node].b;
            if (nch <= 0) continue;
            double lo[D], hi[D], mw = -1.0 / 0.0;
            for (int d = 0; d < D; ++d) {
                lo[d] = 1.0 / 0.0;
                hi[d] = -1.0 / 0.0;
            }
            for (int c = a; c < a + nch; ++c) {
                const TreeNode<D> &ch = A.nodes[c];
                mw = fmax(mw, ch.maxw);
                if (BUILD)
                    for (int d = 0; d < D; ++d) {
                        lo[d] = fmin(lo[d], ch.lo[d]);
                        hi[d] = fmax(hi[d], ch.hi[d]);
                    }
            }
            A.nodes[node].maxw = mw;
            if (BUILD)
                for (int d = 0; d < D; ++d) {
                    A.nodes[node].lo[d] = lo[d];
                    A.nodes[node].hi[d] = hi[d];
                }
        }
    }
    if (BUILD && thread == 0) A.counters[0] = total;
}

// Start of a build: the box of nothing, the root over every Dirac, no children
// counted, no arrival at the barrier.
template <int D>
__global__ void k_tree_init(unsigned long long *bits, TreeNode<D> *nodes, int *level, int *counters, int npass, long long n,
                            unsigned *sync) {
    const int t = threadIdx.x;
    if (t < D) {
        bits[t] = ~0ull;
        bits[D + t] = 0ull;
    }
    if (t < npass) counters[npass + 4 + t] = 0;
    if (t < 4) sync[t] = 0;
    if (t == 0) {
        nodes[0].a = 0;
        nodes[0].b = int(n);
        level[0] = 0;
        counters[1] = 0;
    }
}

template <class T>
void dev_alloc(T *&p, size_t count) {
    SDOT_CUDA(cudaMalloc(reinterpret_cast<void **>(&p), count * sizeof(T) + 16));
}
template <class T>
void dev_free(T *&p) {
    if (p) cudaFree(p);
    p = nullptr;
}

template <int D, bool BUILD>
void tree_launch(const TreeArgs<D> &a, cudaStream_t st) {
    // one block per SM at most: all resident
    int sms = 0, dev = 0;
    SDOT_CUDA(cudaGetDevice(&dev));
    SDOT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int g = int(std::min<long long>(sms, (a.n + 511) / 512));
    TreeArgs<D> b = a;
    void *args[] = {&b};
    SDOT_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(k_tree<D, BUILD>), dim3(g), dim3(TREE_TB), args, 0, st));
    note_launch();
}

int grid_for(long long n, int tb) {
    long long g = (n + tb - 1) / tb;
    if (g < 1) g = 1;
    if (g > 148 * 16) g = 148 * 16;
    return int(g);
}

// Captures the launches `f` makes on `st` into an executable graph; false
// (nothing launched, nothing captured) where the stream cannot be captured:
// the legacy default stream, or a stream already being captured.
template <class F>
bool capture(cudaStream_t st, cudaGraphExec_t &exec, unsigned long long &launches, F &&f) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return false;
    }
    if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaGraph_t g = nullptr;
    unsigned long long counted = 0;
    {
        CaptureCount cc;
        try {
            f();
        } catch (...) {
            cudaStreamEndCapture(st, &g);
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            throw;
        }
        counted = cc.n;
    }
    cudaError_t e = cudaStreamEndCapture(st, &g);
    if (e == cudaSuccess && g) e = cudaGraphInstantiate(&exec, g, 0);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        cudaGetLastError();
        exec = nullptr;
        return false;
    }
    launches = counted;
    return true;
}

}  // namespace

template <int D>
void DeviceTree<D>::reserve(long long nn) {
    if (nn <= cap_n && pos) return;
    release();
    cap_n = nn < 1 ? 1 : nn;
    key_bits = D == 2 ? 16 : 10;
    npass = key_bits + 1;
    max_nodes = int(2 * cap_n + 2);
    dev_alloc(pos, size_t(D) * cap_n);
    dev_alloc(w, cap_n);
    dev_alloc(idx, cap_n);
    dev_alloc(inv, cap_n);
    dev_alloc(nodes, max_nodes);
    dev_alloc(node_level, max_nodes);
    dev_alloc(counters, 2 * npass + 8);
    dev_alloc(sync, 4);
    dev_alloc(keys, cap_n);
    dev_alloc(keys2, cap_n);
    dev_alloc(keys3, cap_n);
    dev_alloc(vals, cap_n);
    dev_alloc(vals2, cap_n);
    dev_alloc(vals3, cap_n);
    tmp_bytes = radix_tmp_size();
    SDOT_CUDA(cudaMalloc(&tmp, tmp_bytes));
    dev_alloc(bbox_bits, 2 * D);
}

template <int D>
void DeviceTree<D>::drop_graphs() {
    if (build_graph) cudaGraphExecDestroy(build_graph);
    if (weights_graph) cudaGraphExecDestroy(weights_graph);
    build_graph = weights_graph = nullptr;
    bg_n = wg_n = -1;
}

template <int D>
void DeviceTree<D>::release() {
    drop_graphs();
    dev_free(pos); dev_free(w); dev_free(idx); dev_free(inv);
    dev_free(nodes); dev_free(node_level); dev_free(counters); dev_free(sync);
    dev_free(keys); dev_free(keys2); dev_free(keys3);
    dev_free(vals); dev_free(vals2); dev_free(vals3);
    if (tmp) cudaFree(tmp);
    tmp = nullptr;
    dev_free(bbox_bits);
    cap_n = 0;
}

template <int D>
void DeviceTree<D>::build(const double *pos_orig, const double *w_orig, long long nn, cudaStream_t st) {
    reserve(nn);
    n = nn;
    if (n == 0) return;
    if (!(build_graph && bg_n == n && bg_pos == pos_orig && bg_w == w_orig && bg_leaf == max_per_leaf)) {
        if (build_graph) cudaGraphExecDestroy(build_graph);
        build_graph = nullptr;
        bg_n = -1;
        if (!capture(st, build_graph, bg_launches, [&] { build_launches(pos_orig, w_orig, st); })) {
            build_launches(pos_orig, w_orig, st);
            return;
        }
        bg_n = n;
        bg_pos = pos_orig;
        bg_w = w_orig;
        bg_leaf = max_per_leaf;
    }
    SDOT_CUDA(cudaGraphLaunch(build_graph, st));
    note_launches(bg_launches);
}

template <int D>
void DeviceTree<D>::build_launches(const double *pos_orig, const double *w_orig, cudaStream_t st) {
    k_tree_init<D><<<1, 32, 0, st>>>(bbox_bits, nodes, node_level, counters, npass, n, sync);
    note_launch();
    k_bbox<D><<<grid_for(n, TB), TB, 0, st>>>(pos_orig, n, bbox_bits);
    note_launch();
    k_morton<D><<<ceil_div(n, TB), TB, 0, st>>>(pos_orig, n, bbox_bits, key_bits, keys, vals);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
    radix_sort_pairs(keys, vals, keys2, vals2, keys3, vals3, n, D * key_bits, tmp, sync + 2, st);
    k_gather<D><<<ceil_div(n, TB), TB, 0, st>>>(pos_orig, w_orig, vals2, sync + 3, n, pos, w, idx, inv);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
    tree_launch<D, true>(TreeArgs<D>{nodes, node_level, counters, keys2, pos, w, nullptr, idx, n, key_bits, max_per_leaf,
                                     max_nodes, npass, sync},
                         st);
}

template <int D>
void DeviceTree<D>::update_weights(const double *w_orig, cudaStream_t st) {
    if (n == 0) return;
    if (!(weights_graph && wg_n == n && wg_w == w_orig)) {
        if (weights_graph) cudaGraphExecDestroy(weights_graph);
        weights_graph = nullptr;
        wg_n = -1;
        if (!capture(st, weights_graph, wg_launches, [&] { weights_launches(w_orig, st); })) {
            weights_launches(w_orig, st);
            return;
        }
        wg_n = n;
        wg_w = w_orig;
    }
    SDOT_CUDA(cudaGraphLaunch(weights_graph, st));
    note_launches(wg_launches);
}

template <int D>
void DeviceTree<D>::weights_launches(const double *w_orig, cudaStream_t st) {
    SDOT_CUDA(cudaMemsetAsync(sync, 0, 2 * sizeof(unsigned), st));
    tree_launch<D, false>(TreeArgs<D>{nodes, node_level, counters, keys2, pos, w, w_orig, idx, n, key_bits, max_per_leaf,
                                      max_nodes, npass, sync},
                          st);
}

template <int D>
void DeviceTree<D>::status(unsigned *err, cudaStream_t st) const {
    if (n == 0) return;
    k_tree_status<<<1, 1, 0, st>>>(sync, err);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

template struct DeviceTree<2>;
template struct DeviceTree<3>;

}  // namespace sdot
