// Exclusive scan and stable LSD radix sort (see prims.cuh).
#include "prims.cuh"

namespace sdot {

namespace {

constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <class T>
__device__ T block_exclusive_scan(T v, T *warp_tot, T *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        T t = lane < nw ? warp_tot[lane] : T(0);
        T ti = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T u = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += u;
        }
        if (lane < nw) warp_tot[lane] = ti - t;
        if (lane == nw - 1) *total = ti;
    }
    __syncthreads();
    T r = warp_tot[warp] + incl - v;
    __syncthreads();
    return r;
}

template <class T>
__global__ void k_block_sums(const T *in, T *sums, long long n) {
    __shared__ T wt[32];
    __shared__ T tot;
    long long base = (long long)blockIdx.x * SCAN_TILE;
    T s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        long long i = base + (long long)k * SCAN_THREADS + threadIdx.x;
        if (i < n) s += in[i];
    }
    block_exclusive_scan<T>(s, wt, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

template <class T>
__global__ void k_block_scan(const T *in, T *out, long long n, const T *offsets, T *grand_total) {
    __shared__ T tile[SCAN_TILE];
    __shared__ T wt[32];
    __shared__ T tot;
    long long base = (long long)blockIdx.x * SCAN_TILE;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        long long i = base + (long long)k * SCAN_THREADS + threadIdx.x;
        tile[k * SCAN_THREADS + threadIdx.x] = i < n ? in[i] : T(0);
    }
    __syncthreads();
    T loc[SCAN_ITEMS];
    T s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        loc[k] = tile[threadIdx.x * SCAN_ITEMS + k];
        s += loc[k];
    }
    T ex = block_exclusive_scan<T>(s, wt, &tot);
    T off = offsets ? offsets[blockIdx.x] : T(0);
    T run = off + ex;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        tile[threadIdx.x * SCAN_ITEMS + k] = run;
        run += loc[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        long long i = base + (long long)k * SCAN_THREADS + threadIdx.x;
        if (i < n) out[i] = tile[k * SCAN_THREADS + threadIdx.x];
    }
    if (grand_total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *grand_total = off + tot;
}

template <class T>
void scan_rec(const T *in, T *out, long long n, char *tmp, T *grand_total, cudaStream_t st) {
    if (n <= 0) {
        if (grand_total) SDOT_CUDA(cudaMemsetAsync(grand_total, 0, sizeof(T), st));
        return;
    }
    long long nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (nb == 1) {
        k_block_scan<T><<<1, SCAN_THREADS, 0, st>>>(in, out, n, nullptr, grand_total);
        note_launch();
        SDOT_CUDA(cudaGetLastError());
        return;
    }
    T *sums = reinterpret_cast<T *>(tmp);
    T *sums_scanned = sums + nb;
    char *next = reinterpret_cast<char *>(sums_scanned + nb);
    next = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(next) + 255) & ~uintptr_t(255));
    k_block_sums<T><<<unsigned(nb), SCAN_THREADS, 0, st>>>(in, sums, n);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
    scan_rec<T>(sums, sums_scanned, nb, next, nullptr, st);
    k_block_scan<T><<<unsigned(nb), SCAN_THREADS, 0, st>>>(in, out, n, sums_scanned, grand_total);
    note_launch();
    SDOT_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------- radix ----
// The whole LSD sort in one cooperative kernel: every block keeps one stretch of
// the pairs, and a pass (8 bits) is a histogram of the stretch, a barrier of the
// grid, the block's starts per digit from the histograms of all blocks, the
// scatter, and a barrier.  As launches a pass was a histogram, a three-kernel
// scan and a scatter whose tiles of 4,096 pairs were a chain of 16 rounds: 50 us a
// pass from 1,000 pairs to 1M.
constexpr int RADIX_TB = 512;
constexpr int RADIX_MAX_BLOCKS = 256;

struct RadixArgs {
    const unsigned *kin, *vin;
    unsigned *kout, *vout, *kalt, *valt;
    unsigned *hist;  // 256 per block
    unsigned *sync;
    long long n;
    int passes;
};

__global__ void __launch_bounds__(RADIX_TB, 1) k_radix_sort(const RadixArgs A) {
    constexpr int NW = RADIX_TB / 32;
    __shared__ unsigned run[256], part[8], wcnt[NW][256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = int(gridDim.x);
    const unsigned lt_mask = (1u << lane) - 1u;
    const long long rounds = (A.n + (long long)nb * RADIX_TB - 1) / ((long long)nb * RADIX_TB);
    const long long beg = rounds * RADIX_TB * blockIdx.x;
    const long long end = beg + rounds * RADIX_TB < A.n ? beg + rounds * RADIX_TB : A.n;
    unsigned target = 0;
    const unsigned *sk = A.kin, *sv = A.vin;
    for (int p = 0; p < A.passes; ++p) {
        const int shift = 8 * p;
        // ping-pong so that the last pass lands in (kout, vout)
        const bool to_out = ((A.passes - 1 - p) & 1) == 0;
        unsigned *dk = to_out ? A.kout : A.kalt, *dv = to_out ? A.vout : A.valt;
        if (tid < 256) run[tid] = 0;
        __syncthreads();
        for (long long i = beg + tid; i < end; i += RADIX_TB) atomicAdd(&run[(sk[i] >> shift) & 255u], 1u);
        __syncthreads();
        if (tid < 256) A.hist[blockIdx.x * 256 + tid] = run[tid];
        if (!grid_barrier(A.sync, target)) return;
        // digit tid: its total, what the blocks before this one hold of it, and
        // the exclusive sum of the totals over the digits
        unsigned before = 0, total = 0, incl = 0;
        if (tid < 256) {
#pragma unroll 8
            for (int b = 0; b < nb; ++b) {
                const unsigned v = A.hist[b * 256 + tid];
                total += v;
                if (b < int(blockIdx.x)) before += v;
            }
            incl = total;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            if (lane == 31) part[warp] = incl;
        }
        __syncthreads();
        if (tid < 256) {
            unsigned base = 0;
            for (int w = 0; w < warp; ++w) base += part[w];
            run[tid] = base + incl - total + before;
        }
        for (long long i0 = beg; i0 < end; i0 += RADIX_TB) {
            const long long i = i0 + tid;
            const bool valid = i < end;
            const unsigned key = valid ? sk[i] : 0u, val = valid ? sv[i] : 0u;
            const unsigned d = valid ? (key >> shift) & 255u : 256u;
            for (int k = tid; k < NW * 256; k += RADIX_TB) wcnt[k >> 8][k & 255] = 0;
            __syncthreads();
            const unsigned peers = __match_any_sync(0xffffffffu, d);
            if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = __popc(peers);
            __syncthreads();
            if (tid < 256) {  // the warps' counts of digit tid become their starts
                unsigned at = run[tid];
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    const unsigned c = wcnt[w][tid];
                    wcnt[w][tid] = at;
                    at += c;
                }
                run[tid] = at;
            }
            __syncthreads();
            if (valid) {
                const unsigned off = wcnt[warp][d] + __popc(peers & lt_mask);
                dk[off] = key;
                dv[off] = val;
            }
            __syncthreads();
        }
        if (p + 1 < A.passes && !grid_barrier(A.sync, target)) return;
        sk = dk;
        sv = dv;
    }
}

}  // namespace

size_t scan_tmp_size(long long n, size_t elem) {
    size_t s = 0;
    while (true) {
        long long nb = (n + SCAN_TILE - 1) / SCAN_TILE;
        if (nb <= 1) break;
        s += 2 * size_t(nb) * elem + 256;
        n = nb;
    }
    return s + 256;
}

template <class T>
void scan_exclusive(const T *in, T *out, long long n, void *tmp, cudaStream_t st) {
    scan_rec<T>(in, out, n, static_cast<char *>(tmp), nullptr, st);
}
template <class T>
void scan_exclusive_total(const T *in, T *out, long long n, void *tmp, cudaStream_t st) {
    scan_rec<T>(in, out, n, static_cast<char *>(tmp), out + n, st);
}

template void scan_exclusive<int>(const int *, int *, long long, void *, cudaStream_t);
template void scan_exclusive<long long>(const long long *, long long *, long long, void *, cudaStream_t);
template void scan_exclusive_total<int>(const int *, int *, long long, void *, cudaStream_t);
template void scan_exclusive_total<long long>(const long long *, long long *, long long, void *, cudaStream_t);

size_t radix_tmp_size() { return size_t(256) * RADIX_MAX_BLOCKS * sizeof(unsigned); }

void radix_sort_pairs(const unsigned *keys_in, const unsigned *vals_in, unsigned *keys_out, unsigned *vals_out,
                      unsigned *keys_alt, unsigned *vals_alt, long long n, int bits, void *tmp, unsigned *sync,
                      cudaStream_t st) {
    if (n <= 0) return;
    int sms = 0, dev = 0;
    SDOT_CUDA(cudaGetDevice(&dev));
    SDOT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // one block per SM at most: all resident
    const int g = int(std::min<long long>((n + RADIX_TB - 1) / RADIX_TB, std::min(sms, RADIX_MAX_BLOCKS)));
    RadixArgs a{keys_in, vals_in, keys_out, vals_out, keys_alt, vals_alt, static_cast<unsigned *>(tmp), sync, n,
                std::max(1, (bits + 7) / 8)};
    void *args[] = {&a};
    SDOT_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(k_radix_sort), dim3(g), dim3(RADIX_TB), args, 0, st));
    note_launch();
}

}  // namespace sdot
