// CSR sparsity pattern on the device, the same pattern SparseMatrix::initFromPDMesh builds
// (src/MathUtils/SparseMatrix.cpp:73-185) and pxb_csr_pattern restates on the host: per node i the column nodes
// {i} u family(i) u {mirror(i)}, sorted and unique, each expanded to ndof x ndof dense blocks, 0-based.
//
// One warp per node sorts the node list in registers (bitonic, padded to a power of two, strides below 32 by
// shuffles), drops the duplicates with a ballot and writes the list out; an exclusive scan of the lists' lengths over
// the nodes (three kernels: block sums, one block over the sums, block scans) gives every node its first block, and a
// second pass copies the lists to the rows: row (i, a) starts at ndof^2 first(i) + a ndof m_i.  It also writes the
// block view (first block per node, column node per block) that the 2-dof solvers read.
// B200, 73,600 nodes in 3D (8.3 million columns): 54 + 27 us; sorting in shared memory, in the count and again in the
// fill, 205 + 224 us.  With the list index packed beside the node (below kPackedNodes) the sort also leaves the bonds' block
// positions and the rows pass the diagonal slots: 60 + 31 us, where block_map_kernel took 103 us more.
#include <climits>

#include "k_kernels.h"
#include "pxb_common.cuh"

namespace pxb {

namespace {

constexpr int kPatCap = kFamMax;  // largest node list (family + self + mirror) a warp sorts
constexpr int kPatWarps = 4;
constexpr int kScanThreads = 512;

// ascending bitonic sort of 32 E values, element 32 q + lane in v[q]
template <int E>
__device__ __forceinline__ void sort_values(int (&v)[E]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int q = 0; q < E; ++q) {
                    const int p = q ^ (j / 32);
                    if (p > q) {
                        const bool up = (32 * q & k) == 0;
                        const int lo = min(v[q], v[p]), hi = max(v[q], v[p]);
                        v[q] = up ? lo : hi;
                        v[p] = up ? hi : lo;
                    }
                }
            } else {
#pragma unroll
                for (int q = 0; q < E; ++q) {
                    const int o = __shfl_xor_sync(kFull, v[q], j);
                    const bool up = ((32 * q + lane) & k) == 0, low = (lane & j) == 0;
                    v[q] = up == low ? min(v[q], o) : max(v[q], o);
                }
            }
        }
}

// node i's own, family and mirror nodes, sorted and unique, to out; returns how many.  PACKED: a value is node << 8 | index
// in the unsorted list, so that every entry's position in the sorted one is known when it is written (bpos, spos, xpos).
template <int E, bool PACKED>
__device__ __forceinline__ int node_list(const PatternArgs &a, int i, int b0, int len, int mir, int *out) {
    const int lane = threadIdx.x & 31, tot = len + 1 + (mir >= 0 ? 1 : 0);
    int v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int k = 32 * q + lane;
        v[q] = k < len ? a.nbr[b0 + k] : (k == len ? i : (k < tot ? mir : INT_MAX));
        if (PACKED && k < tot) v[q] = v[q] << 8 | k;
    }
    sort_values<E>(v);
    int m = 0, last = -1;  // last: the node before element 32 q
    bool own_kept = true;
    int at_mirror = -1;
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int node = PACKED ? v[q] >> 8 : v[q], k = v[q] & 255;
        int before = __shfl_up_sync(kFull, node, 1);
        if (lane == 0) before = last;
        const bool in = 32 * q + lane < tot, keep = in && node != before;
        const unsigned ball = __ballot_sync(kFull, keep);
        const int at = m + __popc(ball & ((1u << lane) - 1u));
        if (keep) out[at] = node;
        if (PACKED && in) {  // of a node listed twice the family's entry comes first, the mirror's last
            if (k < len) a.bpos[b0 + k] = (uint8_t)at;
            else if (k == len) a.spos[i] = (uint8_t)at;
            else if (keep) at_mirror = at;
            if (k <= len && !keep) own_kept = false;
        }
        m += __popc(ball);
        last = __shfl_sync(kFull, node, 31);
    }
    if constexpr (PACKED) {
        at_mirror = __reduce_max_sync(kFull, at_mirror);
        own_kept = __all_sync(kFull, own_kept);
        if (lane == 0) {
            a.xpos[i] = (int16_t)at_mirror;
            if (!own_kept) atomicAdd(a.inexact, 1);
        }
    }
    return m;
}

template <bool PACKED>
__global__ void __launch_bounds__(kPatWarps * 32) pattern_list_kernel(PatternArgs a) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = blockIdx.x * kPatWarps + w; i < a.n; i += gridDim.x * kPatWarps) {
        const int b0 = a.off[i], len = a.off[i + 1] - b0, m0 = a.mirror ? a.mirror[i] : 0;
        const int mir = m0 >= 1 && m0 <= a.n ? m0 - 1 : -1, tot = len + 1 + (mir >= 0 ? 1 : 0);
        int *out = a.list + ((size_t)b0 + 2 * (size_t)i);
        int m = -1;
        if (tot <= 32) m = node_list<1, PACKED>(a, i, b0, len, mir, out);
        else if (tot <= 64) m = node_list<2, PACKED>(a, i, b0, len, mir, out);
        else if (tot <= 128) m = node_list<4, PACKED>(a, i, b0, len, mir, out);
        else if (tot <= kPatCap) m = node_list<8, PACKED>(a, i, b0, len, mir, out);
        if (lane == 0) {
            if (m < 0) atomicAdd(a.overflow, 1);
            a.count[i] = m < 0 ? 0 : m;
        }
    }
}

__global__ void __launch_bounds__(kPatWarps * 32) pattern_rows_kernel(PatternArgs a) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = blockIdx.x * kPatWarps + w; i < a.n; i += gridDim.x * kPatWarps) {
        if (i == a.n - 1 && lane == 0) {
            a.rowptr[(size_t)a.n * a.ndof] = (int)((long long)a.ndof * a.ndof * a.first[a.n]);
            if (a.bptr) a.bptr[a.n] = (int)a.first[a.n];
        }
        const int *list = a.list + ((size_t)a.off[i] + 2 * (size_t)i);
        const long long first = a.first[i];
        const int nd = a.ndof, m = a.count[i];
        for (int k = lane; k < m; k += 32) {
            const int node = list[k];
            if (a.bcol) a.bcol[first + k] = node;
            for (int r = 0; r < nd; ++r) {
                const long long row0 = (long long)nd * nd * first + (long long)r * m * nd;
                for (int b = 0; b < nd; ++b) a.cols[row0 + (long long)k * nd + b] = node * nd + b;
            }
        }
        if (a.diag && lane < nd * nd)
            a.diag[(size_t)i * nd * nd + lane] =
                (int)((long long)nd * nd * first + (long long)(lane / nd) * m * nd + a.spos[i] * nd + lane % nd);
        if (lane < nd) a.rowptr[(size_t)i * nd + lane] = (int)((long long)nd * nd * first + (long long)lane * m * nd);
        if (a.bptr && lane == 0) a.bptr[i] = (int)first;
    }
}

// exclusive scan of count[0, n) into first[0, n] (first[n] = total), 64-bit sums
__global__ void __launch_bounds__(kScanThreads) scan_blocks_kernel(int n, const int *count, long long *bsum,
                                                                   int *maxv) {
    __shared__ long long sh[kScanThreads / 32];
    const int i = blockIdx.x * kScanThreads + threadIdx.x;
    const int mine = i < n ? count[i] : 0;
    if (maxv) {
        const int top = __reduce_max_sync(kFull, mine);
        if ((threadIdx.x & 31) == 0 && top > 0) atomicMax(maxv, top);
    }
    const long long v = group_sum<kWarp>((long long)mine);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long t = 0;
        for (int k = 0; k < kScanThreads / 32; ++k) t += sh[k];
        bsum[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(int nblocks, long long *bsum, long long *total) {
    __shared__ long long carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int c = 0; c < nblocks; c += kScanThreads) {
        const int k = c + threadIdx.x;
        const long long v = k < nblocks ? bsum[k] : 0;
        long long incl = v;  // inclusive warp scan, then across warps
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(kFull, incl, o);
            if ((threadIdx.x & 31) >= o) incl += t;
        }
        __shared__ long long wsum[kScanThreads / 32];
        if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = incl;
        __syncthreads();
        long long before = carry;
        for (int q = 0; q < (int)(threadIdx.x >> 5); ++q) before += wsum[q];
        if (k < nblocks) bsum[k] = before + incl - v;
        __syncthreads();
        if (threadIdx.x == kScanThreads - 1) carry = before + incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

template <typename T>
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(int n, const int *count, const long long *bsum,
                                                                  const long long *total, T *first) {
    __shared__ long long wsum[kScanThreads / 32];
    const int i = blockIdx.x * kScanThreads + threadIdx.x;
    const long long v = i < n ? count[i] : 0;
    long long incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(kFull, incl, o);
        if ((threadIdx.x & 31) >= o) incl += t;
    }
    if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = incl;
    __syncthreads();
    long long before = bsum[blockIdx.x];
    for (int q = 0; q < (int)(threadIdx.x >> 5); ++q) before += wsum[q];
    if (i < n) first[i] = (T)(before + incl - v);
    if (i == n - 1 || (n == 0 && i == 0)) first[n] = (T)*total;
}

int pattern_grid(int n) {
    const int g = (n + kPatWarps - 1) / kPatWarps;
    return g < 1 ? 1 : (g < 148 * 16 ? g : 148 * 16);
}

template <typename T>
cudaError_t scan(int n, const int *count, long long *bsum, long long *total, T *first, int *maxv, cudaStream_t s) {
    const int nb = scan_blocks(n);
    scan_blocks_kernel<<<nb, kScanThreads, 0, s>>>(n, count, bsum, maxv);
    scan_sums_kernel<<<1, kScanThreads, 0, s>>>(nb, bsum, total);
    scan_apply_kernel<T><<<nb, kScanThreads, 0, s>>>(n, count, bsum, total, first);
    return cudaGetLastError();
}

}  // namespace

int scan_blocks(int n) { return (n + kScanThreads - 1) / kScanThreads > 0 ? (n + kScanThreads - 1) / kScanThreads : 1; }

cudaError_t launch_scan(int n, const int *count, long long *bsum, long long *total, int *first, int *maxv, cudaStream_t s) {
    return scan(n, count, bsum, total, first, maxv, s);
}

cudaError_t launch_scan(int n, const int *count, long long *bsum, long long *total, long long *first, int *maxv,
                        cudaStream_t s) {
    return scan(n, count, bsum, total, first, maxv, s);
}

cudaError_t launch_pattern_count(const PatternArgs &a, cudaStream_t s) {
    if (a.bpos) pattern_list_kernel<true><<<pattern_grid(a.n), kPatWarps * 32, 0, s>>>(a);
    else pattern_list_kernel<false><<<pattern_grid(a.n), kPatWarps * 32, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pattern_fill(const PatternArgs &a, cudaStream_t s) {
    pattern_rows_kernel<<<pattern_grid(a.n), kPatWarps * 32, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace pxb
