// CSR Jacobian value assembly on exact block patterns: every row of a node holds the same list of column nodes (its
// own, its family's and its mirror's), each expanded to ndof columns, as SparseMatrix::initFromPDMesh builds it
// (src/MathUtils/SparseMatrix.cpp:73-185).  The element physics is that of k_csr.cu, whose kernels serve any other
// pattern.
//
// What bounds the assembly is memory: the values alone are 8 ndof^2 bytes a bond.  On a block pattern
//   * a bond needs one 1-byte block position instead of ndof^2 4-byte slots (100 bytes at five unknowns);
//   * the rows of a node are one contiguous span of the value array, so the node's values are put together in shared
//     memory and leave as one coalesced copy, every entry written once: no zeroing pass, no 8-byte stores scattered
//     over the rows (each of which cost a 32-byte L2 sector);
//   * the operator rows of a family are one contiguous span too, read coalesced into shared memory.
// B200: 38,912 nodes in 3D with five unknowns (4.29 M bonds, 1.30 GB necessary) 783 us with slots -> 391 us; 81,200
// nodes in 2D with two unknowns (2.25 M bonds, 171 MB) 96 -> 63 us.  What bounds both is the L1 data pipe (65 % of
// its peak at 428 and 66 us, four nodes a tile in 2D: the values pass through shared memory once, with bank conflicts where a family's positions are not
// consecutive), then DRAM latency (24-31 % occupancy there, limited by registers and the tile's shared memory; MINB below).
#include <type_traits>

#include "k_kernels.h"
#include "pxb_common.cuh"

namespace pxb {

namespace {

__device__ __forceinline__ double clamp_c(double c) { return fmax(1.0e-8, fmin(1.0 - 1.0e-8, c)); }

// position of `node` in a sorted list of m nodes read as list(p); -1 when absent
template <typename F>
__device__ __forceinline__ int find_block(F list, int m, int node) {
    int l = 0, h = m - 1;
    while (l <= h) {
        const int mid = (l + h) >> 1, v = list(mid);
        if (v == node) return mid;
        if (v < node) l = mid + 1; else h = mid - 1;
    }
    return -1;
}

__device__ __forceinline__ void copy8_async(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_fence() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int NT>
__device__ __forceinline__ void tile_sync() {
    if constexpr (NT == kWarp) __syncwarp();
    else __syncthreads();
}

// doubles of a tile's shared memory: the values of its nodes' rows, the bonds' residual terms, the operator rows, the nodal
// words and values
template <typename El>
__host__ __device__ constexpr int tile_doubles(int mmax) {
    return El::TN * (mmax * (El::ND * El::ND + El::ND + El::NOP) + El::NQ + 3) + 2;
}

}  // namespace

// ---- block positions ------------------------------------------------------------------------------------------
// Warp per node: checks (verify: a caller's pattern) that node i's rows are one sorted block list, finds every bond's
// position in it, the node's own and that of a mirror block outside the family; *inexact counts the nodes whose rows
// are anything else (then the slot map of k_csr.cu serves the pattern).
__global__ void __launch_bounds__(128) block_map_kernel(BlockMapArgs a) {
    __shared__ unsigned taken[4][kBlockMax / 32];
    __shared__ int nodes[4][kBlockMax];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nd = a.ndof;
    for (int i = blockIdx.x * 4 + w; i < a.n; i += gridDim.x * 4) {
        const int lo = a.rowptr[i * nd], width = a.rowptr[i * nd + 1] - lo, m = width / nd;
        const int b0 = a.off[i], len = a.off[i + 1] - b0;
        bool ok = width == m * nd && m > 0 && m <= kBlockMax;
        if (ok && a.verify) {
            bool same = (i > 0 || lo == 0) && lo >= 0 && lo + (long long)nd * width <= a.nnz;
            for (int r = lane; r <= nd; r += kWarp) same = same && a.rowptr[i * nd + r] == lo + r * width;
            ok = __all_sync(kFull, same);
        }
        if (ok && a.verify) {  // every entry read below lies in [lo, lo + nd width), inside the pattern
            bool same = true;
            for (int p = lane; p < m; p += kWarp) {
                const int node = a.cols[lo + p * nd] / nd;
                same = same && node >= 0 && node < a.n && (p == 0 || a.cols[lo + (p - 1) * nd] < node * nd);
                for (int r = 0; r < nd; ++r)
                    for (int c = 0; c < nd; ++c)
                        same = same && a.cols[lo + (long long)r * width + p * nd + c] == node * nd + c;
            }
            ok = __all_sync(kFull, same);
        }
        if (ok) {
            if (lane < kBlockMax / 32) taken[w][lane] = 0;
            for (int p = lane; p < m; p += kWarp) nodes[w][p] = a.cols[lo + p * nd] / nd;
            __syncwarp();
            auto list = [&](int p) { return nodes[w][p]; };
            const int mir = a.mirror ? a.mirror[i] - 1 : -1;
            bool has_mirror = mir == i, found = true;
            for (int k = lane; k < len; k += kWarp) {
                const int j = a.nbr[b0 + k];
                const int p = find_block(list, m, j);
                if (p >= 0) {
                    atomicOr(&taken[w][p >> 5], 1u << (p & 31));
                    a.bpos[b0 + k] = (uint8_t)p;
                }
                found = found && p >= 0;
                has_mirror = has_mirror || j == mir;
            }
            const bool extra = mir >= 0 && !__any_sync(kFull, has_mirror);
            const int ps = find_block(list, m, i), px = extra ? find_block(list, m, mir) : -1;
            __syncwarp();
            // own block, one block a family member, the extra mirror's block: every position of the list exactly once
            const int fam = __reduce_add_sync(kFull, lane < kBlockMax / 32 ? __popc(taken[w][lane]) : 0);
            ok = __all_sync(kFull, found) && ps >= 0 && !(taken[w][ps >> 5] >> (ps & 31) & 1u) && fam == len &&
                 (!extra || px >= 0) && m == 1 + len + (extra ? 1 : 0);
            if (ok && lane == 0) {
                a.spos[i] = (uint8_t)ps;
                a.xpos[i] = (int16_t)px;
            }
            for (int e = lane; ok && e < nd * nd; e += kWarp)
                a.diag[(size_t)i * nd * nd + e] = lo + (e / nd) * width + ps * nd + e % nd;
            __syncwarp();
        }
        if (!ok && lane == 0) atomicAdd(a.inexact, 1);
    }
}

cudaError_t launch_block_map(const BlockMapArgs &a, cudaStream_t s) {
    const int g = (a.n + 3) / 4;
    block_map_kernel<<<g < 1 ? 1 : (g < 148 * 16 ? g : 148 * 16), 128, 0, s>>>(a);
    return cudaGetLastError();
}

// ---- the assembly skeleton ---------------------------------------------------------------------------------------
// A block of NT threads (a warp in 2D, four warps in 3D) takes TN consecutive nodes at a time, two in 2D and one in 3D, whose
// bonds' ids, operator rows and values are contiguous.  A long tile is a long chain for a mesh that does not fill the chip, a
// short one has fewer bonds than threads.  2D with one, two and four nodes a tile, us a call (kernels with slots last):
//   stress-CH         1,024 nodes 10.7 / 10.3 / 14.4 (10.3), 22,500 64 / 63 / 76 (113), 90,000 228 / 208 / 272 (425)
//   dynamic fracture  1,024 nodes 6.2 / 6.2 / 8.2 (6.2), 22,500 24.6 / 18.5 / 20.5 (22.6), 90,000 109 / 67 / 72 (102)
// Per tile:
//   bonds     a bond a thread and pass: -K_IJ into the tile's rows in shared memory, the residual terms beside them;
//   ahead     the next tile's bond words (registers), nodal values and operator rows (asynchronous copies) start out;
//   nodes     one entry of a diagonal block or right-hand side a thread (SEG threads where there are enough): the sum
//             over the node's blocks in shared memory, plus the nodal term;
//   store     the rows leave as one contiguous copy.
// El: the element.  Bond: what a thread holds of a bond; nodal(): the NQ values of a node the bonds and the epilogue
// read; bond(): -K_IJ at kb (row r at kb + r W) and the ND residual terms; diag() / rhs(): the entry from its sum.
template <typename El, int NT>
__global__ void __launch_bounds__(NT, El::MINB) node_rows_kernel(El el, BlockPattern bp, int mmax) {
    constexpr int ND = El::ND, TN = El::TN, NQ = El::NQ, P = El::P, NE = ND * ND + ND, NOP = El::NOP;
    constexpr int SEG = NT / (TN * NE) >= 16 ? 16 : NT / (TN * NE) >= 8 ? 8 : NT / (TN * NE) >= 4 ? 4 : NT / (TN * NE) >= 2 ? 2 : 1;
    extern __shared__ __align__(16) double sm_blk[];
    const int tid = threadIdx.x;
    double *rows = sm_blk;                            // [values of the tile]
    double *res = rows + TN * mmax * ND * ND;         // [bond][ND]
    double *ops = res + TN * mmax * ND;               // [bond][NOP]
    double *nq = ops + TN * mmax * NOP;               // [node][NQ]
    int *so = reinterpret_cast<int *>(nq + TN * NQ);  // bond offsets within the tile [TN + 1]
    int *sw = so + TN + 1, *sp = sw + TN;                           // row length; own block | (mirror block + 1) << 8 | dead << 24
    const int n = el.a.n, stride = gridDim.x, ntiles = (n + TN - 1) / TN;

    // the tile being fetched: bond range, bond words, and (thread k < TN) the words of node k
    int f0 = 0, f1 = 0, flo = 0, fo = 0, fw = 0, fp = 0;
    typename El::Bond bq[P];
    double fq[NQ];
    auto range = [&](int tile, int &b0, int &b1) {
        b0 = b1 = 0;
        if (tile < ntiles) {
            b0 = __ldg(el.a.off + tile * TN);
            b1 = __ldg(el.a.off + min((tile + 1) * TN, n));
        }
    };
    auto fetch = [&](int tile, int b0, int b1) {
        f0 = b0;
        f1 = b1;
        if (tile < ntiles) {
            const int i0 = tile * TN, i = i0 + tid;
            flo = __ldg(el.a.rowptr + i0 * ND);
#pragma unroll
            for (int p = 0; p < P; ++p)
                if (b0 + tid + p * NT < b1) bq[p] = el.load(b0 + tid + p * NT);
            el.template stage<NT>(b0, b1, tid, ops);
            fo = b1;
            fw = 0;
            fp = 1 << 24;
            if (tid < TN && i < n) {
                fo = __ldg(el.a.off + i);
                fw = __ldg(el.a.rowptr + i * ND + 1) - __ldg(el.a.rowptr + i * ND);
                fp = __ldg(bp.spos + i) | (__ldg(bp.xpos + i) + 1) << 8 | (el.dead(i) ? 1 << 24 : 0);
                el.nodal(i, fq);
            }
        }
    };

    int tile = blockIdx.x;
    int n0, n1;  // bond range of the tile after the one being fetched
    range(tile, n0, n1);
    fetch(tile, n0, n1);
    range(tile + stride, n0, n1);
    for (; tile < ntiles; tile += stride) {
        const int b0 = f0, nb = f1 - f0, i0 = tile * TN;
        const size_t lo = flo;
        tile_sync<NT>();  // the previous tile's rows have left
        if (tid < TN) {
            so[tid] = fo - b0;
            sw[tid] = fw;
            sp[tid] = fp;
#pragma unroll
            for (int k = 0; k < NQ; ++k) nq[tid * NQ + k] = fq[k];
        }
        if (tid == 0) so[TN] = nb;
        copy_fence();
        tile_sync<NT>();  // words, values and operator rows of this tile are here
        int rbase[TN];  // first value of each node's rows
        int len = 0;
#pragma unroll
        for (int k = 0; k < TN; ++k) {
            rbase[k] = len;
            len += sw[k] * ND;
        }
        auto bond = [&](int q, const typename El::Bond &b) {
            int k = 0, r0 = 0;
#pragma unroll
            for (int e = 1; e < TN; ++e)
                if (q >= so[e]) {
                    k = e;
                    r0 = rbase[e];
                }
            const int W = sw[k];
            double *kb = rows + r0 + __ldg(bp.bpos + b0 + q) * ND;
            if (!(sp[k] >> 24)) {
                el.bond(i0 + k, nq + k * NQ, b, ops + q * NOP, kb, W, res + q * ND);
            } else {
#pragma unroll
                for (int r = 0; r < ND; ++r)
#pragma unroll
                    for (int c = 0; c < ND; ++c) kb[r * W + c] = 0.0;
            }
        };
#pragma unroll
        for (int p = 0; p < P; ++p)
            if (tid + p * NT < nb) bond(tid + p * NT, bq[p]);
        for (int q = tid + P * NT; q < nb; q += NT) bond(q, el.load(b0 + q));
        tile_sync<NT>();
        fetch(tile + stride, n0, n1);
        range(tile + 2 * stride, n0, n1);
        // diagonal blocks, mirror blocks and right-hand sides
        for (int x = tid; x < ((TN * NE * SEG + NT - 1) / NT) * NT; x += NT) {
            const int e = x / SEG, sg = x % SEG, k = e / NE, en = e % NE;
            double sum = 0.0;
            int q0 = 0, m = 0, W = 0, w = 1 << 24, r0 = 0;
            const bool on = e < TN * NE && i0 + k < n;
            const int r = en < ND * ND ? en / ND : en - ND * ND, c = en % ND;
            if (on) {
                W = sw[k];
                w = sp[k];
                q0 = so[k];
                m = so[k + 1] - q0;
#pragma unroll
                for (int g = 1; g < TN; ++g)
                    if (k == g) r0 = rbase[g];
                if (!(w >> 24)) {
                    const int ps = w & 255;
                    if (en < ND * ND) {
                        const double *src = rows + r0 + r * W + c;
                        const int blocks = W / ND, px = (w >> 8 & 0xffff) - 1;
                        double s1 = 0.0;  // two chains; the own block and a mirror block hold nothing yet
                        for (int p = sg; p < blocks; p += 2 * SEG) {
                            if (p != ps && p != px) sum -= src[p * ND];
                            const int p2 = p + SEG;
                            if (p2 < blocks && p2 != ps && p2 != px) s1 -= src[p2 * ND];
                        }
                        sum += s1;
                    } else {
                        double s1 = 0.0;
                        for (int p = sg; p < m; p += 2 * SEG) {
                            sum += res[(q0 + p) * ND + r];
                            if (p + SEG < m) s1 += res[(q0 + p + SEG) * ND + r];
                        }
                        sum += s1;
                    }
                }
            }
#pragma unroll
            for (int o = SEG / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
            if (on && sg == 0) {
                const bool dead = w >> 24;
                if (en < ND * ND) {
                    const int px = (w >> 8 & 0xffff) - 1;
                    rows[r0 + r * W + (w & 255) * ND + c] = dead ? 0.0 : el.diag(nq + k * NQ, r, c, sum);
                    if (px >= 0) rows[r0 + r * W + px * ND + c] = 0.0;
                } else {
                    el.a.rhs[(i0 + k) * ND + r] = dead ? 0.0 : el.rhs(nq + k * NQ, r, sum);
                }
            }
        }
        tile_sync<NT>();
        double *dst = el.a.kvals + lo;
        int k = tid;
        for (; k + 3 * NT < len; k += 4 * NT) {
            const double v0 = rows[k], v1 = rows[k + NT], v2 = rows[k + 2 * NT], v3 = rows[k + 3 * NT];
            dst[k] = v0;
            dst[k + NT] = v1;
            dst[k + 2 * NT] = v2;
            dst[k + 3 * NT] = v3;
        }
        for (; k < len; k += NT) dst[k] = rows[k];
    }
}

// ---- stress-coupled Cahn-Hilliard (rows c, mu, u; see assemble_stress_ch_kernel in k_csr.cu for the terms) -------
template <int DIM>
struct StressChEl {
    static constexpr int ND = DIM + 2, NOP = DIM == 3 ? 9 : 5, TN = DIM == 3 ? 1 : 2, P = TN;
    // nodal values: u[ND], V, M, 1/V, (c_old, -, u - u_old - v dt)[ND]
    // resident blocks: 3D (128 threads) 5, against 4 391 us of 427 at the size above, 3 506, 6 455; 2D (one warp a block) 14,
    // against 12 208 us of 217 on 90,000 nodes, 18 221
    static constexpr int NQ = 2 * ND + 3, MINB = DIM == 3 ? 5 : 14;
    // operator slots in the multi-index order: first derivatives, then xx xy [xz] yy [yz zz]
    static constexpr int SXX = DIM, SXY = DIM + 1, SXZ = 5, SYY = DIM == 3 ? 6 : 4, SYZ = 7, SZZ = 8;
    StressChAsmArgs a;
    struct Bond {
        int j;
        uint8_t f;
        double g, lap, lrv;
    };
    __device__ __forceinline__ bool dead(int i) const { return a.degenerate && __ldg(a.degenerate + i); }
    __device__ __forceinline__ void nodal(int i, double *q) const {
#pragma unroll
        for (int b = 0; b < ND; ++b) q[b] = __ldg(a.u + i * ND + b);
        q[ND] = __ldg(a.vol + i);
        q[ND + 1] = __ldg(a.mnode + i);
        q[ND + 2] = 1.0 / q[ND];
#pragma unroll
        for (int b = 0; b < ND; ++b) {
            double o = a.uold ? __ldg(a.uold + i * ND + b) : 0.0;
            if (b >= 2) o = a.vel ? q[b] - o - __ldg(a.vel + (size_t)i * DIM + b - 2) * a.dt : 0.0;
            q[ND + 3 + b] = o;
        }
    }
    template <int NT>
    __device__ __forceinline__ void stage(int b0, int b1, int tid, double *dst) const {
        const double *src = a.ops + (size_t)b0 * NOP;
        for (int k = tid; k < (b1 - b0) * NOP; k += NT) copy8_async(dst + k, src + k);
    }
    __device__ __forceinline__ Bond load(int t) const {
        Bond b;
        b.j = __ldcs(a.nbr + t);
        b.f = __ldcs(a.bfl + t);
        b.g = a.health ? (__ldcs(a.health + t) > 0.0 ? 1.0 : a.kres) : 1.0;
        b.lap = __ldcs(a.lap + t);
        b.lrv = __ldcs(a.lrv + t);
        return b;
    }
    __device__ __forceinline__ void bond(int, const double *q, const Bond &b, const double *op, double *kb, int W,
                                         double *res) const {
        double dv[ND];
#pragma unroll
        for (int e = 0; e < ND; ++e) dv[e] = __ldg(a.u + (size_t)b.j * ND + e) - q[e];
        double kc = 0.0, km = 0.0;
        if (!(b.f & 1)) {  // bonds to ghosts carry no species flux
            const double Mi = q[ND + 1];
            kc = (b.f & 2) && q[ND] > 0.0 ? species_flux(Mi, b.lap, b.lrv, q[ND + 2], __ldg(a.mnode + b.j)) : -(Mi * b.lap);
            km = a.kappa * b.lap;
        }
        const double Gxx = b.g * op[SXX], Gxy = b.g * op[SXY], Gyy = b.g * op[SYY];
        double P[DIM][DIM];
        if constexpr (DIM == 2) {
            P[0][0] = a.C11 * Gxx + a.C66 * Gyy;
            P[0][1] = P[1][0] = (a.C12 + a.C66) * Gxy;
            P[1][1] = a.C66 * Gxx + a.C11 * Gyy;
        } else {
            const double Gzz = b.g * op[SZZ], Gxz = b.g * op[SXZ], Gyz = b.g * op[SYZ], cc = a.C12 + a.C66;
            P[0][0] = a.C11 * Gxx + a.C66 * (Gyy + Gzz);
            P[1][1] = a.C11 * Gyy + a.C66 * (Gxx + Gzz);
            P[2][2] = a.C11 * Gzz + a.C66 * (Gxx + Gyy);
            P[0][1] = P[1][0] = cc * Gxy;
            P[0][2] = P[2][0] = cc * Gxz;
            P[1][2] = P[2][1] = cc * Gyz;
        }
        kb[0] = 0.0;
        kb[1] = -kc;
        kb[W] = -km;
        kb[W + 1] = 0.0;
        res[0] = kc * dv[1];
        double r1 = km * dv[0];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const double G1 = b.g * op[d], kg = a.Omega * a.Kh * G1, kf = -a.A * G1;
            kb[2 + d] = 0.0;
            kb[W + 2 + d] = -kg;
            kb[(2 + d) * W] = -kf;
            kb[(2 + d) * W + 1] = 0.0;
            r1 += kg * dv[2 + d];
            double rd = kf * dv[0];
#pragma unroll
            for (int e = 0; e < DIM; ++e) {
                kb[(2 + d) * W + 2 + e] = -P[d][e];
                rd += P[d][e] * dv[2 + e];
            }
            res[2 + d] = rd;
        }
        res[1] = r1;
    }
    __device__ __forceinline__ double diag(const double *q, int r, int c, double sum) const {
        if (r == 0) return c == 0 ? -(1.0 / a.dt) : sum;
        if (r == 1 && c == 0) {
            const double cc = clamp_c(q[0]);
            return -(-(1.0 / (cc * (1.0 - cc)) - 2.0 * a.chi) + a.Omega * a.Ch) + sum;
        }
        if (r == 1 && c == 1) return -1.0;
        if (r == c && a.rho > 0.0 && a.vel) return a.rho / (a.dt * a.dt) + sum;
        return sum;
    }
    __device__ __forceinline__ double rhs(const double *q, int r, double sum) const {
        const double c = q[0], cc = clamp_c(c);
        double l = 0.0;
        if (r == 0) l = (c - q[ND + 3]) / a.dt;
        else if (r == 1) l = q[1] - (log(cc / (1.0 - cc)) + a.chi * (1.0 - 2.0 * cc)) + a.Omega * a.Ch * (c - a.cref);
        else if (a.rho > 0.0 && a.vel) l = -(a.rho / (a.dt * a.dt)) * q[ND + 3 + r];
        return l + sum;
    }
};

// ---- implicit dynamic fracture (rows u; see assemble_cached_kernel in k_csr.cu) ------------------------------------
template <int DIM>
struct CachedEl {
    static constexpr int ND = DIM, NOP = DIM == 3 ? 9 : 5, NP = DIM == 3 ? 6 : 3, TN = DIM == 3 ? 1 : 2, P = TN;
    static constexpr int NQ = 2 * ND;  // u, u - u_old - v dt
    static constexpr int MINB = DIM == 3 ? 6 : 28;  // 2D: 66.7 us on 90,000 nodes against 69.2 with 10, 68.0 with 24, 67.7 with 32
    static constexpr int SXX = DIM, SXY = DIM + 1, SXZ = 5, SYY = DIM == 3 ? 6 : 4, SYZ = 7, SZZ = 8;
    CachedAsmArgs a;
    struct Bond {
        int j;
        double h;
    };
    __device__ __forceinline__ bool dead(int i) const { return a.degenerate && __ldg(a.degenerate + i); }
    __device__ __forceinline__ void nodal(int i, double *q) const {
#pragma unroll
        for (int b = 0; b < ND; ++b) {
            q[b] = __ldg(a.u + i * ND + b);
            const double uo = a.uold ? __ldg(a.uold + i * ND + b) : 0.0;
            const double v = a.nodecache ? __ldg(a.nodecache + (size_t)i * a.ncache + b) : 0.0;
            q[ND + b] = q[b] - uo - v * a.dt;
        }
    }
    template <int NT>
    __device__ __forceinline__ void stage(int b0, int b1, int tid, double *dst) const {
        const double *src = a.ops + (size_t)b0 * NOP;
        for (int k = tid; k < (b1 - b0) * NOP; k += NT) copy8_async(dst + k, src + k);
    }
    __device__ __forceinline__ Bond load(int t) const {
        return {__ldcs(a.nbr + t), a.bondcache ? __ldg(a.bondcache + (size_t)t * a.nbcache) : 1.0};
    }
    __device__ __forceinline__ void bond(int i, const double *q, const Bond &b, const double *op, double *kb, int W,
                                         double *res) const {
        using PosT = typename Vec<DIM>::T;
        double dv[ND];
#pragma unroll
        for (int e = 0; e < ND; ++e) dv[e] = __ldg(a.u + (size_t)b.j * ND + e) - q[e];
        const double Gxx = op[SXX], Gxy = op[SXY], Gyy = op[SYY], h = b.h;
        bool skip = false;
        if (Gxx == 0.0 && Gxy == 0.0 && Gyy == 0.0) {
            // a zero-length bond carries nothing (not even 0 times a non-finite u); its operators are zero, so only
            // such bonds look at the positions
            const PosT *pos = static_cast<const PosT *>(a.pos);
            const PosT xi = pos[i], xj = pos[b.j];
            double r2 = (xj.x - xi.x) * (xj.x - xi.x) + (xj.y - xi.y) * (xj.y - xi.y);
            if constexpr (DIM == 3) r2 += (xj.z - xi.z) * (xj.z - xi.z);
            skip = !(r2 > 0.0);
        }
        double P[NP];
#pragma unroll
        for (int e = 0; e < NP; ++e) P[e] = 0.0;
        if (h > 0.0 && !skip) {
            if constexpr (DIM == 2) {
                P[0] = h * (a.C11 * Gxx + a.C66 * Gyy);
                P[1] = h * (a.C12 + a.C66) * Gxy;
                P[2] = h * (a.C66 * Gxx + a.C11 * Gyy);
            } else {
                const double Gxz = op[SXZ], Gyz = op[SYZ], Gzz = op[SZZ], cc = a.C12 + a.C66;
                P[0] = h * (a.C11 * Gxx + a.C66 * (Gyy + Gzz));
                P[1] = h * (a.C11 * Gyy + a.C66 * (Gxx + Gzz));
                P[2] = h * (a.C11 * Gzz + a.C66 * (Gxx + Gyy));
                P[3] = h * cc * Gxy;
                P[4] = h * cc * Gxz;
                P[5] = h * cc * Gyz;
            }
        }
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            double rr = 0.0;
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
                const double p = DIM == 2 ? P[r + c] : P[r == c ? r : r + c + 2];
                kb[r * W + c] = -p;
                rr += p * dv[c];
            }
            res[r] = skip ? 0.0 : rr;
        }
    }
    __device__ __forceinline__ double diag(const double *, int r, int c, double sum) const {
        return r == c ? sum + a.rho / (a.dt * a.dt) : sum;
    }
    __device__ __forceinline__ double rhs(const double *q, int r, double sum) const {
        return (a.b[r] - a.rho / (a.dt * a.dt) * q[ND + r]) + sum;
    }
};

// ---- conservative Cahn-Hilliard (rows c, mu; see assemble_ch_kernel in k_csr.cu) ----------------------------------
// LPN lanes a node; a bond's two row pieces are 16 bytes each (VEC: the value array is 16-byte aligned), so they go
// straight to memory: with two unknowns the tile of node_rows_kernel costs more than it saves (256x256: 48.9 us against
// 42.4 us with slots; here the 40 assemblies of a 10-step run take 0.34 ms less than with slots)
template <int LPN, bool VEC>
__global__ void __launch_bounds__(256) ch_block_kernel(ChAsmArgs a, BlockPattern bp) {
    constexpr int GPW = kWarp / LPN;
    const int lane = threadIdx.x & 31, gl = lane & (LPN - 1), grp = lane / LPN;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    auto put = [](double *p, double x, double y) {
        if constexpr (VEC) {
            *reinterpret_cast<double2 *>(p) = make_double2(x, y);
        } else {
            p[0] = x;
            p[1] = y;
        }
    };
    for (int base = warp * GPW; base < a.n; base += nwarps * GPW) {
        const int i = base + grp;
        const bool act = i < a.n;
        double c = 0.0, mu = 0.0, Vi = 0.0, Mi = 0.0, cold = 0.0;
        int b0 = 0, b1 = 0, lo = 0, W = 0, ps = 0;
        if (act) {
            b0 = a.off[i];
            b1 = a.off[i + 1];
            lo = a.rowptr[2 * i];
            W = a.rowptr[2 * i + 1] - lo;
            c = a.u[2 * (size_t)i];
            mu = a.u[2 * (size_t)i + 1];
            Vi = a.vol[i];
            Mi = a.mnode[i];
            cold = a.uold[2 * (size_t)i];
            ps = bp.spos[i];
            const int px = bp.xpos[i];
            if (px >= 0 && gl < 2) put(a.kvals + lo + gl * W + 2 * px, 0.0, 0.0);
        }
        double *kv = a.kvals + lo;
        const double iV = 1.0 / Vi;
        double rcs = 0.0, rms = 0.0, k12 = 0.0, k21 = 0.0;
        for (int t = b0 + gl; t < b1; t += LPN) {
            const int j = __ldg(a.nbr + t);
            const double g2 = a.lap[t];
            const uint8_t f = a.bfl[t];
            double *kb = kv + 2 * bp.bpos[t];
            double kc = 0.0, km = 0.0;
            if (!(f & 1)) {
                kc = (f & 2) && Vi > 0.0 ? species_flux(Mi, g2, a.lrv[t], iV, a.mnode[j]) : -(Mi * g2);
                km = a.kappa * g2;
            }
            rcs += kc * (a.u[2 * (size_t)j + 1] - mu);  // u may be only 8-byte aligned (a caller's pointer)
            rms += km * (a.u[2 * (size_t)j] - c);
            k12 += kc;
            k21 += km;
            put(kb, 0.0, -kc);      // (c,  c_j mu_j)
            put(kb + W, -km, 0.0);  // (mu, c_j mu_j)
        }
        rcs = group_sum<LPN>(rcs);
        rms = group_sum<LPN>(rms);
        k12 = group_sum<LPN>(k12);
        k21 = group_sum<LPN>(k21);
        if (act && gl == 0) {
            const double cc = clamp_c(c);
            put(kv + 2 * ps, -(1.0 / a.dt), k12);
            put(kv + W + 2 * ps, 1.0 / (cc * (1.0 - cc)) - 2.0 * a.chi + k21, -1.0);
            a.rhs[2 * (size_t)i] = (c - cold) / a.dt + rcs;
            a.rhs[2 * (size_t)i + 1] = mu - (log(cc / (1.0 - cc)) + a.chi * (1.0 - 2.0 * cc)) + rms;
        }
    }
}

// ---- Poisson / diffusion (see assemble_scalar_kernel in k_csr.cu): one warp a node, one value a bond ---------------
// (U bonds of a lane in flight)
template <bool MIXED, int DIM, int U>
__global__ void __launch_bounds__(128) scalar_block_kernel(ScalarAsmArgs a, BlockPattern bp) {
    using GT = typename std::conditional<MIXED, float, double>::type;
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i >= a.n) return;
    // the node's own words are all asked for at once, before anything waits
    const int lo = a.rowptr[i], m = a.rowptr[i + 1] - lo, b0 = a.off[i], b1 = a.off[i + 1];
    const double ui = a.u[i];
    const int ps = bp.spos[i], px = bp.xpos[i];
    const bool dead = a.degenerate && a.degenerate[i];
    const double fi = a.f_node ? a.f_node[i] : a.f, uo = a.type == 0 ? 0.0 : a.uold[i];
    if (dead) {  // a singular moment system zeroes the row
        for (int k = lane; k < m; k += kWarp) a.kvals[lo + k] = 0.0;
        if (lane == 0) a.rhs[i] = 0.0;
        return;
    }
    const double coef = a.type == 0 ? a.coef : -a.coef;
    double rsum = 0.0, dsum = 0.0;
#pragma unroll U
    for (int t = b0 + lane; t < b1; t += kWarp) {
        const int j = __ldg(a.nbr + t);
        const GT *g = static_cast<const GT *>(a.ops) + (size_t)t * a.nop;
        double lap = (double)__ldg(g + a.s_xx) + (double)__ldg(g + a.s_yy);
        if constexpr (DIM == 3) lap += (double)__ldg(g + a.s_zz);
        const double co = coef * lap;
        rsum += co * (__ldg(a.u + j) - ui);
        dsum += co;
        a.kvals[lo + bp.bpos[t]] = -co;
    }
    // one exchange gives each half of the warp one of the two sums
    double tot = ((lane & 16) ? dsum : rsum) + __shfl_xor_sync(kFull, (lane & 16) ? rsum : dsum, 16);
    tot = group_sum<16>(tot);
    if (lane == 0) {
        double rn = fi;
        if (a.type != 0) rn = (ui - uo) / a.dt - fi;
        a.rhs[i] = rn + tot;
        if (px >= 0) a.kvals[lo + px] = 0.0;
    }
    if (lane == 16) a.kvals[lo + ps] = -(a.type == 0 ? 0.0 : 1.0 / a.dt) + tot;
}

// ---- launchers ------------------------------------------------------------------------------------------------
namespace {
// resident blocks: the grid is what the chip holds, at most one tile a block
template <int NT, typename El>
cudaError_t launch_nodes(const El &el, const BlockPattern &bp, int mmax, cudaStream_t s) {
    const size_t smem = sizeof(double) * (size_t)tile_doubles<El>(mmax);
    auto kernel = node_rows_kernel<El, NT>;
    // The limit belongs to the kernel, which contexts in other threads launch too: always the most that it may be launched
    // with, so that no call lowers what another has set.
    constexpr size_t most = sizeof(double) * (size_t)tile_doubles<El>(kBlockMax);
    static_assert(most <= 227 * 1024, "shared memory of a block");
    cudaError_t e = cudaSuccess;
    if (smem > 48 * 1024) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    int dev = 0, sms = 148, res = 1;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&res, kernel, NT, smem);
    if (e != cudaSuccess) return e;
    const long long need = ((long long)el.a.n + El::TN - 1) / El::TN, have = (long long)sms * (res > 0 ? res : 1);
    kernel<<<(int)(need < have ? need : have), NT, smem, s>>>(el, bp, mmax);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_stress_ch_block(const StressChAsmArgs &a, const BlockPattern &bp, int mmax, cudaStream_t s) {
    if (a.dim == 3) return launch_nodes<128>(StressChEl<3>{a}, bp, mmax, s);
    return launch_nodes<32>(StressChEl<2>{a}, bp, mmax, s);
}
cudaError_t launch_cached_block(const CachedAsmArgs &a, const BlockPattern &bp, int mmax, cudaStream_t s) {
    if (a.dim == 3) return launch_nodes<128>(CachedEl<3>{a}, bp, mmax, s);
    return launch_nodes<32>(CachedEl<2>{a}, bp, mmax, s);
}
cudaError_t launch_ch_block(const ChAsmArgs &a, const BlockPattern &bp, cudaStream_t s) {
    constexpr int LPN = 8;
    const long long g = ((long long)a.n + 256 / LPN - 1) / (256 / LPN);
    const int grid = (int)(g < 148 * 32 ? g : 148 * 32);
    if ((reinterpret_cast<uintptr_t>(a.kvals) & 15) == 0) ch_block_kernel<LPN, true><<<grid, 256, 0, s>>>(a, bp);
    else ch_block_kernel<LPN, false><<<grid, 256, 0, s>>>(a, bp);
    return cudaGetLastError();
}
template <bool MIXED, int DIM>
static cudaError_t launch_scalar(const ScalarAsmArgs &a, const BlockPattern &bp, cudaStream_t s) {
    const int g = (a.n + 3) / 4;
    // two bonds in flight where the blocks outnumber what the chip holds (16 an SM): 45,600 nodes in 3D FP64 78 -> 72 us,
    // 157,000 mixed 183 -> 150, 151,600 in 2D 68 -> 61; below that the second bond only lengthens the one wave (64x64: 4.1
    // us against 6.0)
    if (g > 148 * 16) scalar_block_kernel<MIXED, DIM, 2><<<g, 128, 0, s>>>(a, bp);
    else scalar_block_kernel<MIXED, DIM, 1><<<g, 128, 0, s>>>(a, bp);
    return cudaGetLastError();
}

cudaError_t launch_scalar_block(const ScalarAsmArgs &a, const BlockPattern &bp, cudaStream_t s) {
    if (a.dim == 3) return a.mixed ? launch_scalar<true, 3>(a, bp, s) : launch_scalar<false, 3>(a, bp, s);
    return a.mixed ? launch_scalar<true, 2>(a, bp, s) : launch_scalar<false, 2>(a, bp, s);
}

}  // namespace pxb
