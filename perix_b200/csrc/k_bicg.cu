// Device-resident BiCGStab for the 2-dof systems of the implicit Cahn-Hilliard run (ch_solver.cpp).
//
// Right-preconditioned BiCGStab (van der Vorst 1992) with the 2x2 block-Jacobi inverse M (rows 2i, 2i+1 of a node),
// run as ONE cooperative persistent kernel per solve: every block takes part in every phase and the phases are
// separated by grid barriers, so the matrix (61 MB of values at 256^2) and the work vectors stay in L2 across the
// iterations and no scalar goes back to the host.  Each dot product is a per-block partial sum followed by a barrier,
// after which every block adds the partials in the same fixed order, so all blocks take the same decisions and the
// result is deterministic.  The partial sums alternate between two buffers, so a block that runs ahead into the next
// reduction never overwrites partials another block is still reading.
//
// The iteration keeps rh = M r and vh = M v per node, so both preconditioned vectors are formed where the products
// gather them (ph_j = rh_j + beta (ph_j - omega vh_j), sh_j = rh_j - alpha vh_j) and an iteration needs three
// barriers (x0 = 0, r = r0 = b, rh = M b, ph = vh = 0, rho = alpha = omega = 1, rho1 = r0.r):
//   A  ph' = rh + beta (ph - omega vh),  v = A ph',  vh' = M v,  r0.v         | barrier   alpha = rho1 / r0.v
//   B  s = r - alpha v,  sh = rh - alpha vh',  t = A sh,  t.t, t.s, s.s        | barrier   omega = t.s / t.t
//      |s| <= tol |b|: x += alpha ph', done
//   C  x += alpha ph' + omega sh,  r = s - omega t,  rh = M r,  r.r, r0.r     | barrier   |r| <= tol |b|: done
//      rho = rho1, rho1 = r0.r, beta = (rho1 / rho)(alpha / omega)
// ph and vh are double-buffered: phase A reads one copy while it writes the other.  The gathered and the stored
// values come from one helper with explicit rounding, so both are bitwise the same.
// The matrix must consist of dense 2x2 node blocks (rows 2i and 2i+1 share one column list of pairs (2j, 2j+1), as
// every pattern the reference builds does, SparseMatrix.cpp:73-185).  The product reads it through a block view: bptr
// (node -> first block) and bcol (block -> column node), with the CSR values of node i's two rows at 4 bptr[i] and
// 4 bptr[i] + 2 nblk_i.  Adjoint solves run the same kernel on an explicit transpose (block_transpose below and a
// value gather).
//
// The implicit run's own systems, whose blocks are known to be anti-diagonal, have the sliced form further down.
//
// The grid barrier waits are bounded: a block that waits longer than kSpinLimit polls sets the abort word and
// returns, and every other block leaves at its next barrier; the host reports the timeout.  The cooperative launch
// makes every block resident at once, so the waits end in normal operation.
#include <vector>

#include "k_kernels.h"
#include "pxb_common.cuh"

namespace pxb {

namespace {

constexpr int kThreads = 256;
constexpr int kBlocksPerSM = 3;  // 80 registers a thread
constexpr int kWarps = kThreads / kWarp;
constexpr int kMaxGrid = 512;  // most blocks of the solve kernel
static_assert(kMaxGrid <= kBicgParts && kMaxGrid % kWarp == 0, "partial sum slots");
constexpr int kSpmvLanes = 8;  // lanes per node (its two rows)
constexpr int kUnroll = 2;     // blocks per lane and pass
constexpr int kSliceThreads = 512, kSliceBlocks = 1;  // sliced solve: 128 registers a thread
constexpr int kSliceMaxGrid = 160;
constexpr int kSliceUnroll = 4, kSliceUnroll1 = 6;     // its blocks per lane and pass (one lane a node)
constexpr unsigned kSpinLimit = 1u << 22;  // barrier polls (a few seconds at most)

// Vector loads are ordinary (L1-cached) loads: within a phase no vector is both written and read by different
// threads, and the fences of the grid barrier order every write of one phase before the reads of the next.
__device__ __forceinline__ double2 ld2(const double *p, int i) { return reinterpret_cast<const double2 *>(p)[i]; }
__device__ __forceinline__ void st2(double *p, int i, double a, double b) {
    reinterpret_cast<double2 *>(p)[i] = make_double2(a, b);
}
__device__ __forceinline__ void block2(const double *binv, int i, double x0, double x1, double &y0, double &y1) {
    const double2 b0 = __ldg(reinterpret_cast<const double2 *>(binv) + 2 * i);
    const double2 b1 = __ldg(reinterpret_cast<const double2 *>(binv) + 2 * i + 1);
    y0 = b0.x * x0 + b0.y * x1;
    y1 = b1.x * x0 + b1.y * x1;
}

// Grid barrier on a monotonic arrival counter: barrier number e (1, 2, ...) ends when e * gridDim.x blocks have
// arrived.  Returns false when the wait gave up or another block aborted.
__device__ bool grid_sync(BicgScalars *sc, unsigned int &epoch) {
    __shared__ int ok;
    __syncthreads();
    ++epoch;
    if (threadIdx.x == 0) {
        const unsigned int target = epoch * gridDim.x;
        volatile unsigned int *count = &sc->bar_count;
        volatile int *abort = &sc->abort;
        __threadfence();
        atomicAdd(&sc->bar_count, 1u);
        int good = 1;
        unsigned int polls = 0;
        while ((int)(*count - target) < 0) {
            if (*abort || ++polls > kSpinLimit) {
                *abort = 1;
                good = 0;
                break;
            }
            __nanosleep(32);
        }
        __threadfence();
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// Grid totals of NV per-thread values: block sums into part, a barrier, then every block adds the partials in the
// same order.  Every thread receives the totals.
template <int NV>
__device__ bool grid_total(const double (&val)[NV], double *part, BicgScalars *sc, unsigned int &epoch,
                           double (&tot)[NV]) {
    static_assert(NV <= kWarps, "one warp per total");
    __shared__ double sh[NV][kWarp];
    __shared__ double res[NV];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const double s = group_sum<kWarp>(val[q]);
        if (lane == 0) sh[q][w] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double t = 0.0;
            for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sh[q][k];
            part[q * kBicgParts + blockIdx.x] = t;
        }
    if (!grid_sync(sc, epoch)) return false;
    if (w < NV) {  // warp q adds the partials of value q, all loads in flight at once
        constexpr int M = kMaxGrid / kWarp;
        double v[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int k = lane + kWarp * m;
            v[m] = k < (int)gridDim.x ? __ldcg(part + w * kBicgParts + k) : 0.0;
        }
        double s = 0.0;
#pragma unroll
        for (int m = 0; m < M; ++m) s += v[m];
        s = group_sum<kWarp>(s);
        if (lane == 0) res[w] = s;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) tot[q] = res[q];
    __syncthreads();
    return true;
}

// the preconditioned vectors of phases A and B, with explicit rounding (gathered and stored copies agree bitwise)
__device__ __forceinline__ double2 new_ph(double2 rh, double2 ph, double2 vh, double beta, double omega) {
    return make_double2(__fma_rn(beta, __fma_rn(-omega, vh.x, ph.x), rh.x),
                        __fma_rn(beta, __fma_rn(-omega, vh.y, ph.y), rh.y));
}
__device__ __forceinline__ double2 new_sh(double2 rh, double2 vh, double alpha) {
    return make_double2(__fma_rn(-alpha, vh.x, rh.x), __fma_rn(-alpha, vh.y, rh.y));
}

struct Scal {
    double alpha, beta, omega;
};

// node i's vector work after its product (y0, y1) with x, and its share of the phase's dot products
template <int STAGE>
__device__ __forceinline__ void node_work(const BicgArgs &a, const Scal &c, int i, double2 x, double y0, double y1,
                                          double *vhn, double *phn, double (&d)[3]) {
    if (STAGE == 0) {
        st2(phn, i, x.x, x.y);
        st2(a.v, i, y0, y1);
        double h0, h1;
        block2(a.binv, i, y0, y1, h0, h1);
        st2(vhn, i, h0, h1);
        const double2 r0 = ld2(a.r0, i);
        d[0] += r0.x * y0 + r0.y * y1;
    } else {
        const double2 r = ld2(a.r, i), v = ld2(a.v, i);
        const double s0 = r.x - c.alpha * v.x, s1 = r.y - c.alpha * v.y;
        st2(a.s, i, s0, s1);
        st2(a.sh, i, x.x, x.y);
        st2(a.t, i, y0, y1);
        d[0] += y0 * y0 + y1 * y1;
        d[1] += y0 * s0 + y1 * s1;
        d[2] += s0 * s0 + s1 * s1;
    }
}

// Phase A (STAGE 0) or B (STAGE 1) over node blocks: the product of A with the preconditioned vector formed at the
// gather, each lane keeping up to kUnroll blocks in flight; the group leader of node i then does node i's vector work
// and accumulates its share of the phase's dot products into d[].
template <int STAGE>
__device__ void product_phase(const BicgArgs &a, const Scal &c, const double *pho, const double *vho, double *phn,
                              double *vhn, double (&d)[3]) {
    constexpr int G = kSpmvLanes, GPW = kWarp / G, U = kUnroll;
    const int lane = threadIdx.x & 31, gl = lane % G;
    const int warp = (blockIdx.x * kThreads + threadIdx.x) >> 5, nwarps = (gridDim.x * kThreads) >> 5;
    for (int base = warp * GPW; base < a.n; base += nwarps * GPW) {
        const int i = base + lane / G;
        double y0 = 0.0, y1 = 0.0;
        if (i < a.n) {
            const int b0 = __ldg(a.bptr + i), nblk = __ldg(a.bptr + i + 1) - b0;
            const double2 *v0 = reinterpret_cast<const double2 *>(a.val + 4 * (size_t)b0), *v1 = v0 + nblk;
            for (int b = gl; b < nblk; b += U * G) {
                int j[U];
                double2 e0[U], e1[U];
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    const int bb = b + q * G;
                    j[q] = bb < nblk ? __ldg(a.bcol + b0 + bb) : -1;
                    if (bb < nblk) {
                        e0[q] = __ldg(v0 + bb);
                        e1[q] = __ldg(v1 + bb);
                    }
                }
#pragma unroll
                for (int q = 0; q < U; ++q)
                    if (j[q] >= 0) {
                        const double2 xj = STAGE == 0
                                               ? new_ph(ld2(a.rh, j[q]), ld2(pho, j[q]), ld2(vho, j[q]), c.beta, c.omega)
                                               : new_sh(ld2(a.rh, j[q]), ld2(vhn, j[q]), c.alpha);
                        y0 += e0[q].x * xj.x + e0[q].y * xj.y;
                        y1 += e1[q].x * xj.x + e1[q].y * xj.y;
                    }
            }
        }
        y0 = group_sum<G>(y0);
        y1 = group_sum<G>(y1);
        if (i < a.n && gl == 0) {
            node_work<STAGE>(a, c, i,
                             STAGE == 0 ? new_ph(ld2(a.rh, i), ld2(pho, i), ld2(vho, i), c.beta, c.omega)
                                        : new_sh(ld2(a.rh, i), ld2(vhn, i), c.alpha),
                             y0, y1, vhn, phn, d);
        }
    }
}

__device__ __forceinline__ void finish(BicgScalars *sc, int status, int its, double relres) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->status = status;
        sc->its = its;
        sc->relres = relres;
    }
}

__global__ void __launch_bounds__(kThreads, kBlocksPerSM) bicg_solve_kernel(BicgArgs a, double tol, int max_its) {
    BicgScalars *sc = a.sc;
    unsigned int epoch = 0;
    int set = 0;
    auto part = [&]() {
        double *p = a.part + (size_t)set * 3 * kBicgParts;
        set ^= 1;
        return p;
    };
    const int tid = blockIdx.x * kThreads + threadIdx.x, nth = gridDim.x * kThreads;
    double bb = 0.0;
    for (int i = tid; i < a.n; i += nth) {
        const double2 b = ld2(a.b, i);
        st2(a.x, i, 0.0, 0.0);
        st2(a.r, i, b.x, b.y);
        st2(a.r0, i, b.x, b.y);
        double h0, h1;
        block2(a.binv, i, b.x, b.y, h0, h1);
        st2(a.rh, i, h0, h1);
        st2(a.ph[0], i, 0.0, 0.0);
        st2(a.vh[0], i, 0.0, 0.0);
        bb += b.x * b.x + b.y * b.y;
    }
    double t1[1], t3[3];
    if (!grid_total<1>({bb}, part(), sc, epoch, t1)) return;
    const double bnorm = sqrt(t1[0]);
    if (!(bnorm > 0.0)) return finish(sc, kBicgDone, 0, 0.0);
    double rho = 1.0, rho1 = t1[0];
    Scal c{1.0, t1[0], 1.0};
    for (int k = 1;; ++k) {
        const double *pho = a.ph[(k - 1) & 1], *vho = a.vh[(k - 1) & 1];
        double *phn = a.ph[k & 1], *vhn = a.vh[k & 1];
        double d[3] = {0.0, 0.0, 0.0};
        product_phase<0>(a, c, pho, vho, phn, vhn, d);
        if (!grid_total<1>({d[0]}, part(), sc, epoch, t1)) return;
        if (t1[0] == 0.0 || !isfinite(t1[0])) return finish(sc, kBicgBreakdown, k - 1, 0.0);
        c.alpha = rho1 / t1[0];
        d[0] = d[1] = d[2] = 0.0;
        product_phase<1>(a, c, pho, vho, phn, vhn, d);
        if (!grid_total<3>({d[0], d[1], d[2]}, part(), sc, epoch, t3)) return;
        const double sn = sqrt(t3[2]);
        if (sn <= tol * bnorm) {
            for (int i = tid; i < a.n; i += nth) {
                const double2 x = ld2(a.x, i), ph = ld2(phn, i);
                st2(a.x, i, x.x + c.alpha * ph.x, x.y + c.alpha * ph.y);
            }
            return finish(sc, kBicgDone, k, sn / bnorm);
        }
        c.omega = t3[0] > 0.0 ? t3[1] / t3[0] : 0.0;
        double rr = 0.0, r0r = 0.0;
        for (int i = tid; i < a.n; i += nth) {
            const double2 x = ld2(a.x, i), ph = ld2(phn, i), sh = ld2(a.sh, i), s = ld2(a.s, i), t = ld2(a.t, i);
            const double2 r0 = ld2(a.r0, i);
            st2(a.x, i, (x.x + c.alpha * ph.x) + c.omega * sh.x, (x.y + c.alpha * ph.y) + c.omega * sh.y);
            const double q0 = s.x - c.omega * t.x, q1 = s.y - c.omega * t.y;
            st2(a.r, i, q0, q1);
            double h0, h1;
            block2(a.binv, i, q0, q1, h0, h1);
            st2(a.rh, i, h0, h1);
            rr += q0 * q0 + q1 * q1;
            r0r += r0.x * q0 + r0.y * q1;
        }
        if (!grid_total<3>({rr, r0r, 0.0}, part(), sc, epoch, t3)) return;
        const double relres = sqrt(t3[0]) / bnorm;
        if (relres <= tol) return finish(sc, kBicgDone, k, relres);
        if (k >= max_its) return finish(sc, kBicgMaxIts, k, relres);
        rho = rho1;
        rho1 = t3[1];
        if (rho1 == 0.0 || !isfinite(rho1) || c.omega == 0.0) return finish(sc, kBicgBreakdown, k, relres);
        c.beta = (rho1 / rho) * (c.alpha / c.omega);
    }
}

// ---- the Newton system on slices (exact block patterns) --------------------------------------------------------------
// Every block of the system but a node's own is anti-diagonal (row c couples to mu_j, row mu to c_j), and a ghost
// node's rows hold its own diagonal and the mirror's.  So a block is one pair of values instead of four, and the rows of
// 32 consecutive nodes are stored block by block (slice: value pair and column of node 32 s + l, block k at
// 32 (row0[s] + k) + l), which a product reads without reductions over a lane group and with neighbouring nodes'
// gathers side by side.  20 bytes a block instead of 36.
// What bounds a solve at 256x256 is not the matrix (39 MB, in L2: holding two thirds of it in shared memory changed
// nothing) but the L1 data pipe under the gathers and the grid barriers, about 3800 cycles each.  So 148 blocks of 512
// threads (two of 512: 10.0 ms a run, one of 1024: 10.1, one of 512: 9.2), the preconditioned direction's
// ph - omega vh formed once a node in phase C instead of at every gather, and the Newton iteration's other sums and its
// update in the same kernel.  256x256, 10 steps (32 solves, 298 iterations): 18.4 ms with the CSR kernels -> 9.7 ms, and
// 8.1 ms with the next iteration queued ahead and the barrier's counter on the faster page (ch_solver.cpp);
// 64x64: 10.8 (one lane a node) -> 5.9 ms with eight.

// K (Picard Jacobian, Neumann ghost rows) and F at (U, Uold): value pairs, block-Jacobi inverse, right-hand side.  The
// entries are those of ch_block_kernel and ch_ghost_rows_kernel; also clears the solver's scalars.
constexpr int kSystemLanes = 4, kSystemUnroll = 2;  // 8 lanes: 3 % more of a 256x256 run
__device__ __forceinline__ double mobility(double M0, double c) {
    const double cc = fmax(1.0e-8, fmin(1.0 - 1.0e-8, c));
    return M0 * cc * (1.0 - cc);
}

__global__ void __launch_bounds__(256) ch_system_kernel(ChSystemArgs a) {
    constexpr int LPN = kSystemLanes, GPW = kWarp / LPN, U = kSystemUnroll;
    if (a.prev && !a.prev->go) return;
    if (blockIdx.x == 0 && threadIdx.x < sizeof(BicgScalars) / 4) reinterpret_cast<int *>(a.sc)[threadIdx.x] = 0;
    const int lane = threadIdx.x & 31, gl = lane & (LPN - 1);
    const int i = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * GPW + lane / LPN;
    const int m = i < a.n && a.mirror ? a.mirror[i] : 0;
    const double2 *U2 = reinterpret_cast<const double2 *>(a.u);
    const bool bulk = i < a.n && m <= 0;
    const int b0 = bulk ? a.off[i] : 0, b1 = bulk ? a.off[i + 1] : 0;
    const double2 ui = i < a.n ? U2[i] : make_double2(0.5, 0.0);
    const double Vi = bulk ? a.vol[i] : 1.0, iV = 1.0 / Vi, Mi = mobility(a.M0, ui.x);
    double2 *pair = a.pair + ((size_t)(bulk ? a.row0[i >> 5] : 0) * kWarp + (i & 31));
    double rcs = 0.0, rms = 0.0, k12 = 0.0, k21 = 0.0;
    for (int t = b0 + gl; t < b1; t += U * LPN) {
        int j[U], pos[U], f[U];
        double g2[U], lr[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {  // past the family: a bond to the node itself that counts for nothing
            const int tt = t + q * LPN;
            const bool in = tt < b1;
            j[q] = in ? __ldg(a.nbr + tt) : i;
            g2[q] = in ? __ldg(a.lap + tt) : 0.0;
            lr[q] = in ? __ldg(a.lrv + tt) : 0.0;
            f[q] = in ? __ldg(a.bfl + tt) : 1;
            pos[q] = in ? __ldg(a.bpos + tt) : -1;
        }
        double2 uj[U];
#pragma unroll
        for (int q = 0; q < U; ++q) uj[q] = U2[j[q]];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            double kc = 0.0, km = 0.0;
            if (!(f[q] & 1)) {
                kc = (f[q] & 2) && Vi > 0.0 ? species_flux(Mi, g2[q], lr[q], iV, mobility(a.M0, uj[q].x)) : -(Mi * g2[q]);
                km = a.kappa * g2[q];
            }
            rcs += kc * (uj[q].y - ui.y);
            rms += km * (uj[q].x - ui.x);
            k12 += kc;
            k21 += km;
            if (pos[q] >= 0) pair[(size_t)pos[q] * kWarp] = make_double2(-kc, -km);
        }
    }
    rcs = group_sum<LPN>(rcs);
    rms = group_sum<LPN>(rms);
    k12 = group_sum<LPN>(k12);
    k21 = group_sum<LPN>(k21);
    if (i >= a.n || gl != 0) return;
    double d0, d1, o12 = 0.0, o21 = 0.0;
    double2 f;
    if (bulk) {
        const double cc = fmax(1.0e-8, fmin(1.0 - 1.0e-8, ui.x));
        d0 = -(1.0 / a.dt);
        d1 = -1.0;
        o12 = k12;
        o21 = 1.0 / (cc * (1.0 - cc)) - 2.0 * a.chi + k21;
        pair[(size_t)a.spos[i] * kWarp] = make_double2(o12, o21);
        f.x = (ui.x - a.uold[2 * (size_t)i]) / a.dt + rcs;
        f.y = ui.y - (log(cc / (1.0 - cc)) + a.chi * (1.0 - 2.0 * cc)) + rms;
    } else {
        const double2 ub = U2[m - 1];
        d0 = ghost_scale(a.dt);
        d1 = 1.0;
        f.x = d0 * (ub.x - ui.x);
        f.y = d1 * (ub.y - ui.y);
    }
    reinterpret_cast<double2 *>(a.rhs)[i] = f;
    const double det = d0 * d1 - o12 * o21;
    const bool good = det != 0.0 && isfinite(det);
    double2 *o = reinterpret_cast<double2 *>(a.binv) + 2 * (size_t)i;
    o[0] = good ? make_double2(d1 / det, -o12 / det) : make_double2(1.0, 0.0);
    o[1] = good ? make_double2(-o21 / det, d0 / det) : make_double2(0.0, 1.0);
}

// columns (a short row's tail points at its own node) and zeroed pairs (ghost rows and tails stay zero)
__global__ void __launch_bounds__(256) ch_slices_fill_kernel(ChSlices a) {
    const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (s * kWarp >= a.n) return;
    const int i = s * kWarp + lane, w0 = a.row0[s], w1 = a.row0[s + 1];
    const bool bulk = i < a.n && !(a.mirror && a.mirror[i] > 0);
    const int b0 = bulk ? a.bptr[i] : 0, len = bulk ? a.bptr[i + 1] - b0 : 0;
    for (int k = 0; k < w1 - w0; ++k) {
        const size_t q = (size_t)(w0 + k) * kWarp + lane;
        a.col[q] = k < len ? a.bcol[b0 + k] : (i < a.n ? i : a.n - 1);
        a.pair[q] = make_double2(0.0, 0.0);
    }
}

// Phase A (STAGE 0) or B (STAGE 1) on the slices: LPN lanes a node, a warp = 32 / LPN nodes (a unit), block k of a row
// with lane group k mod LPN; otherwise as product_phase.
template <int STAGE, int LPN>
__device__ __forceinline__ void slices_phase(const BicgArgs &a, const ChSlices &m, const Scal &c, double *phn,
                                             double *vhn, double (&d)[3]) {
    constexpr int NPW = kWarp / LPN, U = LPN == 1 ? kSliceUnroll1 : kSliceUnroll;
    const int lane = threadIdx.x & 31, h = lane / NPW;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const int units = (a.n + NPW - 1) / NPW;
    auto vec = [&](int j) {
        const double2 rh = ld2(a.rh, j);
        if (STAGE == 0) {
            const double2 q = ld2(a.sh, j);  // ph - omega vh (phase C)
            return make_double2(__fma_rn(c.beta, q.x, rh.x), __fma_rn(c.beta, q.y, rh.y));
        }
        return new_sh(rh, ld2(vhn, j), c.alpha);
    };
    for (int u = warp; u < units; u += nwarps) {
        const int i = u * NPW + lane % NPW, s = u / LPN;
        const int w0 = __ldg(m.row0 + s), w = __ldg(m.row0 + s + 1) - w0;
        const double2 *pr = m.pair + ((size_t)(w0 + h) * kWarp + (i & 31));
        const int *cl = m.col + ((size_t)(w0 + h) * kWarp + (i & 31));
        double y0 = 0.0, y1 = 0.0;
        for (int k = 0; k * LPN < w; k += U) {
            double2 e[U];
            int j[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const bool in = (k + q) * LPN + h < w;
                j[q] = in ? __ldg(cl + (size_t)(k + q) * (LPN * kWarp)) : 0;
                e[q] = in ? __ldg(pr + (size_t)(k + q) * (LPN * kWarp)) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int q = 0; q < U; ++q)
                if ((k + q) * LPN < w) {
                    const double2 x = vec(j[q]);
                    y0 = fma(e[q].x, x.y, y0);
                    y1 = fma(e[q].y, x.x, y1);
                }
        }
#pragma unroll
        for (int o = NPW; o < kWarp; o <<= 1) {
            y0 += __shfl_xor_sync(kFull, y0, o);
            y1 += __shfl_xor_sync(kFull, y1, o);
        }
        if (h == 0 && i < a.n) {
            const int b = m.mirror ? __ldg(m.mirror + i) : 0;
            const double2 xi = vec(i);
            if (b <= 0) {
                y0 = fma(m.d0, xi.x, y0);
                y1 = fma(m.d1, xi.y, y1);
            } else {
                const double2 xb = b - 1 == i ? make_double2(0.0, 0.0) : vec(b - 1);
                y0 = m.g0 * xi.x - m.g0 * xb.x;
                y1 = m.g1 * xi.y - m.g1 * xb.y;
            }
            node_work<STAGE>(a, c, i, xi, y0, y1, vhn, phn, d);
        }
    }
}

// grid_total for the sliced solve's few, wide blocks: the warps' sums and the blocks' sums are added by shuffles.  With
// chains of additions a barrier took 4400 cycles at best, now 3800, the grid's three round trips to L2.  (A word that
// carries both the sum and the arrival, polled by every block, saves a trip but took 5500: the polls get in each
// other's way.)
template <int NV>
__device__ bool grid_sum(const double (&val)[NV], double *part, BicgScalars *sc, unsigned int &epoch, double (&tot)[NV]) {
    constexpr int W = kSliceThreads / kWarp, M = kSliceMaxGrid / kWarp;
    __shared__ double sh[NV][W];
    __shared__ double res[NV];
    __shared__ int ok;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    part += (size_t)(++epoch & 1) * 3 * kBicgParts;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const double s = group_sum<kWarp>(val[q]);
        if (lane == 0) sh[q][w] = s;
    }
    __syncthreads();
    if (w == 0) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const double t = group_sum<W>(sh[q][lane & (W - 1)]);
            if (lane == q) s = t;
        }
        if (lane < NV) __stcg(part + lane * kBicgParts + blockIdx.x, s);
        __threadfence();
        __syncwarp();
        if (lane == 0) {
            const unsigned int target = epoch * gridDim.x;
            volatile unsigned int *count = &sc->bar_count;
            volatile int *abort = &sc->abort;
            atomicAdd(&sc->bar_count, 1u);
            int good = 1;
            unsigned int polls = 0;
            while ((int)(*count - target) < 0)
                if (++polls > kSpinLimit || ((polls & 63) == 0 && *abort)) {
                    *abort = 1;
                    good = 0;
                    break;
                }
            ok = good;
            __threadfence();
        }
        __syncwarp();
        if (ok != 0) {
            double v[NV][M];
#pragma unroll
            for (int q = 0; q < NV; ++q)
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const int k = lane + kWarp * m;
                    v[q][m] = k < (int)gridDim.x ? __ldcg(part + q * kBicgParts + k) : 0.0;
                }
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                double t = 0.0;
#pragma unroll
                for (int m = 0; m < M; ++m) t += v[q][m];
                t = group_sum<kWarp>(t);
                if (lane == 0) res[q] = t;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) tot[q] = res[q];
    return ok != 0;
}

// One Newton iteration's solve: |F| against the stop value, BiCGStab as bicg_solve_kernel (phases A, B, C there), then
// the update U += x with the dot products x.x and U.U (before it) that the iteration's end needs.
template <int LPN>
__global__ void __launch_bounds__(kSliceThreads, kSliceBlocks) ch_newton_kernel(BicgArgs a, ChSlices m, ChNewton nw) {
    BicgScalars *sc = a.sc;
    if (nw.prev && !nw.prev->go) return;
    unsigned int epoch = 0;
    const int tid = blockIdx.x * kSliceThreads + threadIdx.x, nth = gridDim.x * kSliceThreads;
    double bb = 0.0;
    for (int i = tid; i < a.n; i += nth) {
        const double2 b = ld2(a.b, i);
        st2(a.x, i, 0.0, 0.0);
        st2(a.r, i, b.x, b.y);
        double h0, h1;
        block2(a.binv, i, b.x, b.y, h0, h1);
        st2(a.rh, i, h0, h1);
        st2(a.sh, i, 0.0, 0.0);
        bb += b.x * b.x + b.y * b.y;
    }
    double t1[1], t2[2], t3[3];
    if (!grid_sum<1>({bb}, a.part, sc, epoch, t1)) return;
    const double bnorm = sqrt(t1[0]);
    const double res0 = nw.prev ? nw.prev->res0 : bnorm;
    auto finish = [&](int status, int its, double rel, double dd, double uu, bool go) {
        if (tid != 0) return;
        BicgScalars *h = nw.host;
        h->bnorm = bnorm;
        h->dd = dd;
        h->uu = uu;
        h->relres = rel;
        h->its = its;
        h->go = go ? 1 : 0;
        h->status = status;
        sc->res0 = res0;
        sc->go = go ? 1 : 0;
    };
    if (!(bnorm > (nw.prev ? nw.rtol * res0 : 0.0)) || !isfinite(bnorm) || nw.only_norm)
        return finish(kBicgDone, 0, 0.0, 0.0, 0.0, false);
    double rho = 1.0, rho1 = t1[0], relres = 0.0;
    Scal c{1.0, t1[0], 1.0};
    int k = 1;
    bool half = false;  // left after phase B
    for (;; ++k) {
        double *phn = a.ph[0], *vhn = a.vh[0];
        double d[3] = {0.0, 0.0, 0.0};
        slices_phase<0, LPN>(a, m, c, phn, vhn, d);
        if (!grid_sum<1>({d[0]}, a.part, sc, epoch, t1)) return;
        if (t1[0] == 0.0 || !isfinite(t1[0])) return finish(kBicgBreakdown, k - 1, 0.0, 0.0, 0.0, false);
        c.alpha = rho1 / t1[0];
        d[0] = d[1] = d[2] = 0.0;
        slices_phase<1, LPN>(a, m, c, phn, vhn, d);
        if (!grid_sum<3>({d[0], d[1], d[2]}, a.part, sc, epoch, t3)) return;
        const double sn = sqrt(t3[2]);
        if (sn <= nw.tol * bnorm) {
            relres = sn / bnorm;
            half = true;
            break;
        }
        c.omega = t3[0] > 0.0 ? t3[1] / t3[0] : 0.0;
        double rr = 0.0, r0r = 0.0;
        for (int i = tid; i < a.n; i += nth) {
            const double2 x = ld2(a.x, i), ph = ld2(phn, i), sh = ld2(a.sh, i), s = ld2(a.s, i), t = ld2(a.t, i);
            const double2 r0 = ld2(a.b, i), vh = ld2(vhn, i);
            st2(a.sh, i, __fma_rn(-c.omega, vh.x, ph.x), __fma_rn(-c.omega, vh.y, ph.y));
            st2(a.x, i, (x.x + c.alpha * ph.x) + c.omega * sh.x, (x.y + c.alpha * ph.y) + c.omega * sh.y);
            const double q0 = s.x - c.omega * t.x, q1 = s.y - c.omega * t.y;
            st2(a.r, i, q0, q1);
            double h0, h1;
            block2(a.binv, i, q0, q1, h0, h1);
            st2(a.rh, i, h0, h1);
            rr += q0 * q0 + q1 * q1;
            r0r += r0.x * q0 + r0.y * q1;
        }
        if (!grid_sum<2>({rr, r0r}, a.part, sc, epoch, t2)) return;
        relres = sqrt(t2[0]) / bnorm;
        if (relres <= nw.tol) break;
        if (k >= nw.max_its) return finish(kBicgMaxIts, k, relres, 0.0, 0.0, false);
        rho = rho1;
        rho1 = t2[1];
        if (rho1 == 0.0 || !isfinite(rho1) || c.omega == 0.0) return finish(kBicgBreakdown, k, relres, 0.0, 0.0, false);
        c.beta = (rho1 / rho) * (c.alpha / c.omega);
    }
    double dd = 0.0, uu = 0.0;
    for (int i = tid; i < a.n; i += nth) {
        double2 x = ld2(a.x, i);
        if (half) {
            const double2 ph = ld2(a.ph[0], i);
            x = make_double2(x.x + c.alpha * ph.x, x.y + c.alpha * ph.y);
            st2(a.x, i, x.x, x.y);
        }
        const double2 u = ld2(nw.u, i);
        st2(nw.u, i, x.x + u.x, x.y + u.y);
        dd += x.x * x.x + x.y * x.y;
        uu += u.x * u.x + u.y * u.y;
    }
    if (!grid_sum<2>({dd, uu}, a.part, sc, epoch, t2)) return;
    // an update at the rounding level of the state ends the step (the residual of a small step can sit at its
    // evaluation floor, far above rtol times its initial value)
    finish(kBicgDone, k, relres, t2[0], t2[1], !(sqrt(t2[0]) <= nw.update_tol * sqrt(t2[1])));
}

// vt[q] = v[perm[q]]: the values of the transposed matrix
__global__ void gather_values_kernel(long long nnz, const int *perm, const double *v, double *vt) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nnz; q += (long long)gridDim.x * blockDim.x)
        vt[q] = v[__ldg(perm + q)];
}

}  // namespace

bool block_view(int n, const int *rowptr, const int *cols, std::vector<int> &bptr, std::vector<int> &bcol) {
    bptr.assign((size_t)n + 1, 0);
    bcol.clear();
    bcol.reserve((size_t)(rowptr[2 * (size_t)n] / 4));
    for (int i = 0; i < n; ++i) {
        const int lo0 = rowptr[2 * i], lo1 = rowptr[2 * i + 1], hi1 = rowptr[2 * i + 2];
        const int len = lo1 - lo0;
        if (len != hi1 - lo1 || (len & 1) || lo0 != 4 * (int)bcol.size()) return false;
        for (int k = 0; k < len; k += 2) {
            const int c = cols[lo0 + k];
            if ((c & 1) || cols[lo0 + k + 1] != c + 1 || cols[lo1 + k] != c || cols[lo1 + k + 1] != c + 1) return false;
            bcol.push_back(c >> 1);
        }
        bptr[(size_t)i + 1] = (int)bcol.size();
    }
    return true;
}

void block_transpose(int n, const std::vector<int> &bptr, const std::vector<int> &bcol, std::vector<int> &tbptr,
                     std::vector<int> &tbcol, std::vector<int> &perm) {
    const size_t nblk = bcol.size();
    tbptr.assign((size_t)n + 1, 0);
    for (int j : bcol) tbptr[(size_t)j + 1]++;
    for (int j = 0; j < n; ++j) tbptr[(size_t)j + 1] += tbptr[(size_t)j];
    tbcol.assign(nblk, 0);
    std::vector<int> fill(tbptr.begin(), tbptr.end() - 1), pos(nblk);
    for (int i = 0; i < n; ++i)  // rows in ascending order: each transposed row's columns come out sorted
        for (int p = bptr[(size_t)i]; p < bptr[(size_t)i + 1]; ++p) {
            const int q = fill[(size_t)bcol[(size_t)p]]++;
            tbcol[(size_t)q] = i;
            pos[(size_t)p] = q;
        }
    // entry (2j+a, 2i+b) of the transpose is entry (2i+b, 2j+a) of the matrix
    perm.assign(4 * nblk, 0);
    for (int i = 0; i < n; ++i) {
        const int b0 = bptr[(size_t)i], ni = bptr[(size_t)i + 1] - b0;
        for (int p = 0; p < ni; ++p) {
            const int q = pos[(size_t)(b0 + p)], j = bcol[(size_t)(b0 + p)];
            const int t0 = tbptr[(size_t)j], nj = tbptr[(size_t)j + 1] - t0, qq = q - t0;
            for (int ra = 0; ra < 2; ++ra)
                for (int rb = 0; rb < 2; ++rb)
                    perm[4 * (size_t)t0 + (size_t)ra * 2 * nj + 2 * (size_t)qq + rb] =
                        4 * b0 + rb * 2 * ni + 2 * p + ra;
        }
    }
}

cudaError_t launch_gather_values(long long nnz, const int *perm, const double *v, double *vt, cudaStream_t s) {
    const long long g = (nnz + 255) / 256;
    gather_values_kernel<<<(int)(g < 148 * 16 ? (g > 0 ? g : 1) : 148 * 16), 256, 0, s>>>(nnz, perm, v, vt);
    return cudaGetLastError();
}

cudaError_t launch_ch_slices_fill(const ChSlices &a, cudaStream_t s) {
    const int g = (a.n + 255) / 256;
    ch_slices_fill_kernel<<<g > 0 ? g : 1, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_ch_system(const ChSystemArgs &a, cudaStream_t s) {
    constexpr int npb = 256 / kSystemLanes;
    ch_system_kernel<<<(a.n + npb - 1) / npb, 256, 0, s>>>(a);
    return cudaGetLastError();
}

template <int LPN>
static cudaError_t launch_newton(BicgArgs &a, ChSlices &m, ChNewton &nw, int grid, cudaStream_t s) {
    void *params[] = {&a, &m, &nw};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(ch_newton_kernel<LPN>), dim3(grid),
                                       dim3(kSliceThreads), params, 0, s);
}

cudaError_t launch_ch_newton(const BicgArgs &args, const ChSlices &slices, const ChNewton &newton, cudaStream_t s) {
    BicgArgs a = args;
    ChSlices m = slices;
    ChNewton nw = newton;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const int cap = sms * kSliceBlocks < kSliceMaxGrid ? sms * kSliceBlocks : kSliceMaxGrid;
    // lanes a node: enough of them that three quarters of the resident warps have rows (256x256: one lane 9.2 ms, two
    // 9.3, four 11.6; 64x64: one 9.8, eight 5.9)
    const long long warps = (long long)cap * (kSliceThreads / kWarp), slices32 = (a.n + kWarp - 1) / kWarp;
    int lpn = 1;
    while (lpn < 8 && 4 * slices32 * lpn < 3 * warps) lpn *= 2;
    const long long need = (slices32 * lpn + kSliceThreads / kWarp - 1) / (kSliceThreads / kWarp);
    const int grid = (int)(need < cap ? need : cap);
    switch (lpn) {
        case 1: return launch_newton<1>(a, m, nw, grid, s);
        case 2: return launch_newton<2>(a, m, nw, grid, s);
        case 4: return launch_newton<4>(a, m, nw, grid, s);
        default: return launch_newton<8>(a, m, nw, grid, s);
    }
}

cudaError_t launch_bicg_solve(const BicgArgs &a, double tol, int max_its, cudaStream_t s) {
    static int grid = 0;  // resident blocks of the device: at most kBicgParts
    if (grid == 0) {
        int dev = 0, sms = 0, per_sm = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bicg_solve_kernel, kThreads, 0);
        if (e != cudaSuccess) return e;
        const int g = sms * per_sm;
        if (g < 1) return cudaErrorCooperativeLaunchTooLarge;
        grid = g < kMaxGrid ? g : kMaxGrid;
    }
    cudaError_t e = cudaMemsetAsync(a.sc, 0, sizeof(BicgScalars), s);
    if (e != cudaSuccess) return e;
    BicgArgs args = a;
    void *params[] = {&args, &tol, &max_its};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(bicg_solve_kernel), dim3(grid), dim3(kThreads),
                                       params, 0, s);
}

}  // namespace pxb
