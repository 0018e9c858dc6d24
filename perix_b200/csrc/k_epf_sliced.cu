// explicit_pddo_frac step on a sliced, neighbour-sorted copy of the bond streams.
//
// What bounds the step is memory: 53 bytes a bond in 3D FP64 (29 mixed), and the gathers of the neighbours'
// displacements.  The lanes-per-node kernels (k_epf.cu, k_epf_tma.cu) read the streams in family order, where the 32
// lanes of a warp gather 32 unrelated rows of u, three 8-byte loads each, and wait for them with 16-24 warps an SM.
// Here a slice is 32 consecutive nodes, a lane a node, and row k of a slice holds the k-th bond of every node with the
// families sorted by neighbour id.  On a lattice the k-th neighbours of consecutive nodes are consecutive nodes, so a
// gather is one run of u; on any mesh the coefficients and ids are read as full 256- and 128-byte lines, whose
// addresses depend on nothing, so several rows are in flight a warp without shared memory, barriers or waits.
//
// A bond's word is (broken << 31 | q << shift | neighbour): q is its length in units of step = r_max / 2^(31 - shift),
// rounded down (at most 7 bits, what the ids leave of 31).  A bond whose relative displacement satisfies
// |e|^2 < (s_c (1 - 1e-6) - 1e-12)^2 (q step)^2 holds under either criterion, whatever its direction, because its stretch is
// at most |e| / |xi|; only the others gather the position for the reference's test, so every decision is the
// reference's.  (The bound with the mesh's shortest bond in place of q step, the staged kernels' test, clears few
// bonds once the strain passes a third of s_c at a horizon of three spacings.)
// The health bytes stay the truth: a bond that breaks is written there and in its word, and the words are brought up to
// date (sliced_health_kernel) before a step whenever anything else may have written health.
// KW warps share a slice's rows (their sums meet in shared memory), so that a mesh of few slices still fills the chip.
// B200, a state with strains about the threshold: the 44.2 M-bond slab 550 -> 352 us a step in FP64 (2.36 GB of streams:
// 6.7 TB/s, the measured copy rate) and 451 -> 246 us mixed (5.2 TB/s; latency and issue, at 24 warps an SM), against
// the best staged configuration; the 2.25 M-bond plate in a captured loop 21.0 -> 16.1 us FP64, 16.1 -> 13.6 us mixed.
#include <type_traits>

#include "k_kernels.h"
#include "pxb_common.cuh"

namespace pxb {

namespace {


__device__ __forceinline__ unsigned long long stream_policy(bool evict) {
    unsigned long long p;
    if (evict) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    else asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ double ld_stream(const double *p, unsigned long long pol) {
    double v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ float ld_stream(const float *p, unsigned long long pol) {
    float v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
    return v;
}
// a bond's word: a step writes the words of the bonds it breaks, so no read-only path
__device__ __forceinline__ int ld_word(const int *p, unsigned long long pol) {
    int v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
}

// an intact bond by the squared comparison in contracted arithmetic: 1 holds, -1 breaks, 0 within 1e-6 r^2 of the
// threshold (the contraction's rounding is far inside that band; a zero-length bond is never tested and holds)
template <int DIM, typename PosT>
__device__ __forceinline__ int verdict(const PosT &xi, const PosT &xj, const double *e, double hi2, double lo2,
                                       bool tension_only) {
    double x[DIM];
    x[0] = xj.x - xi.x;
    x[1] = xj.y - xi.y;
    if constexpr (DIM == 3) x[2] = xj.z - xi.z;
    double r2 = 0.0, y2 = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const double y = x[d] + e[d];
        r2 = fma(x[d], x[d], r2);
        y2 = fma(y, y, y2);
    }
    const double band = 1.0e-6 * r2, qh = fma(-hi2, r2, y2), ql = fma(lo2, r2, -y2);
    if (!(r2 > 0.0) || (qh < -band && (tension_only || ql < -band))) return 1;
    return qh > band || (!tension_only && ql > band) ? -1 : 0;
}

// whether it breaks, in the reference's rounding where the squared comparison is within 1e-6 r^2 of the threshold
// (ExplicitPDDOFracElement.cpp:239-299)
template <int DIM, typename PosT>
__device__ __forceinline__ bool breaks(const PosT &xi, const PosT &xj, const double *e, const EpfArgs &a) {
    const double x0 = __dsub_rn(xj.x, xi.x), x1 = __dsub_rn(xj.y, xi.y);
    const double y0 = __dadd_rn(x0, e[0]), y1 = __dadd_rn(x1, e[1]);
    double r2 = __dadd_rn(__dmul_rn(x0, x0), __dmul_rn(x1, x1)), y2 = __dadd_rn(__dmul_rn(y0, y0), __dmul_rn(y1, y1));
    if constexpr (DIM == 3) {
        const double x2 = __dsub_rn(xj.z, xi.z), yz = __dadd_rn(x2, e[2]);
        r2 = __dadd_rn(r2, __dmul_rn(x2, x2));
        y2 = __dadd_rn(y2, __dmul_rn(yz, yz));
    }
    if (!(r2 > 0.0)) return false;
    const double band = 1.0e-6 * r2, qh = y2 - a.sc_hi2 * r2, ql = a.sc_lo2 * r2 - y2;
    if (qh > band || (!a.tension_only && ql > band)) return true;
    if (qh < -band && (a.tension_only || ql < -band)) return false;
    const double r = sqrt(r2), s = __ddiv_rn(__dsub_rn(sqrt(y2), r), r);
    return (a.tension_only ? s : fabs(s)) > a.sc;
}

template <int DIM, typename GT>
__device__ __forceinline__ void add_force(const GT *g, const double *e, double *L) {
    if constexpr (DIM == 3) {
        L[0] = fma((double)g[0], e[0], fma((double)g[3], e[1], fma((double)g[4], e[2], L[0])));
        L[1] = fma((double)g[3], e[0], fma((double)g[1], e[1], fma((double)g[5], e[2], L[1])));
        L[2] = fma((double)g[4], e[0], fma((double)g[5], e[1], fma((double)g[2], e[2], L[2])));
    } else {
        L[0] = fma((double)g[0], e[0], fma((double)g[2], e[1], L[0]));
        L[1] = fma((double)g[2], e[0], fma((double)g[1], e[1], L[1]));
    }
}

template <int DIM>
__device__ __forceinline__ void load_u(const double *u, size_t i, double *v) {
    if constexpr (DIM == 2) {
        const double2 w = __ldg(reinterpret_cast<const double2 *>(u) + i);
        v[0] = w.x;
        v[1] = w.y;
    } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = __ldg(u + i * 3 + d);
    }
}

// The nodes' vectors of a warp (lane = node i) as whole 16- or 8-byte pieces of consecutive addresses: the rate call may
// point `out` at pinned host memory, where strided pieces would cross the bus one by one.
template <int DIM>
__device__ __forceinline__ void store_nodes(double *out, int i, bool act, const double (&v)[DIM]) {
    const int lane = threadIdx.x & 31;
    if constexpr (DIM == 2) {
        if ((reinterpret_cast<unsigned long long>(out) & 15) == 0) {
            if (act) reinterpret_cast<double2 *>(out)[i] = make_double2(v[0], v[1]);
            return;
        }
    }
    const unsigned live = __ballot_sync(kFull, act);
    double *base = out + (size_t)(i - lane) * DIM;  // (lane 0's node may be out of range: never written then)
#pragma unroll
    for (int q = 0; q < DIM; ++q) {
        const int e = q * 32 + lane, node = e / DIM, d = e % DIM;
        double x = 0.0;
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
            const double y = __shfl_sync(kFull, v[c], node);
            if (c == d) x = y;
        }
        if (live >> node & 1u) base[e] = x;
    }
}

}  // namespace

// KW warps a slice, SPB slices a block, U rows in flight a lane.  The loop has no bounds of its own: short families are
// padded with broken words and zero coefficients (0.1 % of a 2D lattice's entries, 0.4-2 % in 3D), and the words are
// read U rows ahead, past the slice's end if need be (kSlicedSlack rows after the last slice).
template <int DIM, bool MIXED, int KW, int SPB, int U, int MINB>
__global__ void __launch_bounds__(KW * SPB * 32, MINB) epf_sliced_kernel(EpfArgs a, SlicedArgs sl) {
    using GT = typename std::conditional<MIXED, float, double>::type;
    using PosT = typename Vec<DIM>::T;
    constexpr int NC = DIM == 3 ? 6 : 3;
    static_assert(U <= kSlicedSlack, "words are read U rows ahead");
    __shared__ double part[SPB][KW > 1 ? KW - 1 : 1][DIM][32];
    __shared__ double clear[2 * kSlicedClasses];  // by word >> shift: |e|^2 below it clearly holds; broken: nothing does
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, sub = wib / KW, w = wib % KW;
    const int slice = a.node0 / 32 + blockIdx.x * SPB + sub;
    const int i = slice * 32 + lane;
    const bool act = i < a.n;
    const bool step = a.rate == kEpfStep;
    int r0 = 0, rows = 0;
    if (slice * 32 < a.n) {
        r0 = __ldg(sl.row0 + slice);
        rows = __ldg(sl.row0 + slice + 1) - r0;
    }
    for (int q = threadIdx.x; q < 2 * kSlicedClasses; q += KW * SPB * 32)
        clear[q] = q >> (31 - sl.shift) ? -1.0 : a.damage ? sl.clear * (double)(q * q) : __longlong_as_double(0x7ff0000000000000LL);
    const int kb = rows * w / KW, ke = rows * (w + 1) / KW;
    const GT *P = static_cast<const GT *>(sl.P) + ((size_t)(r0 + kb) * NC * 32 + lane);
    const int *W = sl.word + ((size_t)(r0 + kb) * 32 + lane);
    const unsigned long long pol = stream_policy(a.evict_first);
    const unsigned idmask = (1u << sl.shift) - 1u;
    const PosT *pos = static_cast<const PosT *>(a.pos);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // (words and u are written by the step before)
    double ui[DIM], up[DIM], L[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) ui[d] = up[d] = L[d] = 0.0;
    unsigned own_bits = 0;
    int e0 = 0, e1 = 0;
    int wd[U];
#pragma unroll
    for (int q = 0; q < U; ++q) wd[q] = ld_word(W + q * 32, pol);
    if (act) {
        load_u<DIM>(a.u, i, ui);
        if (w == 0 && step) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) up[d] = a.u_other[(size_t)i * DIM + d];
            if (a.bc_own) own_bits = __ldg(a.bc_own + i);
            if (a.bc_off) {
                e0 = __ldg(a.bc_off + i);
                e1 = __ldg(a.bc_off + i + 1);
            }
        }
    }
    unsigned broken = 0;
    // a bond breaks: in its word and in the health bytes
    auto break_bond = [&](const int *at, int wq) {
        const size_t k = (size_t)(at - sl.word);
        sl.word[k] = wq | (int)0x80000000u;
        a.health[__ldg(a.off + i) + sl.src[k]] = 0;
        return 1u;
    };
    // N rows whose words are in wd: coefficients and displacements, the words U rows on, then the arithmetic
    auto pass = [&](auto count) {
        constexpr int N = decltype(count)::value;
        GT p[N][NC];
#pragma unroll
        for (int q = 0; q < N; ++q)
#pragma unroll
            for (int c = 0; c < NC; ++c) p[q][c] = ld_stream(P + (q * NC + c) * 32, pol);
        double e[N][DIM];
#pragma unroll
        for (int q = 0; q < N; ++q) load_u<DIM>(a.u, (unsigned)wd[q] & idmask, e[q]);
        int wn[N];
#pragma unroll
        for (int q = 0; q < N; ++q) wn[q] = ld_word(W + (U + q) * 32, pol);
        bool hold[N], open = false;  // open: intact bonds that the clear test does not decide
#pragma unroll
        for (int q = 0; q < N; ++q) {
            double ee = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                e[q][d] = __dsub_rn(e[q][d], ui[d]);
                ee = fma(e[q][d], e[q][d], ee);
            }
            hold[q] = ee < clear[(unsigned)wd[q] >> sl.shift];
            open = open || (!hold[q] && wd[q] >= 0);
        }
        unsigned late = 0;
        if (__any_sync(kFull, open)) {  // these rows' positions, all at once
            const PosT xi = ldg_vec(pos + (act ? i : 0));
            PosT xj[N];
#pragma unroll
            for (int q = 0; q < N; ++q) xj[q] = ldg_vec(pos + ((unsigned)wd[q] & idmask));
#pragma unroll
            for (int q = 0; q < N; ++q)
                if (!hold[q] && wd[q] >= 0) {
                    const int v = a.damage ? verdict<DIM>(xi, xj[q], e[q], a.sc_hi2, a.sc_lo2, a.tension_only) : 1;
                    hold[q] = v > 0;
                    if (v == 0) late |= 1u << q;
                    if (v < 0) broken += break_bond(W + q * 32, wd[q]);
                }
        }
#pragma unroll
        for (int q = 0; q < N; ++q)
            if (hold[q]) add_force<DIM>(p[q], e[q], L);
        // the few bonds near the threshold, everything read again (nothing of the fast path is kept for them)
        while (late) {
            const int q = __ffs(late) - 1;
            late &= late - 1;
            const int wq = ld_word(W + q * 32, pol), j = (unsigned)wq & idmask;
            double ej[DIM];
            load_u<DIM>(a.u, j, ej);
#pragma unroll
            for (int d = 0; d < DIM; ++d) ej[d] = __dsub_rn(ej[d], ui[d]);
            if (breaks<DIM>(ldg_vec(pos + i), ldg_vec(pos + j), ej, a)) {
                broken += break_bond(W + q * 32, wq);
            } else {
                GT g[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) g[c] = __ldg(P + (q * NC + c) * 32);
                add_force<DIM>(g, ej, L);
            }
        }
        P += N * NC * 32;
        W += N * 32;
        if constexpr (N == U) {
#pragma unroll
            for (int q = 0; q < U; ++q) wd[q] = wn[q];
        } else {  // (the last rows, one at a time: the words move up)
#pragma unroll
            for (int q = 0; q + 1 < U; ++q) wd[q] = wd[q + 1];
        }
    };
    int k = kb;
    for (; k + U <= ke; k += U) pass(std::integral_constant<int, U>{});
    if constexpr (U > 1)
        for (; k < ke; ++k) pass(std::integral_constant<int, 1>{});
    if (__any_sync(kFull, broken != 0)) {
        broken = __reduce_add_sync(kFull, broken);
        if (lane == 0 && a.n_broken) atomicAdd(a.n_broken, (unsigned long long)broken);
    }
    if constexpr (KW > 1) {
        if (w > 0)
#pragma unroll
            for (int d = 0; d < DIM; ++d) part[sub][w - 1][d][lane] = L[d];
        __syncthreads();
        if (w > 0) return;
#pragma unroll
        for (int q = 0; q < KW - 1; ++q)
#pragma unroll
            for (int d = 0; d < DIM; ++d) L[d] += part[sub][q][d][lane];
    }
    if (a.rate == kEpfRate) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) L[d] = __ddiv_rn(__dadd_rn(L[d], a.b[d]), a.rho);
        store_nodes<DIM>(a.accel, i, act, L);
        return;
    }
    double umax = 0.0, un[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const double acc = __ddiv_rn(__dadd_rn(L[d], a.b[d]), a.rho);
        un[d] = 0.0;
        if (act && a.rate == kEpfStart) {
            const double v = a.v0 ? a.v0[(size_t)i * DIM + d] : 0.0;
            a.u_other[(size_t)i * DIM + d] = __dadd_rn(__dsub_rn(ui[d], __dmul_rn(a.dt, v)), __dmul_rn(a.dt2, acc));
        }
        if (act && step) {
            un[d] = cd_next(ui[d], up[d], acc, a.dt2, a.var_step, a.cv_rho, a.cv_w);
            if (!((own_bits >> d) & 1u)) {
                a.u_other[(size_t)i * DIM + d] = un[d];
                umax = max_nan(umax, fabs(un[d]));
            }
        }
    }
    if (!step) return;
    const double t_new = e1 > e0 ? a.t_sched[a.step_in_chunk] : 0.0;
    for (int q = e0; q < e1; ++q) {  // the BC entries that read this node's new value (see EpfArgs)
        const int comp = a.bc_comp[q], form = a.bc_form[q];
        const double g1 = __dadd_rn(a.bc_val[q], __dmul_rn(a.bc_vel[q], t_new));
        double own = un[0];
#pragma unroll
        for (int d = 1; d < DIM; ++d)
            if (comp == d) own = un[d];
        double v;
        if (form == 0) v = own;
        else if (form == 1) v = g1;
        else if (form == 2) v = __dsub_rn(__dmul_rn(2.0, g1), own);
        else v = __dsub_rn(__dmul_rn(2.0, g1), __dadd_rn(a.bc_val2[q], __dmul_rn(a.bc_vel2[q], t_new)));
        a.u_other[(size_t)a.bc_tgt[q] * DIM + comp] = v;
        umax = max_nan(umax, fabs(v));
    }
    umax = group_max_nan<kWarp>(umax);
    if (lane == 0 && a.umax) {
        const unsigned long long key = dbl_key(umax);
        volatile unsigned long long *m = a.umax + a.step_in_chunk;
        if (key > *m) atomicMax(a.umax + a.step_in_chunk, key);  // most slices find a larger value there
    }
}

// ---- the reverse-only adjoint step on the slices -----------------------------------------------------------------
// The sums of epf_adjoint_tma_kernel (k_epf_tma.cu) with a lane a node: row k of a slice holds the reverse operators of
// the nodes' k-th bonds (sl.P: G in reverse-bond order) and words whose broken bit is the reverse bond's health.  Per bond
// with source node j, L = abar_j and e = u_m - u_j, the force adjoint is split by constant,
//   a1 = (g_d L_d),  a2 = the mixed-derivative part of L,  a3 = ((tr g - g_d) L_d),
//   P(g) L = C11 a1 + (C12 + C66) a2 + C66 a3,   dC11 = a1.e,  dC12 = a2.e,  dC66 = (a2 + a3).e,
// so scale / rho multiplies the nodes' sums once.  11.2 M bonds in 3D FP64 (0.60 GB): 138 us a step staged, 102 us here
// (5.9 TB/s of the 6.5 a copy reaches).  dC: per-block sums into one of kDcSlots slots (an
// address taking three atomics a block would serialise them), added up by dc_collect_kernel.
template <int DIM>
__device__ __forceinline__ void split_force(const double *g, const double *L, double *a1, double *a2, double *a3) {
    if constexpr (DIM == 3) {
        a2[0] = fma(g[4], L[2], g[3] * L[1]);
        a2[1] = fma(g[5], L[2], g[3] * L[0]);
        a2[2] = fma(g[5], L[1], g[4] * L[0]);
        a3[0] = (g[1] + g[2]) * L[0];
        a3[1] = (g[0] + g[2]) * L[1];
        a3[2] = (g[0] + g[1]) * L[2];
    } else {
        a2[0] = g[2] * L[1];
        a2[1] = g[2] * L[0];
        a3[0] = g[1] * L[0];
        a3[1] = g[0] * L[1];
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) a1[d] = g[d] * L[d];
}

template <int DIM, bool MIXED, int KW, int SPB, int U, int MINB>
__global__ void __launch_bounds__(KW * SPB * 32, MINB) adjoint_sliced_kernel(EpfAdjArgs a, SlicedArgs sl) {
    using GT = typename std::conditional<MIXED, float, double>::type;
    constexpr int NC = DIM == 3 ? 6 : 3;
    static_assert(U <= kSlicedSlack, "words are read U rows ahead");
    __shared__ double part[SPB][KW > 1 ? KW - 1 : 1][DIM][32];
    __shared__ double s_dC[KW * SPB][3];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, sub = wib / KW, w = wib % KW;
    const int slice = blockIdx.x * SPB + sub, m = slice * 32 + lane;
    const bool act = m < a.n;
    int r0 = 0, rows = 0;
    if (slice * 32 < a.n) {
        r0 = __ldg(sl.row0 + slice);
        rows = __ldg(sl.row0 + slice + 1) - r0;
    }
    const int kb = rows * w / KW, ke = rows * (w + 1) / KW;
    const GT *P = static_cast<const GT *>(sl.P) + ((size_t)(r0 + kb) * NC * 32 + lane);
    const int *W = sl.word + ((size_t)(r0 + kb) * 32 + lane);
    const unsigned long long pol = stream_policy(a.evict_first);
    const unsigned idmask = (1u << sl.shift) - 1u;
    int wd[U];
#pragma unroll
    for (int q = 0; q < U; ++q) wd[q] = ld_word(W + q * 32, pol);
    double um[DIM], F[DIM], dC[3] = {0.0, 0.0, 0.0};  // F: the force sums with the constants in
#pragma unroll
    for (int d = 0; d < DIM; ++d) um[d] = F[d] = 0.0;
    if (act) load_u<DIM>(a.u, m, um);
    const double ac = a.C12 + a.C66;
    auto pass = [&](auto count) {
        constexpr int N = decltype(count)::value;
        GT p[N][NC];
#pragma unroll
        for (int q = 0; q < N; ++q)
#pragma unroll
            for (int c = 0; c < NC; ++c) p[q][c] = ld_stream(P + (q * NC + c) * 32, pol);
        double uj[N][DIM], L[N][DIM];
#pragma unroll
        for (int q = 0; q < N; ++q) {
            const unsigned j = (unsigned)wd[q] & idmask;
            if (a.UW) {  // one interleaved row (u_j, abar_j): DIM 16-byte loads
                const double2 *row = reinterpret_cast<const double2 *>(a.UW) + (size_t)j * DIM;
                double r[2 * DIM];
#pragma unroll
                for (int h = 0; h < DIM; ++h) {
                    const double2 v = __ldg(row + h);
                    r[2 * h] = v.x;
                    r[2 * h + 1] = v.y;
                }
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    uj[q][d] = r[d];
                    L[q][d] = r[DIM + d];
                }
            } else {
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    uj[q][d] = __ldg(a.u + (size_t)j * DIM + d);
                    L[q][d] = __ldg(a.abar + (size_t)j * DIM + d);
                }
            }
        }
        int wn[N];
#pragma unroll
        for (int q = 0; q < N; ++q) wn[q] = ld_word(W + (U + q) * 32, pol);
#pragma unroll
        for (int q = 0; q < N; ++q)
            if (wd[q] >= 0) {
                double g[NC], a1[DIM], a2[DIM], a3[DIM];
#pragma unroll
                for (int c = 0; c < NC; ++c) g[c] = (double)p[q][c];
                split_force<DIM>(g, L[q], a1, a2, a3);
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double e = um[d] - uj[q][d];
                    F[d] = fma(a.C11, a1[d], fma(ac, a2[d], fma(a.C66, a3[d], F[d])));
                    dC[0] = fma(a1[d], e, dC[0]);
                    dC[1] = fma(a2[d], e, dC[1]);
                    dC[2] = fma(a3[d], e, dC[2]);
                }
            }
        P += N * NC * 32;
        W += N * 32;
        if constexpr (N == U) {
#pragma unroll
            for (int q = 0; q < U; ++q) wd[q] = wn[q];
        } else {
#pragma unroll
            for (int q = 0; q + 1 < U; ++q) wd[q] = wd[q + 1];
        }
    };
    int k = kb;
    for (; k + U <= ke; k += U) pass(std::integral_constant<int, U>{});
    if constexpr (U > 1)
        for (; k < ke; ++k) pass(std::integral_constant<int, 1>{});
#pragma unroll
    for (int q = 0; q < 3; ++q) dC[q] = group_sum<kWarp>(dC[q]);
    if (lane == 0) {
        s_dC[wib][0] = dC[0];
        s_dC[wib][1] = dC[1];
        s_dC[wib][2] = dC[1] + dC[2];
    }
    if constexpr (KW > 1)
        if (w > 0)
#pragma unroll
            for (int d = 0; d < DIM; ++d) part[sub][w - 1][d][lane] = F[d];
    __syncthreads();
    const double lscale = a.scale * a.inv_rho;
    if (threadIdx.x < 3 && a.dC) {
        double s = 0.0;
        for (int q = 0; q < KW * SPB; ++q) s += s_dC[q][threadIdx.x];
        atomicAdd(a.dC + 3 * (blockIdx.x % kDcSlots) + threadIdx.x, lscale * s);
    }
    if (w > 0 || !act) return;
    if constexpr (KW > 1)
#pragma unroll
        for (int q = 0; q < KW - 1; ++q)
#pragma unroll
            for (int d = 0; d < DIM; ++d) F[d] += part[sub][q][d][lane];
    // the own bonds' term - P(SG_m) abar_m, then the central difference's transpose
    double sg[NC], wm[DIM], a1[DIM], a2[DIM], a3[DIM];
#pragma unroll
    for (int c = 0; c < NC; ++c) sg[c] = __ldg(a.SG + (size_t)m * NC + c);
#pragma unroll
    for (int d = 0; d < DIM; ++d) wm[d] = a.abar[(size_t)m * DIM + d];
    split_force<DIM>(sg, wm, a1, a2, a3);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const double own = fma(a.C11, a1[d], fma(ac, a2[d], a.C66 * a3[d]));
        const size_t k2 = (size_t)m * DIM + d;
        const double r = a.rin ? a.rin[k2] : 0.0;
        a.ubar[k2] = a.c_r * r + a.c_w * wm[d] + lscale * (F[d] - own);
        if (a.rout) a.rout[k2] = a.c_o * wm[d];
    }
}

__global__ void dc_collect_kernel(const double *slots, double *dC) {
    if (threadIdx.x < 3) {
        double s = dC[threadIdx.x];
        for (int k = 0; k < kDcSlots; ++k) s += slots[3 * k + threadIdx.x];
        dC[threadIdx.x] = s;
    }
}

// ---- building the slices ----------------------------------------------------------------------------------------
// Warp per node: bond b of the family goes to row rank(b) of the node's column, ranked by (neighbour id, b);
// rmax_key: the largest squared bond length (bit pattern, zeroed by the caller).
template <int DIM>
__global__ void __launch_bounds__(256) sliced_rank_kernel(int n, const int *off, const int *nbr, const void *posv,
                                                          const int *row0, uint16_t *src, unsigned long long *rmax_key) {
    using PosT = typename Vec<DIM>::T;
    const PosT *pos = static_cast<const PosT *>(posv);
    const int lane = threadIdx.x & 31;
    double rmax = 0.0;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const int b0 = off[i], len = off[i + 1] - b0;
        const PosT xi = pos[i];
        uint16_t *dst = src + (size_t)row0[i >> 5] * 32 + (i & 31);
        for (int c = 0; c < len; c += kWarp) {
            const int b = c + lane;
            const int j = b < len ? nbr[b0 + b] : 0;
            int rank = 0;
            for (int o = 0; o < len; ++o) {
                const int x = __ldg(nbr + b0 + o);
                rank += (x < j || (x == j && o < b)) ? 1 : 0;
            }
            if (b < len) {
                dst[(size_t)rank * 32] = (uint16_t)b;
                const PosT xj = pos[j];
                double r2 = (xj.x - xi.x) * (xj.x - xi.x) + (xj.y - xi.y) * (xj.y - xi.y);
                if constexpr (DIM == 3) r2 += (xj.z - xi.z) * (xj.z - xi.z);
                rmax = fmax(rmax, r2);
            }
        }
    }
    rmax = group_max<kWarp>(rmax);
    if (lane == 0) atomicMax(rmax_key, dbl_key(rmax));
}

// Eight warps a slice, each a share of its rows: the words (without the broken bit of real bonds) and the coefficients, row
// by row; rev: those of the reverse bonds.  (A row waits for a chain of three loads: with a warp a slice the first sweep on a
// mesh of 1,728 nodes in 3D spent 0.3 ms here.)
constexpr int kFillWarps = 8;

template <int DIM, typename GT>
__global__ void __launch_bounds__(256) sliced_fill_kernel(int n, const int *off, const int *nbr, const void *posv,
                                                          const int *row0, const uint16_t *src, int shift, double inv_step,
                                                          int qmax, const GT *Pc, long long ldb, const int *rev, int *word,
                                                          GT *P) {
    using PosT = typename Vec<DIM>::T;
    constexpr int NC = DIM == 3 ? 6 : 3;
    const PosT *pos = static_cast<const PosT *>(posv);
    const int lane = threadIdx.x & 31, nsl = (n + 31) / 32;
    for (int x = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < nsl * kFillWarps; x += (gridDim.x * blockDim.x) >> 5) {
        const int s = x / kFillWarps, w = x % kFillWarps, r0 = row0[s], rows = row0[s + 1] - r0, i = s * 32 + lane;
        const int b0 = i < n ? off[i] : 0, len = i < n ? off[i + 1] - b0 : 0;
        PosT xi{};
        if (i < n) xi = pos[i];
        for (int k = rows * w / kFillWarps; k < rows * (w + 1) / kFillWarps; ++k) {
            const size_t at = (size_t)(r0 + k) * 32 + lane;
            const int t = b0 + (k < len ? src[at] : 0);
            if (word) {
                int wd = (int)0x80000000u | (i < n ? i : 0);
                if (k < len) {
                    const int j = nbr[t];
                    const PosT xj = pos[j];
                    double r2 = (xj.x - xi.x) * (xj.x - xi.x) + (xj.y - xi.y) * (xj.y - xi.y);
                    if constexpr (DIM == 3) r2 += (xj.z - xi.z) * (xj.z - xi.z);
                    // rounded down with a margin far above the rounding of r: q step never exceeds the length
                    const int q = min(qmax, (int)(sqrt(r2) * inv_step * (1.0 - 1.0e-9)));
                    wd = j | q << shift;
                }
                word[at] = wd;
            }
            const int tc = k >= len ? -1 : (rev ? rev[t] : t);
#pragma unroll
            for (int c = 0; c < NC; ++c)
                P[((size_t)(r0 + k) * NC + c) * 32 + lane] = tc >= 0 ? Pc[(size_t)c * ldb + tc] : GT(0);
        }
    }
}

// The words' broken bits from the health bytes (rev: those of the reverse bonds): four warps a slice, eight rows in
// flight a lane (a warp a slice and a row at a time, each row waited for a chain of two or three loads: 147 us for
// 11.2 M bonds with rev, 70 us now)
__global__ void __launch_bounds__(256) sliced_health_kernel(int n, const int *off, const int *row0, const uint16_t *src,
                                                            const uint8_t *health, const int *rev, int *word) {
    constexpr int U = 8, KW = 4;
    const int lane = threadIdx.x & 31, nsl = (n + 31) / 32;
    for (int x = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < nsl * KW; x += (gridDim.x * blockDim.x) >> 5) {
        const int s = x / KW, w = x % KW, r0 = row0[s], rows = row0[s + 1] - r0, i = s * 32 + lane;
        const int b0 = i < n ? off[i] : 0, len = i < n ? off[i + 1] - b0 : 0;
        const int ke = min(len, rows * (w + 1) / KW);
        for (int k = rows * w / KW; k < ke; k += U) {
            int t[U], v[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const size_t at = (size_t)(r0 + k + q) * 32 + lane;
                t[q] = k + q < ke ? b0 + (int)src[at] : -1;
                v[q] = k + q < ke ? word[at] : 0;
            }
            if (rev)
#pragma unroll
                for (int q = 0; q < U; ++q) t[q] = t[q] >= 0 ? __ldg(rev + t[q]) : -1;
            uint8_t h[U];
#pragma unroll
            for (int q = 0; q < U; ++q) h[q] = t[q] >= 0 ? health[t[q]] : (uint8_t)0;
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int x2 = (v[q] & 0x7fffffff) | (h[q] ? 0 : (int)0x80000000u);
                if (k + q < ke && x2 != v[q]) word[(size_t)(r0 + k + q) * 32 + lane] = x2;
            }
        }
    }
}

namespace {
int slice_grid(long long n) {
    const long long g = ((n + 31) / 32 + 7) / 8;
    return (int)(g < 1 ? 1 : (g < 148 * 8 ? g : 148 * 8));
}

template <int DIM, bool MIXED, int KW, int SPB, int U, int MINB>
cudaError_t launch_sliced(const EpfArgs &a, const SlicedArgs &sl, cudaStream_t s) {
    auto k = epf_sliced_kernel<DIM, MIXED, KW, SPB, U, MINB>;
    const int slices = (a.n - a.node0 + 31) / 32, grid = (slices + SPB - 1) / SPB;
    if (grid <= 0) return cudaSuccess;
    epf_note_shape(LaunchShape{grid, KW * SPB * 32, 0});
    if (a.pdl && a.rate == kEpfStep) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3(KW * SPB * 32);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k, a, sl);
        if (e != cudaSuccess) return e;
    } else {
        k<<<grid, KW * SPB * 32, 0, s>>>(a, sl);
    }
    return cudaGetLastError();
}

// Sliced configurations (the autotuner picks): warps a slice, slices a block, rows in flight, minimum resident blocks.
// Measured in a captured 50-step loop, FP64 / mixed us a step: the 44.2 M-bond slab 4,1,2,6 352 / 246, 4,1,3,4 359 / 278,
// 4,1,1,8 356 / 269, 8,1,2,3 412 / 285, 3,1,2,8 376 / 245, 5,1,2,4 362 / 285; the 2.25 M-bond plate 3,1,2,10 14.2 / 12.4,
// 4,1,2,8 14.9 / 12.9, 2,2,4,5 15.2 / 13.0, 2,2,2,8 15.7 / 13.4, 5,1,2,6 15.1 / 13.1, 3,1,2,11 18.3 / 13.5, 1,2,4,10
// 17.4 / 14.0.  The last of each dimension, eight warps a slice, is for meshes of a few hundred slices.
template <int DIM, bool MIXED>
cudaError_t launch_cfg(const EpfArgs &a, const SlicedArgs &sl, int which, cudaStream_t s) {
    if constexpr (DIM == 3) {
        switch (which) {
            case 0: return launch_sliced<3, MIXED, 4, 1, 2, 6>(a, sl, s);
            case 1: return launch_sliced<3, MIXED, 4, 1, 3, 4>(a, sl, s);
            case 2: return launch_sliced<3, MIXED, 4, 1, 1, 8>(a, sl, s);
            default: return launch_sliced<3, MIXED, 8, 1, 1, 4>(a, sl, s);
        }
    } else {
        switch (which) {
            case 0: return launch_sliced<2, MIXED, 4, 1, 2, 8>(a, sl, s);
            case 1: return launch_sliced<2, MIXED, 2, 2, 4, 5>(a, sl, s);
            case 2: return launch_sliced<2, MIXED, 3, 1, 2, 10>(a, sl, s);
            default: return launch_sliced<2, MIXED, 8, 1, 2, 4>(a, sl, s);
        }
    }
}
}  // namespace

cudaError_t launch_epf_sliced(const EpfArgs &a, const SlicedArgs &sl, int dim, bool mixed, int which, cudaStream_t s) {
    if (!sl.word || !sl.P || !sl.row0 || !sl.src) return cudaErrorInvalidValue;
    if (dim == 3) return mixed ? launch_cfg<3, true>(a, sl, which, s) : launch_cfg<3, false>(a, sl, which, s);
    return mixed ? launch_cfg<2, true>(a, sl, which, s) : launch_cfg<2, false>(a, sl, which, s);
}

template <int DIM, bool MIXED, int KW, int SPB, int U, int MINB>
static cudaError_t launch_adj(const EpfAdjArgs &a, const SlicedArgs &sl, cudaStream_t s) {
    const int grid = ((a.n + 31) / 32 + SPB - 1) / SPB;
    adjoint_sliced_kernel<DIM, MIXED, KW, SPB, U, MINB><<<grid > 0 ? grid : 1, KW * SPB * 32, 0, s>>>(a, sl);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_sliced(const EpfAdjArgs &a, const SlicedArgs &sl, int dim, bool mixed, cudaStream_t s) {
    if (!sl.word || !sl.P || !sl.row0 || !a.SG) return cudaErrorInvalidValue;
    if (dim == 3) return mixed ? launch_adj<3, true, 4, 1, 2, 5>(a, sl, s) : launch_adj<3, false, 4, 1, 2, 5>(a, sl, s);
    return mixed ? launch_adj<2, true, 4, 1, 2, 6>(a, sl, s) : launch_adj<2, false, 4, 1, 2, 6>(a, sl, s);
}

cudaError_t launch_dc_collect(const double *slots, double *dC, cudaStream_t s) {
    dc_collect_kernel<<<1, 32, 0, s>>>(slots, dC);
    return cudaGetLastError();
}

cudaError_t launch_sliced_rank(int n, int dim, const int *off, const int *nbr, const void *pos, const int *row0, uint16_t *src,
                               unsigned long long *rmax_key, cudaStream_t s) {
    const int g = (n + 7) / 8 < 148 * 8 ? (n + 7) / 8 : 148 * 8;
    if (dim == 3) sliced_rank_kernel<3><<<g, 256, 0, s>>>(n, off, nbr, pos, row0, src, rmax_key);
    else sliced_rank_kernel<2><<<g, 256, 0, s>>>(n, off, nbr, pos, row0, src, rmax_key);
    return cudaGetLastError();
}

cudaError_t launch_sliced_fill(int n, int dim, bool mixed, const int *off, const int *nbr, const void *pos, const int *row0,
                               const uint16_t *src, int shift, double inv_step, int qmax, const void *Pc, long long ldb,
                               const int *rev, int *word, void *P, cudaStream_t s) {
    const int g = slice_grid((long long)kFillWarps * n);
    if (dim == 3) {
        if (mixed) sliced_fill_kernel<3, float><<<g, 256, 0, s>>>(n, off, nbr, pos, row0, src, shift, inv_step, qmax, (const float *)Pc, ldb, rev, word, (float *)P);
        else sliced_fill_kernel<3, double><<<g, 256, 0, s>>>(n, off, nbr, pos, row0, src, shift, inv_step, qmax, (const double *)Pc, ldb, rev, word, (double *)P);
    } else {
        if (mixed) sliced_fill_kernel<2, float><<<g, 256, 0, s>>>(n, off, nbr, pos, row0, src, shift, inv_step, qmax, (const float *)Pc, ldb, rev, word, (float *)P);
        else sliced_fill_kernel<2, double><<<g, 256, 0, s>>>(n, off, nbr, pos, row0, src, shift, inv_step, qmax, (const double *)Pc, ldb, rev, word, (double *)P);
    }
    return cudaGetLastError();
}

cudaError_t launch_sliced_health(int n, const int *off, const int *row0, const uint16_t *src, const uint8_t *health,
                                 const int *rev, int *word, cudaStream_t s) {
    sliced_health_kernel<<<slice_grid(4LL * n), 256, 0, s>>>(n, off, row0, src, health, rev, word);
    return cudaGetLastError();
}

// ---- the rate call's ends for page-locked buffers ------------------------------------------------------------------
// The displacement up and the broken-bond count before the kernel, and the counters (and, unless the kernel wrote it
// there itself, the acceleration) down after it, by threads that read and write the host's memory: a copy-engine node
// each costs the call several microseconds of hand-over.  A call on a plate of 81,200 nodes: 81 us with the copies, 75
// with these; on one of 2,600 nodes 35 and 19.
__global__ void __launch_bounds__(256) rate_up_kernel(size_t n, const double *host_u, double *u, unsigned long long *cnt,
                                                      bool wide) {
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k == 0) cnt[4] = cnt[0];
    if (wide) {
        if (2 * k + 1 < n) reinterpret_cast<double2 *>(u)[k] = reinterpret_cast<const double2 *>(host_u)[k];
        else if (2 * k < n) u[2 * k] = host_u[2 * k];
    } else if (k < n) {
        u[k] = host_u[k];
    }
}

__global__ void __launch_bounds__(256) rate_down_kernel(const unsigned long long *cnt, unsigned long long *host, size_t n,
                                                        const double *accel, double *host_a, bool wide) {
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k < 5) host[k] = cnt[k];
    if (wide) {
        if (2 * k + 1 < n) reinterpret_cast<double2 *>(host_a)[k] = reinterpret_cast<const double2 *>(accel)[k];
        else if (2 * k < n) host_a[2 * k] = accel[2 * k];
    } else if (k < n) {
        host_a[k] = accel[k];
    }
}

cudaError_t launch_rate_up(size_t n, const double *host_u, double *u, unsigned long long *cnt, cudaStream_t s) {
    const bool wide = ((reinterpret_cast<uintptr_t>(host_u) | reinterpret_cast<uintptr_t>(u)) & 15) == 0;
    const size_t words = wide ? (n + 1) / 2 : n;
    rate_up_kernel<<<(unsigned)((words + 255) / 256), 256, 0, s>>>(n, host_u, u, cnt, wide);
    return cudaGetLastError();
}

cudaError_t launch_rate_down(const unsigned long long *cnt, unsigned long long *host, size_t n, const double *accel,
                             double *host_a, cudaStream_t s) {
    const bool wide = ((reinterpret_cast<uintptr_t>(host_a) | reinterpret_cast<uintptr_t>(accel)) & 15) == 0;
    const size_t words = wide ? (n + 1) / 2 : n;
    rate_down_kernel<<<(unsigned)(words / 256 + 1), 256, 0, s>>>(cnt, host, n, accel, host_a, wide);
    return cudaGetLastError();
}

}  // namespace pxb
