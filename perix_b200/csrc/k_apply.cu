// Family-sum derivative apply D^k u_i = sum_j g^k_ij (u_j - u_i) and its transpose (reference pattern:
// PoissonElement::computeNodalProjection, src/ElmtSystem/PoissonElement.cpp:67-105; V_j is baked into g).
// Plus the small utility kernels (reverse-bond map, layout packing, health conversion, L2 flush).
#include <algorithm>
#include <type_traits>

#include "k_kernels.h"
#include "pxb_common.cuh"

namespace pxb {

constexpr int kMaxK = 20;

// Any operator row and slot list; rows of 2, 3, 5 and 9 operators go to apply_rows_kernel below instead.
// MIXED: FP32-stored operators widened to FP64 for the products and sums (HBM-bound: the arithmetic is free);
// with a.defect (mixed, order 2) every requested second derivative is corrected by the first-moment defect of
// its stored operator, D^k -= sum_m defect[k][m] D^m, the first derivatives D^m being summed alongside.
template <bool MIXED>
__global__ void __launch_bounds__(kApplyThreads) apply_kernel(ApplyArgs a) {
    constexpr int WPB = kApplyThreads / kWarp;
    using GT = typename std::conditional<MIXED, float, double>::type;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const GT *ops = static_cast<const GT *>(a.ops);
    for (int i = blockIdx.x * WPB + wib; i < a.n; i += gridDim.x * WPB) {
        const int b0 = a.off[i], b1 = a.off[i + 1];
        const double ui = a.u[i];
        double acc[kMaxK], d1[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int s = 0; s < kMaxK; ++s) acc[s] = 0.0;
        for (int t = b0 + lane; t < b1; t += kWarp) {
            const int j = __ldg(a.nbr + t);
            const double du = a.u[j] - ui;
            const GT *g = ops + (size_t)t * a.nop;
#pragma unroll
            for (int s = 0; s < kMaxK; ++s)
                if (s < a.nk) acc[s] = fma((double)__ldg(g + a.slots[s]), du, acc[s]);
            if (a.defect) {
#pragma unroll
                for (int m = 0; m < 3; ++m)
                    if (m < a.dim) d1[m] = fma((double)__ldg(g + m), du, d1[m]);
            }
        }
        double mine = 0.0;
#pragma unroll
        for (int s = 0; s < kMaxK; ++s) {
            if (s < a.nk) {
                const double v = group_sum<kWarp>(acc[s]);
                if (lane == s) mine = v;
            }
        }
        if (a.defect) {
#pragma unroll
            for (int m = 0; m < 3; ++m) d1[m] = (m < a.dim) ? group_sum<kWarp>(d1[m]) : 0.0;
            if (lane < a.nk && a.slots[lane] >= a.dim) {
                const int nd = (a.nop - a.dim) * a.dim;
                const float *dv = a.defect + (size_t)i * nd + (a.slots[lane] - a.dim) * a.dim;
                for (int m = 0; m < a.dim; ++m) mine -= (double)dv[m] * d1[m];
            }
        }
        if (lane < a.nk) a.out[(size_t)i * a.nk + lane] = mine;
    }
}

// Transpose of the defect correction, ahead of the transpose scatter: the corrected forward is
// D = G u - C (G1 u) with G1 the first-derivative rows, so ubar = G^T ybar' where ybar' equals ybar on the
// requested slots and every first-derivative slot m additionally receives -sum_k C[k][m] ybar[k], once however often
// it is requested.  p.ext lists the scatter's slots (the requested ones, then any first-derivative slot not requested);
// yeff is N x next.
__global__ void apply_adjoint_prep_kernel(AdjPrepArgs p) {
    const int nd = (p.nop - p.dim) * p.dim;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += gridDim.x * blockDim.x) {
        double *y = p.yeff + (size_t)i * p.next;
        for (int e = 0; e < p.next; ++e) y[e] = e < p.nk ? p.ybar[(size_t)i * p.nk + e] : 0.0;
        for (int s = 0; s < p.nk; ++s) {
            const int k = p.slots[s];
            if (k < p.dim) continue;
            const double yk = p.ybar[(size_t)i * p.nk + s];
            const float *dv = p.defect + (size_t)i * nd + (k - p.dim) * p.dim;
            for (int e = 0; e < p.next; ++e)
                if (p.once >> e & 1u) y[e] -= (double)dv[p.ext[e]] * yk;
        }
    }
}

cudaError_t launch_apply_adjoint_prep(const AdjPrepArgs &p, cudaStream_t s) {
    const int grid = (int)std::min<long long>(((long long)p.n + 255) / 256, 148LL * 8);
    apply_adjoint_prep_kernel<<<grid > 0 ? grid : 1, 256, 0, s>>>(p);
    return cudaGetLastError();
}

// One pass, no scratch: rows of other lengths, small meshes (apply_two_pass), and every row where the scratch of the two
// passes below is not to be had (memory, stream capture).
template <bool MIXED>
__global__ void __launch_bounds__(kApplyThreads) apply_adjoint_kernel(ApplyArgs a) {
    constexpr int WPB = kApplyThreads / kWarp;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    for (int m = blockIdx.x * WPB + wib; m < a.n; m += gridDim.x * WPB) {
        const int b0 = a.off[m], b1 = a.off[m + 1];
        double ym[kMaxK];
#pragma unroll
        for (int s = 0; s < kMaxK; ++s) ym[s] = (s < a.nk) ? a.u[(size_t)m * a.nk + s] : 0.0;
        double acc = 0.0;
        for (int t = b0 + lane; t < b1; t += kWarp) {
            const int j = __ldg(a.nbr + t);
            const int r = __ldg(a.rev + t);
#pragma unroll
            for (int s = 0; s < kMaxK; ++s) {
                if (s < a.nk) {
                    double gt, gr = 0.0;
                    if constexpr (MIXED) {
                        gt = (double)__ldg(static_cast<const float *>(a.ops) + (size_t)t * a.nop + a.slots[s]);
                        if (r >= 0) gr = (double)__ldg(static_cast<const float *>(a.ops) + (size_t)r * a.nop + a.slots[s]);
                    } else {
                        gt = __ldg(static_cast<const double *>(a.ops) + (size_t)t * a.nop + a.slots[s]);
                        if (r >= 0) gr = __ldg(static_cast<const double *>(a.ops) + (size_t)r * a.nop + a.slots[s]);
                    }
                    acc += gr * a.u[(size_t)j * a.nk + s] - gt * ym[s];
                }
            }
        }
        acc = group_sum<kWarp>(acc);
        if (lane == 0) a.out[m] = acc;
    }
}

// ---- operator rows of a size known at compile time ---------------------------------------------------------
// Operators of first and second order (2 and 5 in 2D, 3 and 9 in 3D) and of third order in 2D (9): LPN lanes a
// node stride its family, so that a warp's loads cover consecutive operator rows and every sector of a row is
// used by the loads issued with it, and one butterfly over the group closes each sum.  `used` masks the
// operators that some slot asks for; a slot list in any order, with repeats, is met by selecting from the sums.
// What bounds both kernels is the operator stream (72 bytes a bond in 3D FP64), read once.
// 124,416 nodes, 14.2 million bonds, 9 FP64 operators (1.08 GB): 190 us, 0.87 of the measured copy rate; the warp a
// node over a run-time slot list (apply_kernel) 431 us.
template <int NOP>
__device__ __forceinline__ double pick(const double (&v)[NOP], int k) {
    double r = v[0];
#pragma unroll
    for (int q = 1; q < NOP; ++q) r = k == q ? v[q] : r;
    return r;
}

template <bool MIXED, int NOP, int LPN>
__global__ void __launch_bounds__(kApplyThreads) apply_rows_kernel(ApplyArgs a, unsigned int used) {
    using GT = typename std::conditional<MIXED, float, double>::type;
    const int q = (blockIdx.x * kApplyThreads + threadIdx.x) / LPN;
    const int gl = threadIdx.x & (LPN - 1);
    const bool act = q < a.n;
    const int i = act ? q : a.n - 1;
    const int b0 = a.off[i], b1 = act ? a.off[i + 1] : b0;
    const double ui = a.u[i];
    const GT *ops = static_cast<const GT *>(a.ops);
    double acc[NOP];
#pragma unroll
    for (int k = 0; k < NOP; ++k) acc[k] = 0.0;
    for (int t = b0 + gl; t < b1; t += LPN) {
        const double du = __ldg(a.u + __ldg(a.nbr + t)) - ui;
        const GT *g = ops + (size_t)t * NOP;
#pragma unroll
        for (int k = 0; k < NOP; ++k)
            if (used >> k & 1u) acc[k] = fma((double)__ldg(g + k), du, acc[k]);
    }
#pragma unroll
    for (int k = 0; k < NOP; ++k) acc[k] = group_sum<LPN>(acc[k]);
    for (int s = gl; s < a.nk && act; s += LPN) {
        const int k = a.slots[s];
        double v = pick<NOP>(acc, k);
        if (MIXED && a.defect && k >= a.dim) {
            const float *dv = a.defect + ((size_t)i * (NOP - a.dim) + (k - a.dim)) * a.dim;
            for (int m = 0; m < a.dim; ++m) v -= (double)__ldg(dv + m) * pick<NOP>(acc, m);
        }
        a.out[(size_t)i * a.nk + s] = v;
    }
}

// Transpose in two passes.  The first streams the operators in their own order and keeps one scalar a bond,
// s_t = sum_k g^k_t ybar_i^k (8 bytes), and the node's -sum_t s_t in out; the second adds the s of the reverse
// bonds.  Gathering the reverse bonds' operator rows instead reads 72 bytes a bond a second time, out of order.
// (apply_two_pass: the sizes where this pays.)
// Same mesh: 197 + 61 us (1.19 and 0.17 GB) against 717 us for the gather of rows (apply_adjoint_kernel).
template <bool MIXED, int NOP, int LPN>
__global__ void __launch_bounds__(kApplyThreads) adjoint_bonds_kernel(ApplyArgs a, unsigned int used, double *bond) {
    using GT = typename std::conditional<MIXED, float, double>::type;
    const int q = (blockIdx.x * kApplyThreads + threadIdx.x) / LPN;
    const int gl = threadIdx.x & (LPN - 1);
    const bool act = q < a.n;
    const int i = act ? q : a.n - 1;
    const int b0 = a.off[i], b1 = act ? a.off[i + 1] : b0;
    const GT *ops = static_cast<const GT *>(a.ops);
    double y[NOP];
#pragma unroll
    for (int k = 0; k < NOP; ++k) y[k] = 0.0;
    for (int s = 0; s < a.nk; ++s) {
        const double v = __ldg(a.u + (size_t)i * a.nk + s);
#pragma unroll
        for (int k = 0; k < NOP; ++k) y[k] += a.slots[s] == k ? v : 0.0;
    }
    double own = 0.0;
    for (int t = b0 + gl; t < b1; t += LPN) {
        const GT *g = ops + (size_t)t * NOP;
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < NOP; ++k)
            if (used >> k & 1u) v = fma((double)__ldg(g + k), y[k], v);
        bond[t] = v;
        own += v;
    }
    own = group_sum<LPN>(own);
    if (act && gl == 0) a.out[i] = -own;
}

template <int LPN>
__global__ void __launch_bounds__(kApplyThreads) adjoint_gather_kernel(ApplyArgs a, const double *bond) {
    const int q = (blockIdx.x * kApplyThreads + threadIdx.x) / LPN;
    const int gl = threadIdx.x & (LPN - 1);
    const bool act = q < a.n;
    const int i = act ? q : a.n - 1;
    const int b0 = a.off[i], b1 = act ? a.off[i + 1] : b0;
    double acc = 0.0;
#pragma unroll 4
    for (int t = b0 + gl; t < b1; t += LPN) {
        const int r = __ldg(a.rev + t);
        if (r >= 0) acc += __ldg(bond + r);
    }
    acc = group_sum<LPN>(acc);
    if (act && gl == 0) a.out[i] += acc;
}

static unsigned int used_ops(const ApplyArgs &a) {
    unsigned int m = 0;
    for (int s = 0; s < a.nk; ++s) m |= 1u << a.slots[s];
    if (a.defect)
        for (int s = 0; s < a.nk; ++s)
            if (a.slots[s] >= a.dim) m |= (1u << a.dim) - 1u;
    return m;
}

template <int LPN>
static int rows_grid(int n) {
    return (int)(((long long)n * LPN + kApplyThreads - 1) / kApplyThreads);
}

template <bool MIXED, int NOP, int LPN>
static cudaError_t rows_forward(const ApplyArgs &a, cudaStream_t s) {
    apply_rows_kernel<MIXED, NOP, LPN><<<rows_grid<LPN>(a.n), kApplyThreads, 0, s>>>(a, used_ops(a));
    return cudaGetLastError();
}

template <bool MIXED, int NOP, int LPN>
static cudaError_t rows_adjoint(const ApplyArgs &a, double *bond, cudaStream_t s) {
    ApplyArgs b = a;
    b.defect = nullptr;  // already transposed into ybar
    adjoint_bonds_kernel<MIXED, NOP, LPN><<<rows_grid<LPN>(a.n), kApplyThreads, 0, s>>>(b, used_ops(b), bond);
    adjoint_gather_kernel<LPN><<<rows_grid<LPN>(a.n), kApplyThreads, 0, s>>>(b, bond);
    return cudaGetLastError();
}

// `f(mixed, nop, lanes)` for an operator row with a kernel of its own; false: the general kernels
template <typename F>
static bool with_rows(const ApplyArgs &a, bool mixed, F f) {
    auto lanes = [&](auto nop) {
        using N = decltype(nop);
        auto by_type = [&](auto lpn) {
            if (mixed) f(std::true_type{}, N{}, lpn);
            else f(std::false_type{}, N{}, lpn);
        };
        if (a.dim == 3) by_type(std::integral_constant<int, 16>{});
        else by_type(std::integral_constant<int, 8>{});
    };
    switch (a.nop) {
        case 2: lanes(std::integral_constant<int, 2>{}); return true;
        case 3: lanes(std::integral_constant<int, 3>{}); return true;
        case 5: lanes(std::integral_constant<int, 5>{}); return true;
        case 9: lanes(std::integral_constant<int, 9>{}); return true;
        default: return false;
    }
}

// The two passes are two launches, and the first call on a mesh allocates their scratch (0.3-0.6 ms); the one pass gathers
// reverse rows, which costs little while they stay in L2.  In 3D what it costs goes with the operators asked for, in 2D
// hardly.  One pass against two, FP64, us a call among others:
//   3D, nine operators   142 K bonds 14.4 / 14.4, 363 K 26.6 / 17.5, 1.3 M 69 / 35;   one operator 363 K 10.3 / 13.4,
//   1.3 M 32.7 / 26.0, 3.2 M 67.7 / 60.9
//   2D, five operators   106 K 8.3 / 12.3, 431 K 16.5 / 14.1, 1.7 M 67.6 / 31.1;      one operator 431 K 11.8 / 12.3,
//   1.7 M 47.2 / 26.1
// The lines below lie where a call saves 5 to 10 us, so that some tens of calls pay for the scratch.  Mixed 3D calls, whose
// rows are half as long and whose one pass is hidden behind the host's work up to there (363 K bonds 32.8 / 24.4, 1.3 M
// 61.5 / 34.7 of some 120 us for both directions through torch): later.
bool apply_two_pass(const ApplyArgs &a, bool mixed, long long nb) {
    if (a.nop != 2 && a.nop != 3 && a.nop != 5 && a.nop != 9) return false;
    if (a.dim == 2) return nb >= 800000;
    ApplyArgs b = a;
    b.defect = nullptr;
    return nb * (2 + __builtin_popcount(used_ops(b))) >= (mixed ? 8000000 : 2900000);
}

cudaError_t launch_apply(const ApplyArgs &a, bool mixed, int grid, cudaStream_t s) {
    if (a.nk > kMaxK) return cudaErrorInvalidValue;
    cudaError_t e = cudaSuccess;
    if (with_rows(a, mixed, [&](auto mx, auto nop, auto lpn) {
            e = rows_forward<decltype(mx)::value, decltype(nop)::value, decltype(lpn)::value>(a, s);
        }))
        return e;
    if (mixed) apply_kernel<true><<<grid, kApplyThreads, 0, s>>>(a);
    else apply_kernel<false><<<grid, kApplyThreads, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_apply_adjoint(const ApplyArgs &a, bool mixed, double *bond, int grid, cudaStream_t s) {
    if (a.nk > kMaxK) return cudaErrorInvalidValue;
    cudaError_t e = cudaSuccess;
    if (bond && with_rows(a, mixed, [&](auto mx, auto nop, auto lpn) {
            e = rows_adjoint<decltype(mx)::value, decltype(nop)::value, decltype(lpn)::value>(a, bond, s);
        }))
        return e;
    if (mixed) apply_adjoint_kernel<true><<<grid, kApplyThreads, 0, s>>>(a);
    else apply_adjoint_kernel<false><<<grid, kApplyThreads, 0, s>>>(a);
    return cudaGetLastError();
}

// ---- batched clouds: all order-2 derivatives of a scalar field, every cloud in one persistent launch -----------
// D^k u_i = sum_t g^k_t (u_j - u_i) for k < nop (5 in 2D, 9 in 3D); LPN lanes per node stride the family
// (coalesced reads of consecutive operator rows), a butterfly over the group reduces the nop sums.
// MIXED: the operators are stored in FP32 and widened; products and sums stay FP64 (the kernel is HBM-bound,
// the arithmetic is free), and each second derivative is corrected by the first-moment defect of its stored
// operator: D^k -= sum_m defect[k][m] D^m (GBuildArgs::defect).
template <bool MIXED, int DIM, int LPN>
__device__ __forceinline__ void apply_batch_group(const BatchArgs &b, const BatchCloud &cd, int i, bool act, int gl) {
    constexpr int NOP = DIM == 3 ? 9 : 5;
    constexpr int ND = (NOP - DIM) * DIM;
    using GT = typename std::conditional<MIXED, float, double>::type;
    const GT *ops = static_cast<const GT *>(b.ops) + cd.ops_off;
    const int b0 = act ? b.off[i] : 0, b1 = act ? b.off[i + 1] : 0;
    const double ui = act ? b.u[i] : 0.0;
    double acc[NOP];
#pragma unroll
    for (int k = 0; k < NOP; ++k) acc[k] = 0.0;
    for (int t = b0 + gl; t < b1; t += LPN) {
        const int j = __ldg(b.nbr + t);
        const double du = __ldg(b.u + j) - ui;
        const GT *g = ops + (size_t)(t - cd.bond0) * NOP;
#pragma unroll
        for (int k = 0; k < NOP; ++k) acc[k] = fma((double)__ldg(g + k), du, acc[k]);
    }
#pragma unroll
    for (int k = 0; k < NOP; ++k) acc[k] = group_sum<LPN>(acc[k]);
    if constexpr (MIXED) {
        if (b.defect && act) {
            const float *dv = b.defect + cd.def_off + (size_t)(i - cd.node0) * ND;
#pragma unroll
            for (int k = DIM; k < NOP; ++k)
#pragma unroll
                for (int m = 0; m < DIM; ++m) acc[k] -= (double)__ldg(dv + (k - DIM) * DIM + m) * acc[m];
        }
    }
    // lane gl writes the derivatives k = gl, gl + LPN, ... (groups narrower than nop write several)
    double *o = b.out + cd.out_off + (size_t)(i - cd.node0) * NOP;
#pragma unroll
    for (int k = 0; k < NOP; ++k)
        if (act && gl == (k & (LPN - 1))) o[k] = acc[k];
}

template <bool MIXED, int LPN2, int LPN3, int DIMS>
__global__ void __launch_bounds__(kApplyThreads) apply_batch_kernel(BatchArgs b) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        int task = 0;
        if (lane == 0) task = (int)atomicAdd(b.counter, 1u);
        task = __shfl_sync(kFull, task, 0);
        if (task >= b.ntasks) break;
        const BatchTask tk = b.tasks[b.task0 + task];
        const BatchCloud cd = b.clouds[tk.cloud];
        if constexpr ((DIMS & 1) != 0) {
            if (tk.dim == 2) {
                constexpr int GPW = kWarp / LPN2;
                for (int k0 = 0; k0 < tk.count; k0 += GPW) {
                    const int q = k0 + lane / LPN2;
                    apply_batch_group<MIXED, 2, LPN2>(b, cd, tk.first + (q < tk.count ? q : 0), q < tk.count,
                                                      lane & (LPN2 - 1));
                }
            }
        }
        if constexpr ((DIMS & 2) != 0) {
            if (tk.dim == 3) {
                constexpr int GPW = kWarp / LPN3;
                for (int k0 = 0; k0 < tk.count; k0 += GPW) {
                    const int q = k0 + lane / LPN3;
                    apply_batch_group<MIXED, 3, LPN3>(b, cd, tk.first + (q < tk.count ? q : 0), q < tk.count,
                                                      lane & (LPN3 - 1));
                }
            }
        }
    }
}

BatchSchedule batch_apply_schedule(int v) {
    switch (v) {
        case 0: return {8, 16, false};
        case 1: return {4, 16, false};
        case 2: return {8, 32, false};
        case 3: return {8, 16, true};
        case 4: return {16, 16, false};
        case 5: return {4, 16, true};
        case 6: return {4, 32, false};
        case 7: return {16, 32, true};
        case 8: return {4, 32, true};
        default: return {8, 32, true};
    }
}

template <bool MIXED, int LPN2, int LPN3, int DIMS>
static cudaError_t launch_ab(const BatchArgs &a, cudaStream_t s) {
    auto k = apply_batch_kernel<MIXED, LPN2, LPN3, DIMS>;
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kApplyThreads, 0);
    const long long want = ((long long)a.ntasks + (kApplyThreads / kWarp) - 1) / (kApplyThreads / kWarp);
    const long long cap = (long long)sms * (per_sm > 0 ? per_sm : 1);
    const int grid = (int)(want < cap ? (want > 0 ? want : 1) : cap);
    k<<<grid, kApplyThreads, 0, s>>>(a);
    return cudaGetLastError();
}

template <bool MIXED>
static cudaError_t launch_ab_m(const BatchArgs &a, int variant, int dims, cudaStream_t s) {
    switch (variant) {
        case 0: return launch_ab<MIXED, 8, 16, 3>(a, s);
        case 1: return launch_ab<MIXED, 4, 16, 3>(a, s);
        case 2: return launch_ab<MIXED, 8, 32, 3>(a, s);
        case 3: return dims == 1 ? launch_ab<MIXED, 8, 16, 1>(a, s) : launch_ab<MIXED, 8, 16, 2>(a, s);
        case 4: return launch_ab<MIXED, 16, 16, 3>(a, s);
        case 5: return dims == 1 ? launch_ab<MIXED, 4, 16, 1>(a, s) : launch_ab<MIXED, 4, 16, 2>(a, s);
        case 6: return launch_ab<MIXED, 4, 32, 3>(a, s);
        case 7: return dims == 1 ? launch_ab<MIXED, 16, 32, 1>(a, s) : launch_ab<MIXED, 16, 32, 2>(a, s);
        case 8: return dims == 1 ? launch_ab<MIXED, 4, 32, 1>(a, s) : launch_ab<MIXED, 4, 32, 2>(a, s);
        case 9: return dims == 1 ? launch_ab<MIXED, 8, 32, 1>(a, s) : launch_ab<MIXED, 8, 32, 2>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_apply_batch(const BatchArgs &a, bool mixed, int variant, int dims, cudaStream_t s) {
    return mixed ? launch_ab_m<true>(a, variant, dims, s) : launch_ab_m<false>(a, variant, dims, s);
}

// ---- reverse bond: rev[t] = position of i in fam(j) for t = (i -> j), -1 when absent ------------------
__global__ void build_rev_kernel(int n, const int *off, const int *nbr, int *rev) {
    constexpr int WPB = kApplyThreads / kWarp;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    for (int i = blockIdx.x * WPB + wib; i < n; i += gridDim.x * WPB) {
        for (int t = off[i] + lane; t < off[i + 1]; t += kWarp) {
            const int j = nbr[t];
            int found = -1;
            for (int q = off[j]; q < off[j + 1]; ++q)
                if (nbr[q] == i) { found = q; break; }
            rev[t] = found;
        }
    }
}

cudaError_t launch_build_rev(int n, const int *off, const int *nbr, int *rev, int grid, cudaStream_t s) {
    build_rev_kernel<<<grid, kApplyThreads, 0, s>>>(n, off, nbr, rev);
    return cudaGetLastError();
}

// ---- layout packing -------------------------------------------------------------------------------------
__global__ void pos_pack_kernel(int n, int dim, const double *c3, void *pos) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (dim == 2) static_cast<double2 *>(pos)[i] = make_double2(c3[3 * i], c3[3 * i + 1]);
        else static_cast<double4 *>(pos)[i] = make_double4(c3[3 * i], c3[3 * i + 1], c3[3 * i + 2], 0.0);
    }
}

cudaError_t launch_pos_pack(int n, int dim, const double *coords3, void *pos, cudaStream_t s) {
    const int g = (n + 255) / 256;
    pos_pack_kernel<<<g > 0 ? g : 1, 256, 0, s>>>(n, dim, coords3, pos);
    return cudaGetLastError();
}

__global__ void ids_to0_kernel(long long nb, const int *ids1, int *ids0) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nb; t += (long long)gridDim.x * blockDim.x)
        ids0[t] = ids1[t] - 1;
}

cudaError_t launch_ids_to0(long long nb, const int *ids1, int *ids0, cudaStream_t s) {
    long long g = (nb + 255) / 256;
    if (g > 65535LL * 8) g = 65535LL * 8;
    ids_to0_kernel<<<(int)(g > 0 ? g : 1), 256, 0, s>>>(nb, ids1, ids0);
    return cudaGetLastError();
}

__global__ void health_from_double_kernel(long long nb, const double *h, uint8_t *out) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nb; t += (long long)gridDim.x * blockDim.x)
        out[t] = h[t] > 0.0 ? 1 : 0;
}

__global__ void health_to_double_kernel(long long nb, const uint8_t *h, double *out) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nb; t += (long long)gridDim.x * blockDim.x)
        out[t] = h[t] ? 1.0 : 0.0;
}

__global__ void count_zero_kernel(long long nb, const uint8_t *h, unsigned long long *count) {
    unsigned long long c = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nb; t += (long long)gridDim.x * blockDim.x)
        c += (h[t] == 0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

static int grid_for(long long nb) {
    long long g = (nb + 255) / 256;
    if (g > 4096) g = 4096;
    return (int)(g > 0 ? g : 1);
}

cudaError_t launch_health_from_double(long long nb, const double *h, uint8_t *out, cudaStream_t s) {
    health_from_double_kernel<<<grid_for(nb), 256, 0, s>>>(nb, h, out);
    return cudaGetLastError();
}

cudaError_t launch_health_to_double(long long nb, const uint8_t *h, double *out, cudaStream_t s) {
    health_to_double_kernel<<<grid_for(nb), 256, 0, s>>>(nb, h, out);
    return cudaGetLastError();
}

cudaError_t launch_count_zero(long long nb, const uint8_t *h, unsigned long long *count, cudaStream_t s) {
    count_zero_kernel<<<grid_for(nb), 256, 0, s>>>(nb, h, count);
    return cudaGetLastError();
}

// L2 flush between timed launches: write `bytes` (a multiple of 16, larger than L2) so that the previous
// working set is evicted, then read the buffer back so that the dirty lines of the write are written back
// before the timed kernel starts (L2 then holds clean lines of this buffer only, none of the kernel's inputs).
__global__ void l2_flush_kernel(uint4 *buf, size_t n16, unsigned seed) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n16; k += (size_t)gridDim.x * blockDim.x)
        buf[k] = make_uint4(seed, (unsigned)k, seed ^ 0x9e3779b9u, 0u);
}

__global__ void l2_flush_read_kernel(uint4 *buf, size_t n16, unsigned seed) {
    unsigned acc = 0;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n16; k += (size_t)gridDim.x * blockDim.x) {
        const uint4 v = __ldcg(buf + k);
        acc += v.x ^ v.y ^ v.z ^ v.w;
    }
    if (acc == seed * 0x85ebca6bu + 1u) buf[0].w = acc;  // keeps the reads; the value never matters
}

__global__ void empty_kernel() {}

cudaError_t launch_empty(int grid, int block, size_t smem, cudaStream_t s) {
    static size_t configured = 0;
    if (smem > configured) {
        cudaError_t e = cudaFuncSetAttribute(empty_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured = smem;
    }
    empty_kernel<<<grid, block, smem, s>>>();
    return cudaGetLastError();
}

cudaError_t launch_l2_flush(void *buf, size_t bytes, cudaStream_t s) {
    static unsigned seed = 1;
    l2_flush_kernel<<<1184, 256, 0, s>>>(static_cast<uint4 *>(buf), bytes / 16, seed);
    l2_flush_read_kernel<<<1184, 256, 0, s>>>(static_cast<uint4 *>(buf), bytes / 16, seed++);
    return cudaGetLastError();
}

}  // namespace pxb
