// Families on the device, in the reference's order (src/PDMesh/CreatePDMesh.cpp:910-1082; the host restatement is
// pxb_families in host_mesh.cpp, which these kernels reproduce bit for bit).
//
// The reference opens cells of size `radius` in node order and, cell by cell, pairs the cell's members (a < b)
// and then each member with the members of the forward half of its neighbour cells (4 offsets in 2D, 13 in 3D);
// every accepted pair appends j to fam(i) and i to fam(j).  So every accepted pair has a visit key
//   (rank of the processing cell, phase = 0 intra / 1 + offset index, outer position, inner position)
// and fam(x) lists the partners of x in increasing key.  A cell's rank is the order in which it was opened, i.e.
// the order of its smallest node id, so that id stands in for the rank.
//
// The partners that x finds in one cell are in key order when the cell's members are taken by node id, and no two
// of the surrounding cells share (rank, phase).  So a family needs no sort of its own: the 3^dim cells are put in the
// order of (rank, phase), and the members that pass the test are written as they come.
//
// Steps: cell coordinates and a hash table of cells (min node id, member count); members per cell, by node id; per
// node: the surrounding cells in order, the reference's distance test on their members, counted, and in a second pass
// written.
// B200, 73,600 nodes in 3D (families of 113 from some 700 candidates): count 205 + write 150 + cells and scans 45 us; a
// thread a node with keyed candidates and a bitonic sort of every family by key: 206 + 383 + 337 + 75 us, and 12 bytes
// a bond of temporaries where the votes take 128 a node.
#include <cstdint>

#include "k_kernels.h"
#include "pxb_common.cuh"

namespace pxb {

namespace {

constexpr unsigned long long kEmpty = ~0ULL;
constexpr int kFamRun = 4;  // nodes a warp looks after at a time

__device__ __forceinline__ unsigned long long cell_key(long ix, long iy, long iz) {
    const long b = 1L << 20;
    return ((unsigned long long)(ix + b) << 42) | ((unsigned long long)(iy + b) << 21) | (unsigned long long)(iz + b);
}

__device__ __forceinline__ unsigned long long hash64(unsigned long long k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdULL;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ULL;
    k ^= k >> 33;
    return k;
}

__device__ __forceinline__ int find_slot(const unsigned long long *keys, unsigned mask, unsigned long long key) {
    unsigned s = (unsigned)hash64(key) & mask;
    for (unsigned probe = 0; probe <= mask; ++probe) {
        const unsigned long long k = keys[s];
        if (k == key) return (int)s;
        if (k == kEmpty) return -1;
        s = (s + 1) & mask;
    }
    return -1;
}

// Forward stencils of the reference (CreatePDMesh.cpp:1001-1010): offset (dx, dy, dz) has phase 1 + its index, the
// opposite offset the same phase with the roles exchanged.
constexpr int kSt2[4][3] = {{1, -1, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}};
constexpr int kSt3[13][3] = {{1, -1, -1}, {1, -1, 0}, {1, -1, 1}, {1, 0, -1}, {1, 0, 0}, {1, 0, 1}, {1, 1, -1},
                             {1, 1, 0},   {1, 1, 1},  {0, 1, -1}, {0, 1, 0},  {0, 1, 1}, {0, 0, 1}};
struct Phases {
    signed char v[27];  // cell (dx + 1) + 3 (dy + 1) + 9 (dz + 1): phase, negative where the other cell processes
};
constexpr Phases make_phases(bool is3d) {
    Phases p{};
    for (int o = 0; o < (is3d ? 13 : 4); ++o) {
        const int x = is3d ? kSt3[o][0] : kSt2[o][0], y = is3d ? kSt3[o][1] : kSt2[o][1], z = is3d ? kSt3[o][2] : 0;
        p.v[(x + 1) + 3 * (y + 1) + 9 * (z + 1)] = (signed char)(1 + o);
        p.v[(1 - x) + 3 * (1 - y) + 9 * (1 - z)] = (signed char)(-1 - o);
    }
    return p;
}
__constant__ Phases c_phases[2] = {make_phases(false), make_phases(true)};

}  // namespace

// cell coordinates of every node and insertion into the cell table (key, member count, smallest node id)
__global__ void fam_cells_kernel(FamArgs a) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const double *p = a.coords + 3 * (size_t)i;
        const long ix = (int)floor((p[0] - a.lo[0]) / a.radius);
        const long iy = (int)floor((p[1] - a.lo[1]) / a.radius);
        const long iz = a.is3d ? (int)floor((p[2] - a.lo[2]) / a.radius) : 0;
        if (ix < -(1L << 20) || ix >= (1L << 20) || iy < -(1L << 20) || iy >= (1L << 20) || iz < -(1L << 20) ||
            iz >= (1L << 20)) {
            atomicExch(&a.tot->err, 1);
            a.cell_of[i] = -1;
            continue;
        }
        a.cxyz[3 * (size_t)i] = (int)ix;
        a.cxyz[3 * (size_t)i + 1] = (int)iy;
        a.cxyz[3 * (size_t)i + 2] = (int)iz;
        const unsigned long long key = cell_key(ix, iy, iz);
        unsigned s = (unsigned)hash64(key) & a.mask;
        int slot = -1;
        for (unsigned probe = 0; probe <= a.mask; ++probe) {
            const unsigned long long prev = atomicCAS(a.keys + s, kEmpty, key);
            if (prev == kEmpty || prev == key) {
                slot = (int)s;
                break;
            }
            s = (s + 1) & a.mask;
        }
        if (slot < 0) {
            atomicExch(&a.tot->err, 2);
            a.cell_of[i] = -1;
            continue;
        }
        a.cell_of[i] = slot;
        atomicAdd(a.ccount + slot, 1);
        atomicMin(a.cminid + slot, i);
    }
}

// members of every cell as they come, then each to its place by node id (its rank among the cell's members)
__global__ void fam_members_kernel(FamArgs a) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const int s = a.cell_of[i];
        if (s < 0) continue;
        const int k = atomicAdd(a.cfill + s, 1);
        a.unsorted[a.cstart[s] + k] = i;
    }
}

__global__ void fam_order_members_kernel(FamArgs a) {
    if (a.tot->maxcell >= kFamCell) return;  // refused
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const int s = a.cell_of[i];
        if (s < 0) continue;
        const int b = a.cstart[s], c = a.ccount[s];
        int rank = 0;
        for (int k = 0; k < c; ++k) rank += a.unsorted[b + k] < i;
        a.members[b + rank] = i;
    }
}

// Warp per kFamRun nodes that follow each other in the cells' member lists, nearly always of one cell: the cell's
// surroundings are looked up and put in order once, and every candidate that a lane loads is tested against all of
// them.  The first pass counts, and keeps each pass of 32 candidates' votes (a word a pass and node, 32 words a node
// at most); the second writes the partners from the votes, or, for a node with more passes, from the tests again.
// What bounds it is instruction issue.  Cells with 16 members or more on average are taken one by one, a lane a
// member; smaller ones (2D: 9) are laid end to end, a lane a candidate, its cell found by bisection.
template <bool WRITE>
__global__ void __launch_bounds__(128) fam_partners_kernel(FamArgs a) {
    constexpr int WPB = 4, R = kFamRun;
    __shared__ int s_start[WPB][kWarp], s_first[WPB][kWarp];
    if (a.tot->err || a.tot->maxcell >= kFamCell) return;  // refused
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ncell = a.is3d ? 27 : 9, cell = a.is3d ? lane : 9 + lane;
    const unsigned before = (1u << lane) - 1u;
    for (int p0 = (blockIdx.x * WPB + w) * R; p0 < a.n; p0 += gridDim.x * WPB * R) {
        const int xl = lane < R && p0 + lane < a.n ? a.members[p0 + lane] : -1;
        const int sl = xl >= 0 ? a.cell_of[xl] : -1;
        for (int r = 0, r1; r < R && p0 + r < a.n; r = r1) {
            const int own = __shfl_sync(kFull, sl, r), x0 = __shfl_sync(kFull, xl, r);
            r1 = r + __popc(__ballot_sync(kFull, lane >= r && xl >= 0 && sl == own));
            // the cells around x0's, a lane a cell, in the order in which the reference processes them
            unsigned long long order = kEmpty;
            int start = 0, count = 0;
            if (lane < ncell) {
                const int dx = cell % 3 - 1, dy = cell / 3 % 3 - 1, dz = cell / 9 - 1, phase = c_phases[a.is3d].v[cell];
                const int *c = a.cxyz + 3 * (size_t)x0;
                const int s = find_slot(a.keys, a.mask, cell_key(c[0] + dx, c[1] + dy, c[2] + dz));
                if (s >= 0) {
                    start = a.cstart[s];
                    count = a.ccount[s];
                    const unsigned rank = (unsigned)a.cminid[phase < 0 ? s : own];
                    order = (unsigned long long)rank << 8 | (unsigned)abs(phase);
                }
            }
            int place = 0;  // the cells that are not there come last, empty
            for (int k = 0; k < ncell; ++k) {
                const unsigned long long o = __shfl_sync(kFull, order, k);
                place += o < order || (o == order && k < lane);
            }
            if (lane >= ncell) place = lane;
            __syncwarp();
            s_start[w][place] = start;
            s_first[w][place] = count;
            __syncwarp();
            start = s_start[w][lane];
            count = s_first[w][lane];
            int upto = count;
#pragma unroll
            for (int o = 1; o < kWarp; o <<= 1) {
                const int v = __shfl_up_sync(kFull, upto, o);
                if (lane >= o) upto += v;
            }
            const int total = __shfl_sync(kFull, upto, kWarp - 1);
            __syncwarp();
            s_first[w][lane] = upto - count;
            __syncwarp();
            const bool by_cell = total >= 16 * ncell;
            const int passes = by_cell ? __reduce_add_sync(kFull, (count + kWarp - 1) / kWarp) : (total + kWarp - 1) / kWarp;
            const bool votes = passes <= kWarp;
            double px[R], py[R], pz[R];
            int x[R], found[R], *out[R];
            unsigned vote[R];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                x[q] = __shfl_sync(kFull, xl, q);
                const bool in = q >= r && q < r1;
                const double *c = a.coords + 3 * (size_t)(in ? x[q] : 0);
                px[q] = in ? c[0] : __longlong_as_double(0x7ff8000000000000LL);  // no candidate passes
                py[q] = c[1];
                pz[q] = a.is3d ? c[2] : 0.0;
                found[q] = 0;
                vote[q] = WRITE && in && votes ? a.votes[(size_t)x[q] * kWarp + lane] : 0u;
                out[q] = WRITE && in ? a.nbr + a.off[x[q]] : nullptr;
            }
            auto pass = [&](int it, bool in, int at) {
                const int j = in ? __ldg(a.members + at) : -1;
                unsigned got[R];
                if (WRITE && votes) {
#pragma unroll
                    for (int q = 0; q < R; ++q) got[q] = __shfl_sync(kFull, vote[q], it);
                } else {
                    // the reference's test on (outer - inner); the squared differences do not depend on the order;
                    // (dx^2 + dy^2) + dz^2 with separate roundings, as the host computes it (no contraction)
                    const double *pj = a.coords + 3 * (size_t)(in ? j : 0);
                    const double jx = __ldg(pj), jy = __ldg(pj + 1), jz = a.is3d ? __ldg(pj + 2) : 0.0;
#pragma unroll
                    for (int q = 0; q < R; ++q) {
                        const double dx = px[q] - jx, dy = py[q] - jy, dz = pz[q] - jz;
                        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                        got[q] = __ballot_sync(kFull, in && j != x[q] && d2 <= a.r2 + a.r2tol);
                        if (!WRITE && lane == it) vote[q] = got[q];
                    }
                }
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    if (WRITE && (got[q] >> lane & 1u)) out[q][found[q] + __popc(got[q] & before)] = j + a.id_base;
                    found[q] += __popc(got[q]);
                }
            };
            int it = 0;
            if (by_cell) {
                for (int k = 0; k < ncell; ++k) {
                    const int b = __shfl_sync(kFull, start, k), c = __shfl_sync(kFull, count, k);
                    for (int m = lane; m - lane < c; m += kWarp) pass(it++, m < c, b + m);
                }
            } else {
                for (int m = lane; m - lane < total; m += kWarp) {
                    int k = 0;  // the last cell that starts at or before m
#pragma unroll
                    for (int h = kWarp / 2; h > 0; h >>= 1)
                        if (s_first[w][k + h] <= m) k += h;
                    pass(it++, m < total, s_start[w][k] + m - s_first[w][k]);
                }
            }
            if (!WRITE) {
#pragma unroll
                for (int q = 0; q < R; ++q)
                    if (q >= r && q < r1) {
                        if (votes) a.votes[(size_t)x[q] * kWarp + lane] = vote[q];
                        if (lane == 0) a.fcount[x[q]] = found[q];
                    }
            }
            __syncwarp();
        }
    }
}

cudaError_t launch_fam_cells(const FamArgs &a, cudaStream_t s) {
    const int g = (int)((a.n + 255) / 256 < 148 * 16 ? (a.n + 255) / 256 : 148 * 16);
    fam_cells_kernel<<<g > 0 ? g : 1, 256, 0, s>>>(a);
    return cudaGetLastError();
}
cudaError_t launch_fam_members(const FamArgs &a, cudaStream_t s) {
    const int g = (int)((a.n + 255) / 256 < 148 * 16 ? (a.n + 255) / 256 : 148 * 16);
    fam_members_kernel<<<g > 0 ? g : 1, 256, 0, s>>>(a);
    fam_order_members_kernel<<<g > 0 ? g : 1, 256, 0, s>>>(a);
    return cudaGetLastError();
}
cudaError_t launch_fam_partners(const FamArgs &a, bool write, cudaStream_t s) {
    const int per = 4 * kFamRun, g = (int)((a.n + per - 1) / per < 148 * 64 ? (a.n + per - 1) / per : 148 * 64);
    if (write) fam_partners_kernel<true><<<g > 0 ? g : 1, 128, 0, s>>>(a);
    else fam_partners_kernel<false><<<g > 0 ? g : 1, 128, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace pxb
