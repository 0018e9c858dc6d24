// Host side of the device family build (see k_families.cu and fam_builder.h).
#include <algorithm>
#include <limits>
#include <string>
#include <vector>

#include "fam_builder.h"

namespace pxb {

int FamBuilder::count(pxb_ctx *c, int n, bool is3d, const double *coords_host, double radius, std::vector<int> &hoff,
                      int &maxf, long long &tot) {
    FamArgs &a = a_;
    a = FamArgs{};
    a.n = n;
    a.is3d = is3d ? 1 : 0;
    for (int d = 0; d < 3; ++d) a.lo[d] = std::numeric_limits<double>::max();
    for (int i = 0; i < n; ++i)
        for (int d = 0; d < 3; ++d) a.lo[d] = std::min(a.lo[d], coords_host[3 * (size_t)i + d]);
    if (!is3d) a.lo[2] = 0.0;
    a.radius = radius;
    a.r2 = radius * radius;
    a.r2tol = 64.0 * std::numeric_limits<double>::epsilon() * a.r2;
    unsigned slots = 1024;
    while (slots < 2u * (unsigned)n && slots < (1u << 31)) slots <<= 1;
    a.mask = slots - 1;
    cudaStream_t s = c->stream;
    PXB_TRY(pool_upload(c, coords_, coords_host, sizeof(double) * 3 * (size_t)n));
    PXB_TRY(pool_alloc(c, keys_, sizeof(unsigned long long) * slots));
    PXB_CUDA_TRY(cudaMemsetAsync(keys_.p, 0xff, keys_.bytes, s));
    PXB_TRY(pool_alloc(c, cminid_, sizeof(int) * slots));
    PXB_CUDA_TRY(cudaMemsetAsync(cminid_.p, 0x7f, cminid_.bytes, s));
    PXB_TRY(pool_alloc(c, cfill_, 2 * sizeof(int) * slots + sizeof(FamTotals)));  // counts, fill levels, totals: zeroed
    PXB_CUDA_TRY(cudaMemsetAsync(cfill_.p, 0, cfill_.bytes, s));
    PXB_TRY(pool_alloc(c, cstart_, sizeof(int) * ((size_t)slots + 1)));
    PXB_TRY(pool_alloc(c, members_, 2 * sizeof(int) * (size_t)n));
    PXB_TRY(pool_alloc(c, cell_of_, sizeof(int) * (size_t)n));
    PXB_TRY(pool_alloc(c, cxyz_, sizeof(int) * 3 * (size_t)n));
    PXB_TRY(pool_alloc(c, votes_, 32 * sizeof(unsigned) * (size_t)n));
    PXB_TRY(pool_alloc(c, fcount_, sizeof(int) * (size_t)n));
    PXB_TRY(pool_alloc(c, off_, sizeof(int) * ((size_t)n + 1)));
    PXB_TRY(pool_alloc(c, bsum_, sizeof(long long) * (size_t)std::max(scan_blocks((int)slots), scan_blocks(n))));
    a.coords = coords_.as<double>();
    a.keys = keys_.as<unsigned long long>();
    a.tot = cfill_.as<FamTotals>();
    a.ccount = reinterpret_cast<int *>(a.tot + 1);
    a.cfill = a.ccount + slots;
    a.cminid = cminid_.as<int>();
    a.cstart = cstart_.as<int>();
    a.unsorted = members_.as<int>();
    a.members = a.unsorted + n;
    a.cell_of = cell_of_.as<int>();
    a.cxyz = cxyz_.as<int>();
    a.fcount = fcount_.as<int>();
    a.votes = votes_.as<unsigned>();
    PXB_CUDA_TRY(launch_fam_cells(a, s));
    PXB_CUDA_TRY(launch_scan((int)slots, a.ccount, bsum_.as<long long>(), &a.tot->members, a.cstart, &a.tot->maxcell, s));
    PXB_CUDA_TRY(launch_fam_members(a, s));
    PXB_CUDA_TRY(launch_fam_partners(a, false, s));
    PXB_CUDA_TRY(launch_scan(n, a.fcount, bsum_.as<long long>(), &a.tot->bonds, off_.as<int>(), &a.tot->maxfam, s));
    FamTotals t{};
    hoff.resize((size_t)n + 1);
    PXB_TRY(d2h(c, &t, a.tot, sizeof(t)));
    PXB_TRY(d2h(c, hoff.data(), off_.p, sizeof(int) * ((size_t)n + 1)));
    PXB_TRY(sync(c));
    if (t.err) return fail(PXB_ERR_INVALID, "device families: cell index out of range or cell table full");
    if (t.maxcell >= kFamCell)
        return fail(PXB_ERR_UNSUPPORTED, "device families: more than " + std::to_string(kFamCell - 1) +
                                             " nodes in one cell of size radius (use pxb_families on the host)");
    if (t.bonds > std::numeric_limits<int>::max()) return fail(PXB_ERR_INVALID, "device families: more than 2^31-1 bonds");
    tot = t.bonds;
    maxf = t.maxfam;
    if (maxf > kFamMax)
        return fail(PXB_ERR_UNSUPPORTED, "device families: a family exceeds " + std::to_string(kFamMax) +
                                             " members (use pxb_families on the host)");
    return PXB_OK;
}

int FamBuilder::fill(pxb_ctx *c, const int *off_d, int *nbr_d, int id_base) {
    FamArgs &a = a_;
    a.off = off_d;
    a.nbr = nbr_d;
    a.id_base = id_base;
    PXB_CUDA_TRY(launch_fam_partners(a, true, c->stream));
    return check_launch(c, "device families");
}

}  // namespace pxb
