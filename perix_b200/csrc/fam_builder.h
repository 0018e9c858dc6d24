// Device family build (k_families.cu) in two phases, shared by pxb_set_geometry_points and pxb_batch_set_points.
#pragma once

#include <vector>

#include "k_kernels.h"
#include "pxb_context.h"

namespace pxb {

// count(): cells, members, candidate counts -> host offsets hoff[n+1], largest family, bond total.
// fill(): the families in the reference's order, written 0-based (+ id_base) at nbr_d[off_d[x] + k].
// The device temporaries live until the builder is destroyed; fill() needs the count() of the same builder.
class FamBuilder {
public:
    int count(pxb_ctx *c, int n, bool is3d, const double *coords_host, double radius, std::vector<int> &hoff,
              int &maxf, long long &tot);
    int fill(pxb_ctx *c, const int *off_d, int *nbr_d, int id_base);
    const double *coords_d() const { return coords_.as<double>(); }
    const int *offsets_d() const { return off_.as<int>(); }  // hoff on the device

private:
    FamArgs a_;
    DevBuf coords_, keys_, cminid_, cstart_, cfill_, members_, cell_of_, cxyz_, fcount_, votes_, off_, bsum_;
};

}  // namespace pxb
