// iface_host.h - the interface misfit and Gauss-Newton product of an inversion
// on host arrays (invert.cpp): what stays the same over the iterations (column
// densities, stations, data) is uploaded once, and an evaluation moves only the
// depths in and the gradient out, through pinned buffers of the context.
#pragma once

#include "../../include/ztm_grav.h"

struct IfaceHost {  // host arrays of one entry per column, owned by the context
  double* depth;    // in: column tops (m)
  double* v;        // in: direction of a Gauss-Newton product (m)
  double* g;        // out: gradient or product, per metre
};

// Uploads the constant arrays and hands out the buffers (valid until the next
// begin on this context).
int ztm_iface_host_begin(ztm_ctx* c, const ztm_imesh* mesh, const double* rho, int ns,
                         const double* sxyz, const double* data, IfaceHost* h);
// Misfit of `depth` and its depth gradient: started, and waited for (in `g`).
int ztm_iface_host_start(ztm_ctx* c, const ztm_imesh* mesh, int ns, const ztm_opts* o);
int ztm_iface_host_wait(ztm_ctx* c, const ztm_imesh* mesh, int ns, double* misfit);
// J^T J `v` at `depth` in `g`, J the depth derivative of the forward.
int ztm_iface_host_product(ztm_ctx* c, const ztm_imesh* mesh, int ns, const ztm_opts* o);
