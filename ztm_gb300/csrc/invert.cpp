// invert.cpp - nonlinear interface (Moho depth) inversion driven through the
// C ABI: every iteration runs the forward and the adjoint on the GPU
// and the optimiser on the host.
//
// Objective, with m = depth in km (column tops) and r = gz(m) - data:
//   phi(m) = 0.5 |r|^2 + 0.5 * lambda * sum over neighbouring columns of
//            (m_i - m_j)^2            (first-order Tikhonov smoothing)
// minimised by L-BFGS (two-loop recursion, history 8) with a backtracking
// Armijo line search (ztm_invert_interface), or by Gauss-Newton with
// conjugate-gradient inner solves whose Hessian products are one J v
// (ztm_gfm_interface_jvp) and one J^T w (the depth adjoint) each
// (ztm_invert_interface_gn); depths kept inside [0, -z_base] by projection.
//
// The reference's optimiser is a damped Gauss-Newton (Levenberg-Marquardt)
// over a grid of damping factors (TFM.cpp:155-167) whose gravity Jacobian
// columns come from one full forward per parameter (TFM.cpp:124-135); the
// adjoint gradient replaces those columns, so an iteration costs one
// forward and one adjoint whatever the number of depth parameters.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "iface_host.h"

namespace {

struct Problem {
  ztm_ctx* ctx;
  const ztm_imesh* mesh;
  int ns;
  double lambda;
  ztm_opts opts;
  int nx, ny;
  IfaceHost io;
};

// Sums run in index order: the iterations can turn a last bit into 1e-8 of the
// result, and runs are to repeat those of earlier versions.
double dot(const double* a, const double* b, size_t n) {
  double s = 0.0;
  for (size_t i = 0; i < n; i++) s += a[i] * b[i];
  return s;
}
// d = (d - a y) scale, and the new d . z (the sum's chain of adds hides the rest)
double step_dot(size_t n, double* __restrict d, double a, const double* __restrict y, double scale,
                const double* __restrict z) {
  double s = 0.0;
  for (size_t i = 0; i < n; i++) {
    const double v = (d[i] - a * y[i]) * scale;
    d[i] = v;
    s += v * z[i];
  }
  return s;
}
double dot(const std::vector<double>& a, const std::vector<double>& b) {
  return dot(a.data(), b.data(), a.size());
}

// out = 1000 g + lambda L x: a gradient per metre to one per km plus the
// smoothing term's (graph Laplacian of the column grid, first-order differences),
// a row at a time.
void add_smoothing(const Problem& P, const double* x, const double* g, double* out) {
  const double lam = P.lambda;
  const int nx = P.nx;
  for (int iy = 0; iy < P.ny; iy++) {
    const size_t r = (size_t)nx * iy;
    const double *m = x + r, *up = m - nx, *down = m + nx;
    double* o = out + r;
    for (int i = 0; i < nx; i++) o[i] = 1000.0 * g[r + i];
    if (iy > 0)
      for (int i = 0; i < nx; i++) o[i] -= lam * (up[i] - m[i]);
    for (int i = 1; i < nx; i++) o[i] -= lam * (m[i - 1] - m[i]);
    for (int i = 0; i + 1 < nx; i++) o[i] += lam * (m[i] - m[i + 1]);
    if (iy + 1 < P.ny)
      for (int i = 0; i < nx; i++) o[i] += lam * (m[i] - down[i]);
  }
}

// phi and its gradient (per km) at depth m (km).
int evaluate(Problem& P, const std::vector<double>& m, double* f, std::vector<double>& g,
             double* data_misfit) {
  const size_t nc = m.size();
  for (size_t c = 0; c < nc; c++) P.io.depth[c] = 1000.0 * m[c];
  if (int rc = ztm_iface_host_start(P.ctx, P.mesh, P.ns, &P.opts)) return rc;
  // the smoothing term meanwhile
  double reg = 0.0;
  for (int iy = 0; iy < P.ny; iy++) {
    const double* r = m.data() + (size_t)P.nx * iy;
    const double* q = r + P.nx;
    const bool down = iy + 1 < P.ny;
    for (int ix = 0; ix < P.nx; ix++) {
      if (ix + 1 < P.nx) reg += (r[ix] - r[ix + 1]) * (r[ix] - r[ix + 1]);
      if (down) reg += (r[ix] - q[ix]) * (r[ix] - q[ix]);
    }
  }
  double mis = 0.0;
  if (int rc = ztm_iface_host_wait(P.ctx, P.mesh, P.ns, &mis)) return rc;
  add_smoothing(P, m.data(), P.io.g, g.data());  // d/dm (km) = 1000 d/ddepth (m)
  *f = mis + 0.5 * P.lambda * reg;
  if (data_misfit) *data_misfit = mis;
  return ZTM_OK;
}

// Gauss-Newton Hessian product at depth m (km): (J^T J + lambda L) v, with J
// the depth derivative of the forward per km (one J v and one J^T w).
int gn_product(Problem& P, const std::vector<double>& m, const std::vector<double>& v,
               std::vector<double>& out) {
  const size_t nc = m.size();
  for (size_t c = 0; c < nc; c++) {
    P.io.depth[c] = 1000.0 * m[c];
    P.io.v[c] = 1000.0 * v[c];  // km -> m
  }
  if (int rc = ztm_iface_host_product(P.ctx, P.mesh, P.ns, &P.opts)) return rc;
  add_smoothing(P, v.data(), P.io.g, out.data());
  return ZTM_OK;
}

}  // namespace

extern "C" int ztm_invert_interface(ztm_ctx* ctx, const ztm_imesh* mesh, double* depth,
                                    const double* rho_col, int ns, const double* sxyz,
                                    const double* data, double lambda, int iterations,
                                    const ztm_opts* opt, double* history, int* n_done) {
  if (!ctx || !mesh || !depth || !rho_col || !sxyz || !data || ns < 1 || iterations < 0 ||
      !(lambda >= 0))
    return ZTM_ERR_ARG;
  if (opt && (opt->flags & ZTM_FLAG_DEVICE_PTRS)) return ZTM_ERR_ARG;  // host arrays only
  Problem P;
  P.ctx = ctx;
  P.mesh = mesh;
  P.ns = ns;
  P.lambda = lambda;
  memset(&P.opts, 0, sizeof P.opts);
  if (opt) P.opts = *opt;
  P.nx = mesh->nx;
  P.ny = mesh->ny;
  int rc = ztm_iface_host_begin(ctx, mesh, rho_col, ns, sxyz, data, &P.io);
  if (rc) return rc;
  const size_t nc = (size_t)mesh->nx * mesh->ny;
  const double dmax = -mesh->z_base / 1000.0;  // tops stay above the bases
  std::vector<double> m(nc), g(nc), mt(nc), gt(nc), d(nc);
  for (size_t c = 0; c < nc; c++) m[c] = std::min(std::max(depth[c] / 1000.0, 0.0), dmax);
  double f = 0.0, mis = 0.0;
  rc = evaluate(P, m, &f, g, &mis);
  if (rc) return rc;
  const int H = 8;
  // steps and gradient changes: S[p], Y[p] for p = kept.front() .. kept.back()
  std::vector<std::vector<double>> S(H), Y(H);
  std::vector<int> kept;
  double rhoh[H], alpha[H], sy[H], yy[H];
  std::vector<double> spare_s, spare_y;
  int it = 0;
  for (; it < iterations; it++) {
    if (history) history[it] = mis;
    // two-loop recursion: d = -H g; a pass over d both updates it and forms the
    // next dot product
    const int n = (int)kept.size();
    if (n) {
      d = g;
      const double gamma = sy[kept[n - 1]] / yy[kept[n - 1]];
      double sd = dot(S[kept[n - 1]], d);
      for (int k = n - 1; k >= 0; k--) {
        const int q = kept[k];
        alpha[q] = rhoh[q] * sd;
        sd = step_dot(nc, d.data(), alpha[q], Y[q].data(), k ? 1.0 : gamma,
                      k ? S[kept[k - 1]].data() : Y[q].data());
      }
      for (int k = 0; k < n; k++) {
        const int q = kept[k], z = kept[std::min(k + 1, n - 1)];
        sd = step_dot(nc, d.data(), rhoh[q] * sd - alpha[q], S[q].data(), k + 1 < n ? 1.0 : -1.0,
                      Y[z].data());
      }
    } else {
      const double gn = sqrt(dot(g, g));
      const double gamma = gn > 0 ? 1.0 / gn : 1.0;  // first step: 1 km along -g/|g|
      for (size_t i = 0; i < nc; i++) d[i] = -(g[i] * gamma);
    }
    double slope = dot(g, d);
    if (!(slope < 0)) {  // not a descent direction: restart on steepest descent
      kept.clear();
      double gn = sqrt(dot(g, g));
      if (gn == 0) break;
      for (size_t i = 0; i < nc; i++) d[i] = -g[i] / gn;
      slope = dot(g, d);
    }
    // backtracking Armijo line search with projection
    double step = 1.0, ft = 0.0, mist = 0.0;
    bool accepted = false;
    for (int ls = 0; ls < 20; ls++) {
      for (size_t i = 0; i < nc; i++) mt[i] = std::min(std::max(m[i] + step * d[i], 0.0), dmax);
      rc = evaluate(P, mt, &ft, gt, &mist);
      if (rc) return rc;
      if (ft <= f + 1e-4 * step * slope) {
        accepted = true;
        break;
      }
      step *= 0.5;
    }
    if (!accepted) break;
    // the pair in a place that is free: the oldest's once there are H
    int p = kept.size() < (size_t)H ? 0 : kept[0];
    if (kept.size() < (size_t)H)
      while (std::find(kept.begin(), kept.end(), p) != kept.end()) p++;
    spare_s.resize(nc);
    spare_y.resize(nc);
    double *s = spare_s.data(), *y = spare_y.data();
    for (size_t i = 0; i < nc; i++) s[i] = mt[i] - m[i];
    for (size_t i = 0; i < nc; i++) y[i] = gt[i] - g[i];
    double s_y = 0.0, ss = 0.0, y2 = 0.0;
    for (size_t i = 0; i < nc; i++) {
      s_y += s[i] * y[i];
      ss += s[i] * s[i];
      y2 += y[i] * y[i];
    }
    if (s_y > 1e-12 * sqrt(ss * y2)) {
      S[p].swap(spare_s);
      Y[p].swap(spare_y);
      rhoh[p] = 1.0 / s_y;
      sy[p] = s_y;
      yy[p] = y2;
      if (kept.size() == (size_t)H) kept.erase(kept.begin());
      kept.push_back(p);
    }
    m.swap(mt);
    g.swap(gt);
    f = ft;
    mis = mist;
  }
  if (history) history[it] = mis;
  if (n_done) *n_done = it;
  for (size_t c = 0; c < nc; c++) depth[c] = 1000.0 * m[c];
  return ZTM_OK;
}

// Gauss-Newton with conjugate-gradient inner solves: each iteration solves
// (J^T J + lambda L) d = -g for the step by at most cg_iterations CG steps
// (one J v and one J^T w on the GPU per step, J never formed), then takes
// the projected step with a backtracking line search on phi.  Same objective,
// units, bounds and history as ztm_invert_interface.
extern "C" int ztm_invert_interface_gn(ztm_ctx* ctx, const ztm_imesh* mesh, double* depth,
                                       const double* rho_col, int ns, const double* sxyz,
                                       const double* data, double lambda, int iterations,
                                       int cg_iterations, const ztm_opts* opt, double* history,
                                       int* n_done) {
  if (!ctx || !mesh || !depth || !rho_col || !sxyz || !data || ns < 1 || iterations < 0 ||
      cg_iterations < 1 || !(lambda >= 0))
    return ZTM_ERR_ARG;
  if (opt && (opt->flags & ZTM_FLAG_DEVICE_PTRS)) return ZTM_ERR_ARG;  // host arrays only
  Problem P;
  P.ctx = ctx;
  P.mesh = mesh;
  P.ns = ns;
  P.lambda = lambda;
  memset(&P.opts, 0, sizeof P.opts);
  if (opt) P.opts = *opt;
  P.nx = mesh->nx;
  P.ny = mesh->ny;
  int rc = ztm_iface_host_begin(ctx, mesh, rho_col, ns, sxyz, data, &P.io);
  if (rc) return rc;
  const size_t nc = (size_t)mesh->nx * mesh->ny;
  const double dmax = -mesh->z_base / 1000.0;
  std::vector<double> m(nc), g(nc), mt(nc), gt(nc), x(nc), r(nc), p(nc), Ap(nc);
  for (size_t c = 0; c < nc; c++) m[c] = std::min(std::max(depth[c] / 1000.0, 0.0), dmax);
  double f = 0.0, mis = 0.0;
  rc = evaluate(P, m, &f, g, &mis);
  if (rc) return rc;
  int it = 0;
  for (; it < iterations; it++) {
    if (history) history[it] = mis;
    // CG on (J^T J + lambda L) x = -g from x = 0
    std::fill(x.begin(), x.end(), 0.0);
    for (size_t i = 0; i < nc; i++) r[i] = -g[i];
    p = r;
    double rr = dot(r, r);
    const double rr0 = rr;
    if (rr0 == 0.0) break;
    for (int k = 0; k < cg_iterations; k++) {
      if ((rc = gn_product(P, m, p, Ap))) return rc;
      const double pAp = dot(p, Ap);
      if (!(pAp > 0)) break;
      const double alpha = rr / pAp;
      for (size_t i = 0; i < nc; i++) {
        x[i] += alpha * p[i];
        r[i] -= alpha * Ap[i];
      }
      const double rr1 = dot(r, r);
      if (rr1 <= 1e-12 * rr0) break;
      const double beta = rr1 / rr;
      rr = rr1;
      for (size_t i = 0; i < nc; i++) p[i] = r[i] + beta * p[i];
    }
    if (dot(x, g) >= 0) {  // not a descent step (CG broke down at once): steepest descent
      const double gn = sqrt(dot(g, g));
      for (size_t i = 0; i < nc; i++) x[i] = -g[i] / gn;
    }
    // projected step with backtracking
    double step = 1.0, ft = 0.0, mist = 0.0;
    bool accepted = false;
    for (int ls = 0; ls < 20; ls++) {
      for (size_t i = 0; i < nc; i++) mt[i] = std::min(std::max(m[i] + step * x[i], 0.0), dmax);
      if ((rc = evaluate(P, mt, &ft, gt, &mist))) return rc;
      if (ft < f) {
        accepted = true;
        break;
      }
      step *= 0.5;
    }
    if (!accepted) break;
    m.swap(mt);
    g.swap(gt);
    f = ft;
    mis = mist;
  }
  if (history) history[it] = mis;
  if (n_done) *n_done = it;
  for (size_t c = 0; c < nc; c++) depth[c] = 1000.0 * m[c];
  return ZTM_OK;
}
