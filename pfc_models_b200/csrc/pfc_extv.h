// Log PFC with an external potential: types and device code of the per-step decision and the
// coefficient rebuild (pfc_extv.cu says what they compute).
#pragma once
#include <cuda_runtime.h>

namespace pfc {

// Log PFC with an external potential: the state of the M shift, kept in
// device memory, and the arguments of the coefficient rebuild.
struct ExtvState {
  double M, phi_min, phi_max;   // shift and the range it was optimised for
  double floor_tol, ceil_tol;   // relative tolerances of ValidatePhiRange (0.1, 0.1)
  double min_phi;               // replaces a non-positive minimum in OptimizeM
  double last_min, last_max;    // the field's range seen by the last step
  int init, changed, count;
  int v_dirty;                  // nonzero: V changed since the forcing was built
  unsigned done;                // row CTAs whose range is stored (the last one decides)
};
struct ExtvCoefArgs {
  int nx, ny, m, nyh;
  double fx, fy, gamma, beta, q0, epsilon, dt, small_z_tol;
  double2* coef;          // (A - 1 - M Bg, Bg), [kx][ky <= ny/2]
  const double2* vhat;    // rfft2 of V, (ny, m + 1) row-major
  double2* forcing;       // B lap V_hat, [kx][ky], kx <= m
};

#ifdef __CUDACC__
// ValidatePhiRange (:375-405) and OptimizeM (:332-373) on a field's range, in FP64 (one thread).
__device__ __forceinline__ void extv_apply(ExtvState* st, double lo, double hi, double g) {
  st->last_min = lo;
  st->last_max = hi;
  bool opt = !st->init;
  if (!opt) {
    const bool floor_breached = (st->phi_min - lo) / st->phi_min > st->floor_tol;
    const bool ceiling_breached = (hi - st->phi_max) / st->phi_max > st->ceil_tol;
    opt = floor_breached || ceiling_breached;
  }
  if (opt) {
    const double plo = lo > 0 ? lo : st->min_phi;
    const double nhi = g * hi * hi + hi * hi * hi + log(hi);
    const double nlo = g * plo * plo + plo * plo * plo + log(plo);
    st->M = (nhi - nlo) / (hi - plo);
    st->phi_min = plo;
    st->phi_max = hi;
    st->init = 1;
    st->count += 1;
  }
  st->changed = (opt || st->v_dirty) ? 1 : 0;
  st->v_dirty = 0;
}

// (A_M - 1 - M Bg_M, Bg_M) at (kx, ky) and the factor B_M lap of the forcing; the same
// expressions as the host build of the coefficients (kernel_etd,
// discretization/spectral/kernels.py:55-71).
__device__ __forceinline__ double2 extv_coefficient(const ExtvCoefArgs& a, double M, int kx, int ky, double& force) {
  const double twopi = 6.283185307179586;
  const int kys = (ky <= (a.ny - 1) / 2) ? ky : ky - a.ny;
  const double kyp = twopi * ((double)kys * a.fy);
  const double kxp = twopi * ((double)kx * a.fx);
  const double lap = -(kxp * kxp + kyp * kyp);
  const double t = a.q0 * a.q0 + lap;
  const double lmu = a.beta * (t * t) + a.epsilon + M;
  const double gl = a.gamma * lap;
  const double ln = gl * lmu;
  const double z = ln * a.dt;
  const double A = exp(z);
  const double B = (fabs(z) > a.small_z_tol) ? (A - 1) / ln : a.dt * (1 + z / 2 + z * z / 6);
  const double Bg = B * gl;
  force = B * lap;
  return make_double2(expm1(z) - M * Bg, Bg);
}

// The coefficients of column kx (ky <= ny/2) and its forcing F_M (every ky), rebuilt by the
// calling CTA. Out of line: it runs on the few steps that change M or V.
static __device__ __noinline__ void extv_rebuild_column(const ExtvCoefArgs& a, double M, int kx) {
  for (int ky = threadIdx.x; ky < a.ny; ky += blockDim.x) {
    double f;
    const double2 c = extv_coefficient(a, M, kx, ky, f);
    if (ky < a.nyh) a.coef[(size_t)kx * a.nyh + ky] = c;
    const double2 v = a.vhat[(size_t)ky * (a.m + 1) + kx];
    a.forcing[(size_t)kx * a.ny + ky] = make_double2(f * v.x, f * v.y);
  }
}
#endif

}  // namespace pfc
