// Log PFC with an external potential and a re-optimised linear shift M (the reference's
// logpfc_extv model, models/logpfc_extv/simulation.py): the per-step decision and the
// coefficient rebuild, on the device, between the row and the column pass of a step.
//
// The reference's step (TimeStep :301-330) is ValidatePhiRange, then the ETD1 update
//   phi_hat' = A_M phi_hat + B_M (Gamma lap N_hat_M + lap V_hat),  N_M = N - M phi,
// with A_M, B_M from L_M = Gamma lap (beta (q0^2 + lap)^2 + eps + M). Because -M phi is
// linear it is folded into the coefficient of phi_hat: the column kernel applies
//   phi_hat' = phi_hat + (A_M - 1 - M Bg_M) phi_hat + Bg_M N_hat + F_M,
// Bg_M = B_M Gamma lap, F_M = B_M lap V_hat, so the row pass computes the plain clamped
// logPFC nonlinearity (plus the field's minimum and maximum) and the spectra it leaves in
// V stay those of the reference's nonlinearity without M, from which mu follows as in
// the reference (M cancels between its linear and nonlinear parts).
#include <algorithm>
#include <cmath>

#include <cuda_runtime.h>

#include "pfc_registry.h"

namespace pfc {

// The decision on the row pass's per-CTA (min, max) pairs: one CTA.
__global__ void extv_decide_kernel(const double* __restrict__ minmax, int nparts, ExtvState* st, double g) {
  __shared__ double smin[256], smax[256];
  double lo = INFINITY, hi = -INFINITY;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
    lo = fmin(lo, minmax[2 * i]);
    hi = fmax(hi, minmax[2 * i + 1]);
  }
  smin[threadIdx.x] = lo;
  smax[threadIdx.x] = hi;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      smin[threadIdx.x] = fmin(smin[threadIdx.x], smin[threadIdx.x + s]);
      smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + s]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) extv_apply(st, smin[0], smax[0], g);
}

// The rebuild, one CTA per column (kx <= m), when the decision changed M or V changed.
__global__ void extv_coef_kernel(ExtvCoefArgs a, const ExtvState* __restrict__ st) {
  if (st->changed) extv_rebuild_column(a, st->M, blockIdx.x);
}

cudaError_t launch_extv_decide(const double* minmax, int nparts, ExtvState* st, double g, cudaStream_t s) {
  extv_decide_kernel<<<1, 256, 0, s>>>(minmax, nparts, st, g);
  return cudaGetLastError();
}

cudaError_t launch_extv_coef(const ExtvCoefArgs& a, const ExtvState* st, cudaStream_t s) {
  extv_coef_kernel<<<a.m + 1, 256, 0, s>>>(a, st);
  return cudaGetLastError();
}

}  // namespace pfc
