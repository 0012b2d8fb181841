// Host side of the one-CTA step (pfc_onecta.cuh). Its kernels are in units by model and radix set:
// the driver loads a unit's code as one, at its first kernel's first use, and the twelve builds
// together took 23 ms of a process's first plan that runs one.
#include "pfc_kernels.cuh"
#include "pfc_registry.h"

namespace pfc {

namespace {

template <int MODEL>
void* pick_model(int rset, bool dense) {
  switch (rset) {
    case kRadixPow2: return OnectaInst<MODEL, kRadixPow2>::kernel(dense);
    case kRadixSmall: return OnectaInst<MODEL, kRadixSmall>::kernel(dense);
    case kRadixAll: return OnectaInst<MODEL, kRadixAll>::kernel(dense);
    default: return nullptr;
  }
}

void* pick(int model, int rset, bool dense) {
  return model == kModelLog ? pick_model<kModelLog>(rset, dense) : pick_model<kModelStd>(rset, dense);
}

}  // namespace

size_t onecta_smem_bytes(int m, int ny, int row_ld, int col_ld) {
  const size_t rows = (size_t)ny * row_ld, cols = (size_t)m * col_ld;
  return (2 * (rows > cols ? rows : cols) + (size_t)m * ny) * sizeof(cplx<double>);
}

cudaError_t onecta_allow_smem(size_t bytes, int model, int rset) {
  for (bool dense : {false, true}) {
    cudaError_t e = cudaFuncSetAttribute(pick(model, rset, dense), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

bool onecta_supported(int rset) { return rset == kRadixPow2 || rset == kRadixSmall || rset == kRadixAll; }

cudaError_t launch_onecta_step(const RowArgs<double>& ra, const ColArgs<double>& ca, const BatchBufs* table,
                               int count, long long nsteps, int model, int rset, bool dense, int threads,
                               size_t smem, cudaStream_t stream) {
  void* fn = pick(model, rset, dense);
  if (!fn) return cudaErrorInvalidValue;
  RowArgs<double> r = ra;
  ColArgs<double> c = ca;
  void* args[] = {(void*)&r, (void*)&c, (void*)&table, (void*)&nsteps};
  return cudaLaunchKernel(fn, dim3(count), dim3(threads), args, smem, stream);
}

}  // namespace pfc
