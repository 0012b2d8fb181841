// One-CTA step kernels, stdPFC, radices up to 8 (pfc_onecta.cuh).
#include "pfc_onecta.cuh"

namespace pfc {

template <>
void* OnectaInst<kModelStd, kRadixPow2>::kernel(bool dense) {
  return dense ? (void*)onecta_step_kernel<kModelStd, kRadixPow2, 2> : (void*)onecta_step_kernel<kModelStd, kRadixPow2, 1>;
}

template <>
void* OnectaInst<kModelStd, kRadixSmall>::kernel(bool dense) {
  return dense ? (void*)onecta_step_kernel<kModelStd, kRadixSmall, 2> : (void*)onecta_step_kernel<kModelStd, kRadixSmall, 1>;
}

}  // namespace pfc
