// One-CTA step kernels, log model, radices up to 8 (pfc_onecta.cuh).
#include "pfc_onecta.cuh"

namespace pfc {

template <>
void* OnectaInst<kModelLog, kRadixPow2>::kernel(bool dense) {
  return dense ? (void*)onecta_step_kernel<kModelLog, kRadixPow2, 2> : (void*)onecta_step_kernel<kModelLog, kRadixPow2, 1>;
}

template <>
void* OnectaInst<kModelLog, kRadixSmall>::kernel(bool dense) {
  return dense ? (void*)onecta_step_kernel<kModelLog, kRadixSmall, 2> : (void*)onecta_step_kernel<kModelLog, kRadixSmall, 1>;
}

}  // namespace pfc
