// One-CTA step kernels, both models, radices 11 and 13 too (pfc_onecta.cuh).
#include "pfc_onecta.cuh"

namespace pfc {

template <>
void* OnectaInst<kModelStd, kRadixAll>::kernel(bool dense) {
  return dense ? (void*)onecta_step_kernel<kModelStd, kRadixAll, 2> : (void*)onecta_step_kernel<kModelStd, kRadixAll, 1>;
}

template <>
void* OnectaInst<kModelLog, kRadixAll>::kernel(bool dense) {
  return dense ? (void*)onecta_step_kernel<kModelLog, kRadixAll, 2> : (void*)onecta_step_kernel<kModelLog, kRadixAll, 1>;
}

}  // namespace pfc
