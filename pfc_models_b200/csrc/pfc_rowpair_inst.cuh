// Definitions of PairInst (pfc_registry.h): included by the .cu file of each precision.
#pragma once
#include <type_traits>

#include "pfc_registry.h"
#include "pfc_rowpair.cuh"

namespace pfc {

namespace pair_detail {

// The kernels that pair_rows can ask for, with pair_ee's values per thread.
template <class T, int ROWS, int MODEL, int L>
bool row_l(int lg, PairKernel* out) {
  constexpr bool fp64 = sizeof(T) == 8, log = MODEL == kModelLog;
  if constexpr (L <= kFastMaxLogRow) {
    if (lg != L) return row_l<T, ROWS, MODEL, L + 1>(lg, out);
    if constexpr (pair_rows(fp64, L, log, 4) == ROWS || pair_rows(fp64, L, log, 8) == ROWS) {
      constexpr int EE = pair_ee(fp64, L, log);
      using S = PairSeq<(1 << L), EE>;
      static_assert(ROWS * S::TPF * PairMinBlocks<T, EE, ROWS * S::TPF>::regs <= 65536, "a CTA's registers");
      out->fn = (void*)row_step_pair<T, (1 << L), EE, ROWS, MODEL>;
      out->threads = ROWS * S::TPF;
      out->smem = (size_t)S::SLOTS * ROWS * sizeof(cplx<T>);
      out->radices.clear();
      for (int p = 0; p < S::NP; ++p) out->radices.push_back(S::radA(p));
      return true;
    }
  }
  return false;
}

}  // namespace pair_detail

template <class T>
bool PairInst<T>::row(int lg, int rows, int model, PairKernel* out) {
  using namespace pair_detail;
  if (lg < kPairMinLog) return false;
  auto pick = [&](auto r) {
    constexpr int ROWS = decltype(r)::value;
    return model == kModelLog ? row_l<T, ROWS, kModelLog, kPairMinLog>(lg, out)
                              : row_l<T, ROWS, kModelStd, kPairMinLog>(lg, out);
  };
  constexpr int RB = sizeof(T) == 4 ? 8 : 4;   // rows of a 64-byte run
  if (rows == RB) return pick(std::integral_constant<int, RB>{});
  if (rows == RB / 2) return pick(std::integral_constant<int, RB / 2>{});
  return false;
}

}  // namespace pfc
