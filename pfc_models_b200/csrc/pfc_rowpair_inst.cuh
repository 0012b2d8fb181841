// Definitions of PairInst (pfc_registry.h): included by the .cu file of each precision.
#pragma once
#include <cmath>

#include "pfc_registry.h"
#include "pfc_rowpair.cuh"

namespace pfc {

namespace pair_detail {

template <class T, int EE, int ROWS, int L>
constexpr bool fits() {
  // two passes or more; registers of a CTA within an SM's, its exchange buffer within 200 KB
  constexpr int threads = ROWS * (1 << L) / EE;
  if constexpr ((1 << L) < 2 * EE || threads < 32 || threads > 1024) return false;
  else
    return threads * PairMinBlocks<T, EE, threads>::regs <= 65536 &&
           (size_t)PairSeq<(1 << L), EE>::SLOTS * ROWS * sizeof(cplx<T>) <= 200 * 1024;
}

template <class T, int EE, int ROWS, int L>
bool row_l(int lg, int model, PairKernel* out) {
  if constexpr (L <= kFastMaxLogRow) {
    if (lg != L) return row_l<T, EE, ROWS, L + 1>(lg, model, out);
    if constexpr (fits<T, EE, ROWS, L>()) {
      using S = PairSeq<(1 << L), EE>;
      out->fn = model == kModelLog ? (void*)row_step_pair<T, (1 << L), EE, ROWS, kModelLog>
                                   : (void*)row_step_pair<T, (1 << L), EE, ROWS, kModelStd>;
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
bool PairInst<T>::row(int lg, int ee, int rows, int model, PairKernel* out) {
  using namespace pair_detail;
  constexpr int RB = sizeof(T) == 4 ? 8 : 4;   // rows of a 64-byte run
  if (lg < kFastMinLog || (rows != RB && rows != RB / 2)) return false;
  auto pick = [&](auto e) {
    constexpr int EE = decltype(e)::value;
    return rows == RB ? row_l<T, EE, RB, kFastMinLog>(lg, model, out) : row_l<T, EE, RB / 2, kFastMinLog>(lg, model, out);
  };
  if (ee == 8) return pick(std::integral_constant<int, 8>{});
  if (ee == 16) return pick(std::integral_constant<int, 16>{});
  if constexpr (sizeof(T) == 4)
    if (ee == 32) return pick(std::integral_constant<int, 32>{});
  return false;
}

}  // namespace pfc
