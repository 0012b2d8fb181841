// Definitions of GenericInst (pfc_registry.h): included by the .cu file of each precision.
#pragma once
#include "pfc_mixed.cuh"
#include "pfc_registry.h"

namespace pfc {

namespace generic_detail {

// The nonlinearity only matters in the step and reduce modes; other modes use the std instance.
template <int MODE> constexpr bool row_uses_model() { return MODE == kRowStep || MODE == kRowReduce; }

template <class T, int MODE, int MODEL>
void* pick_row_model(int rset) {
  switch (rset) {
    case kRadixPow2: return (void*)mixed_row_kernel<T, MODE, MODEL, kRadixPow2>;
    case kRadixSmall: return (void*)mixed_row_kernel<T, MODE, MODEL, kRadixSmall>;
    case kRadixAll: return (void*)mixed_row_kernel<T, MODE, MODEL, kRadixAll>;
    case kRadixPow2Big: return (void*)row_kernel<T, MODE, MODEL, kRadixPow2, 1024>;
    case kRadixSmallBig: return (void*)row_kernel<T, MODE, MODEL, kRadixSmall, 1024>;
    default: return nullptr;
  }
}

template <class T, int MODE>
void* pick_row(int model, int rset) {
  if constexpr (row_uses_model<MODE>())
    if (model == kModelLog) return pick_row_model<T, MODE, kModelLog>(rset);
  return pick_row_model<T, MODE, kModelStd>(rset);
}

template <class T, int MODE>
void* pick_col(int rset) {
  // (the Parseval and export modes transform nothing)
  if constexpr (MODE == kColParseval || MODE == kColExport) {
    return (void*)col_kernel<T, MODE, kRadixPow2, kParThreads>;
  } else {
    switch (rset) {
      case kRadixPow2: return (void*)mixed_col_kernel<T, MODE, kRadixPow2>;
      case kRadixSmall: return (void*)mixed_col_kernel<T, MODE, kRadixSmall>;
      case kRadixAll: return (void*)mixed_col_kernel<T, MODE, kRadixAll>;
      case kRadixPow2Big: return (void*)col_kernel<T, MODE, kRadixPow2, 1024>;
      case kRadixSmallBig: return (void*)col_kernel<T, MODE, kRadixSmall, 1024>;
      default: return nullptr;
    }
  }
}

}  // namespace generic_detail

template <class T>
void* GenericInst<T>::row(int mode, int model, int rset) {
  using namespace generic_detail;
  switch (mode) {
    case kRowStep: return pick_row<T, kRowStep>(model, rset);
    case kRowForward: return pick_row<T, kRowForward>(model, rset);
    case kRowMaterialize: return pick_row<T, kRowMaterialize>(model, rset);
    case kRowReduce: return pick_row<T, kRowReduce>(model, rset);
    default: return nullptr;
  }
}

template <class T>
void* GenericInst<T>::col(int mode, int rset) {
  using namespace generic_detail;
  switch (mode) {
    case kColStep: return pick_col<T, kColStep>(rset);
    case kColInit: return pick_col<T, kColInit>(rset);
    case kColCombine: return pick_col<T, kColCombine>(rset);
    case kColParseval: return pick_col<T, kColParseval>(rset);
    case kColExport: return pick_col<T, kColExport>(rset);
    default: return nullptr;
  }
}

}  // namespace pfc
