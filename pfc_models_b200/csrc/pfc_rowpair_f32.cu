#include "pfc_rowpair_inst.cuh"

namespace pfc { template struct PairInst<float>; }
