// Instantiations: ArithFast, the default shapes of the plans' forward transforms
// (BNTT_PLAN_SHAPES).
#include "ntt_kernels.cuh"

namespace bntt {
void append_fast_plan(std::vector<SubKernel>& v) {
#define BNTT_ADD(M, LOGR, TPC, MAP, MINB, SRC, USE) \
  v.push_back(BNTT_SUBK_FN(M, LOGR, TPC, MAP, ArithFast, MINB, (k_ntt_sub<M, LOGR, TPC, MAP, ArithFast, MINB, SRC>), USE));
  BNTT_PLAN_SHAPES(BNTT_ADD)
#undef BNTT_ADD
}
}  // namespace bntt
