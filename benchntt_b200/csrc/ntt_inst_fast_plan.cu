// Instantiations: ArithFast, the default shapes of the plans' forward transforms
// (BNTT_PLAN_SHAPES).
#include "ntt_kernels.cuh"

namespace bntt {
void append_fast_plan(std::vector<SubKernel>& v) {
#define BNTT_ADD(M, LOGR, TPC, MAP, MINB, USE) v.push_back(BNTT_SUBK_U(M, LOGR, TPC, MAP, ArithFast, MINB, USE));
  BNTT_PLAN_SHAPES(BNTT_ADD)
#undef BNTT_ADD
}
}  // namespace bntt
