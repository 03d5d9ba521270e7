// Instantiations: ArithFast, the default shapes of the plans' forward transforms
// (BNTT_PLAN_SHAPES_*), compiled once per part (BNTT_PART).
#include "ntt_kernels.cuh"

namespace bntt {
#define BNTT_ADD(M, LOGR, TPC, MAP, MINB, SRC, USE) \
  v.push_back(BNTT_SUBK_FN(M, LOGR, TPC, MAP, ArithFast, MINB, (k_ntt_sub<M, LOGR, TPC, MAP, ArithFast, MINB, SRC>), USE));
#define BNTT_OF_PART(p) \
  void append_fast_plan_##p(std::vector<SubKernel>& v) { BNTT_PLAN_SHAPES_##p(BNTT_ADD) }
#define BNTT_THE_PART(p) BNTT_OF_PART(p)
BNTT_THE_PART(BNTT_PART)
}  // namespace bntt
