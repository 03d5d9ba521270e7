// Instantiations: ArithFast, interleaved sub-transforms (HBM passes whose
// elements are strided; TPC adjacent columns per CTA keep loads coalesced).
#include "ntt_kernels.cuh"

namespace bntt {
void append_fast_il(std::vector<SubKernel>& v) {
  using A = ArithFast;
  v.push_back(BNTT_SUBK(5, 4, 8, MAP_INTERLEAVED, A));
  v.push_back(BNTT_SUBK(6, 4, 8, MAP_INTERLEAVED, A));
  v.push_back(BNTT_SUBK(7, 4, 8, MAP_INTERLEAVED, A));
  // 4 elements per thread, 4 resident CTAs per SM, 2^(10 - M) adjacent columns
  // (that of 7 stages is a default shape)
  v.push_back(BNTT_SUBK_B(5, 2, 32, MAP_INTERLEAVED, A, 4));
  v.push_back(BNTT_SUBK_B(6, 2, 16, MAP_INTERLEAVED, A, 4));
}
}  // namespace bntt
