// Instantiations: ArithRef (word-for-word replica of the reference multiply),
// compiled once per part (BNTT_PART; ntt_kernels.cuh).
#include "ntt_kernels.cuh"

namespace bntt {
namespace {
using A = ArithRef;

// Parts 0 to 3, the defaults: 4 elements per thread, 4 resident CTAs of 256
// threads per SM.  Its butterfly is twice as long as the fast one, so index and
// exchange instructions weigh less than resident warps (2^24 elements of 2^10:
// 598 us against 654 with 8 elements per thread; a strided pass of 6 stages 371
// against 400).  Part 4: autotuner candidates.
template <int PART>
void append(std::vector<SubKernel>& v) {
  if constexpr (PART == 0) {
    v.push_back(BNTT_SUBK_U(1, 1, 256, MAP_CONTIG, A, 1, USE_ALL));
    v.push_back(BNTT_SUBK_U(2, 2, 256, MAP_CONTIG, A, 1, USE_ALL));
    v.push_back(BNTT_SUBK_U(3, 2, 128, MAP_CONTIG, A, 4, USE_ALL));
    v.push_back(BNTT_SUBK_U(4, 2, 64, MAP_CONTIG, A, 4, USE_ALL));
    v.push_back(BNTT_SUBK_U(5, 2, 32, MAP_CONTIG, A, 4, USE_ALL));
  } else if constexpr (PART == 1) {
    v.push_back(BNTT_SUBK_U(6, 2, 16, MAP_CONTIG, A, 4, USE_ALL));
    v.push_back(BNTT_SUBK_U(7, 2, 8, MAP_CONTIG, A, 4, USE_ALL));
    v.push_back(BNTT_SUBK_U(8, 2, 4, MAP_CONTIG, A, 4, USE_ALL));
  } else if constexpr (PART == 2) {
    v.push_back(BNTT_SUBK_U(9, 2, 2, MAP_CONTIG, A, 4, USE_ALL));
    v.push_back(BNTT_SUBK_U(10, 2, 1, MAP_CONTIG, A, 4, USE_ALL));
  } else if constexpr (PART == 3) {
    v.push_back(BNTT_SUBK_U(5, 2, 32, MAP_INTERLEAVED, A, 4, USE_ALL));
    v.push_back(BNTT_SUBK_U(6, 2, 16, MAP_INTERLEAVED, A, 4, USE_ALL));
    v.push_back(BNTT_SUBK_U(7, 2, 8, MAP_INTERLEAVED, A, 4, USE_ALL));
  } else {
    v.push_back(BNTT_SUBK(3, 3, 256, MAP_CONTIG, A));
    v.push_back(BNTT_SUBK(4, 4, 128, MAP_CONTIG, A));
    v.push_back(BNTT_SUBK(5, 3, 64, MAP_CONTIG, A));
    v.push_back(BNTT_SUBK(6, 3, 32, MAP_CONTIG, A));
    v.push_back(BNTT_SUBK(7, 3, 16, MAP_CONTIG, A));
    v.push_back(BNTT_SUBK(8, 3, 8, MAP_CONTIG, A));
    v.push_back(BNTT_SUBK(9, 3, 4, MAP_CONTIG, A));
    v.push_back(BNTT_SUBK(10, 3, 2, MAP_CONTIG, A));
    v.push_back(BNTT_SUBK(5, 4, 8, MAP_INTERLEAVED, A));
    v.push_back(BNTT_SUBK(6, 4, 8, MAP_INTERLEAVED, A));
    v.push_back(BNTT_SUBK(7, 4, 8, MAP_INTERLEAVED, A));
  }
}
}  // namespace

#define BNTT_OF_PART(p) \
  void append_ref_##p(std::vector<SubKernel>& v) { append<p>(v); }
#define BNTT_THE_PART(p) BNTT_OF_PART(p)
BNTT_THE_PART(BNTT_PART)
}  // namespace bntt
