// Instantiations: the inverse transform's kernels, in the shapes of the plans'
// forward transforms (BNTT_PLAN_SHAPES_*), compiled once per part (BNTT_PART).
#include "ntt_kernels.cuh"

namespace bntt {
namespace {

// One HBM pass of the inverse on the compile-time tile (NttTile::run_inv), one
// CTA per tile, in the shapes of the forward transform:
// whole transforms of up to 2^10 points (contiguous), or one pass of a larger
// transform (interleaved for the strided passes).  `finishing` marks the
// pass that ends the transform (stage 0 inside it), which applies N^-1 from
// entry 0 of the inverse table.
template <int M, int LOGR, int TPC, int MAP, int MINB, int SRC>
__global__ void __launch_bounds__(NttTile<M, LOGR, TPC, MAP, ArithFast>::THREADS, MINB)
    k_ntt_tile_inv(SubGeom g, ModParams mp, int layout, int finishing) {
  using T = NttTile<M, LOGR, TPC, MAP, ArithFast>;
  extern __shared__ uint4 smem[];
  const int sub = T::sub_of(threadIdx.x), lane = T::lane_of(threadIdx.x);
  const uint4* scale_at = finishing ? g.tw : nullptr;
  stream_wait();
  const uint64_t sid = (uint64_t)blockIdx.x * TPC + (uint64_t)sub;
  const SubRef sr = MAP == MAP_CONTIG ? make_subref_contig<M>(g, sid) : make_subref(g, sid);
  if (layout == LAYOUT_HILO) T::template run_inv<SRC>(sr, sub, lane, smem, mp, LAYOUT_HILO, scale_at);
  else T::template run_inv<SRC>(sr, sub, lane, smem, mp, LAYOUT_U128, scale_at);
}

}  // namespace

#define BNTT_ADD(M, LOGR, TPC, MAP, MINB, SRC, USE) \
  v.push_back(BNTT_SUBK_FN(M, LOGR, TPC, MAP, ArithFast, MINB, (k_ntt_tile_inv<M, LOGR, TPC, MAP, MINB, SRC>), USE));
#define BNTT_OF_PART(p) \
  void append_inverse_##p(std::vector<SubKernel>& v) { BNTT_PLAN_SHAPES_##p(BNTT_ADD) }
#define BNTT_THE_PART(p) BNTT_OF_PART(p)
BNTT_THE_PART(BNTT_PART)
}  // namespace bntt
