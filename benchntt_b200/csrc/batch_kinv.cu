// batch_kinv.cu -- the persistent batch kernel for inverse transforms
// (bntt_batch_run_inverse_dev).  Same work queue, items and tiles as k_batch;
// each item runs the tile's inverse network (run_inv: stages last to first
// with the plans' inverse tables), the passes of a large job run from the last
// to the first, and whatever finishes a transform -- a small tile, or pass 0
// of a large job -- multiplies by N^-1 as it stores, read from entry 0 of the
// job's inverse table (no stage uses that entry).
// Fast moduli only, like the plans' inverse.  Compiled once per part (BNTT_PART,
// batch_part).
#include "batch_dev.cuh"

namespace bntt {

namespace {

template <int M, int LOGR, int TPC, int MAP, int LY, int THREADS>
__device__ __forceinline__ void run_item_inv(const WorkItem& it, const BatchArgs& ba, uint4* smem,
                                          const ModParams& mp, int* s_flag) {
  constexpr int HELD = THREADS >> (M - LOGR);
  using T = NttTile<M, LOGR, HELD, MAP, ArithFast>;
  static_assert(T::THREADS == THREADS && TPC % HELD == 0, "tile shape");
  if (!item_wait<true>(it, ba, s_flag)) return;
  const bool finishes = it.kind == ITEM_SMALL || it.pass == 0;
#pragma unroll 1
  for (int turn = 0; turn < TPC / HELD; ++turn) {
    const int sub = T::sub_of(threadIdx.x), lane = T::lane_of(threadIdx.x);
    const SubRef sr = item_subref<M, MAP>(it, ba, turn * HELD + sub);
    if (turn > 0) T::sync();  // smem is reused
    T::template run_inv<TW_CONST>(sr, sub, lane, smem, mp, LY, finishes ? sr.tw : nullptr);
  }
  item_publish(it, ba);
}

// LY: the element layout as a constant, as in k_batch.
template <int LY, int THREADS>
__global__ void __launch_bounds__(THREADS, batch_ctas(THREADS)) k_batch_inv(BatchArgs ba, ModParams mp, int) {
  extern __shared__ uint4 smem[];
  __shared__ uint32_t s_item;
  __shared__ int s_flag;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&ba.ctl[0], 1u);
    __syncthreads();
    const uint32_t i = s_item;
    if (i >= ba.nitems) break;
    const WorkItem it = ba.items[i];
    switch (it.shape) {
#define BNTT_RUN_SHAPE(id, M, LOGR, TPC, MAP)                     \
  case id:                                                        \
    run_item_inv<M, batch_logr(LOGR, THREADS), TPC, MAP, LY, THREADS>(it, ba, smem, mp, &s_flag); \
    break;
      BNTT_BATCH_SHAPES(BNTT_RUN_SHAPE)
#undef BNTT_RUN_SHAPE
      default: break;
    }
    __syncthreads();  // smem and s_item are reused by the next item
  }
}

}  // namespace

template <>
const void* batch_kernel_inverse<BNTT_PART>() {
  return (const void*)&k_batch_inv<part_layout(BNTT_PART), part_threads(BNTT_PART)>;
}

}  // namespace bntt
