// batch_kfast.cu -- the persistent batch kernel with ArithFast, one per element
// layout.
#include "batch_dev.cuh"

namespace bntt {
template <int THREADS>
static const void* kernel_of(int layout) {
  return layout == LAYOUT_HILO ? (const void*)&k_batch<ArithFast, LAYOUT_HILO, THREADS>
                               : (const void*)&k_batch<ArithFast, LAYOUT_U128, THREADS>;
}
const void* batch_kernel_fast(int layout, int threads) {
  return threads == kBatchThreads ? kernel_of<kBatchThreads>(layout) : kernel_of<kShortThreads>(layout);
}
}  // namespace bntt
