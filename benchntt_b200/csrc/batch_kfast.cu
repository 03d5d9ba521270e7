// batch_kfast.cu -- the persistent batch kernel with ArithFast, one per element
// layout.
#include "batch_dev.cuh"

namespace bntt {
const void* batch_kernel_fast(int layout) {
  return layout == LAYOUT_HILO ? (const void*)&k_batch<ArithFast, LAYOUT_HILO>
                               : (const void*)&k_batch<ArithFast, LAYOUT_U128>;
}
}  // namespace bntt
