// batch_kfast.cu -- the persistent batch kernel with ArithFast, compiled once per
// part (BNTT_PART, batch_part): one element layout and one number of threads each.
#include "batch_dev.cuh"

namespace bntt {
template <>
const void* batch_kernel_fast<BNTT_PART>() {
  return (const void*)&k_batch<ArithFast, part_layout(BNTT_PART), part_threads(BNTT_PART)>;
}
}  // namespace bntt
