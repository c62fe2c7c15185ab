// Mixed-precision instantiation of the ragged-batch solver.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<float, kRgRefine>())(RgArgs<float>) {
  return k_ragged<float, kRgRefine>;
}
}  // namespace socu
