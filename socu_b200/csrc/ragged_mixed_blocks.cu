// Mixed-precision instantiation of the ragged-batch solver, block workers.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<float, kRgRefine, true>())(RgArgs<float>) {
  return k_ragged<float, kRgRefine, true>;
}
}  // namespace socu
