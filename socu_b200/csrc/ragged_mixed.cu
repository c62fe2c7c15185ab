// Mixed-precision instantiation of the ragged-batch solver, warp workers.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<float, kRgRefine, false>())(RgArgs<float>) {
  return k_ragged<float, kRgRefine, false>;
}
}  // namespace socu
