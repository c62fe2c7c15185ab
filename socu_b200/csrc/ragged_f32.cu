// float instantiation of the ragged-batch solver.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<float, kRgPlain>())(RgArgs<float>) {
  return k_ragged<float, kRgPlain>;
}
}  // namespace socu
