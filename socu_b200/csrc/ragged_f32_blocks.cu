// float instantiation of the ragged-batch solver, block workers.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<float, kRgPlain, true>())(RgArgs<float>) {
  return k_ragged<float, kRgPlain, true>;
}
}  // namespace socu
