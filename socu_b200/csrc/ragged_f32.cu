// float instantiation of the ragged-batch solver, warp workers.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<float, kRgPlain, false>())(RgArgs<float>) {
  return k_ragged<float, kRgPlain, false>;
}
}  // namespace socu
