// double instantiation of the ragged-batch solver, warp workers.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<double, kRgPlain, false>())(RgArgs<double>) {
  return k_ragged<double, kRgPlain, false>;
}
}  // namespace socu
