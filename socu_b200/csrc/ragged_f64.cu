// double instantiation of the ragged-batch solver.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<double, kRgPlain>())(RgArgs<double>) {
  return k_ragged<double, kRgPlain>;
}
}  // namespace socu
