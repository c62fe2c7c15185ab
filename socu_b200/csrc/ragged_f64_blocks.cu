// double instantiation of the ragged-batch solver, block workers.
#include "ragged.cuh"

namespace socu {
template <>
void (*ragged_kernel<double, kRgPlain, true>())(RgArgs<double>) {
  return k_ragged<double, kRgPlain, true>;
}
}  // namespace socu
