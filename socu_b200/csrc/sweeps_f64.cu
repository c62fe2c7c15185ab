// double instantiations of the sweep kernels.
#include "top_sweep.cuh"

namespace socu {
SOCU_SWEEP_KERNELS(double)
}  // namespace socu
