// double instantiations of the Schur update.
#include "update_rows.cuh"

namespace socu {
SOCU_UPDATE_ROWS_KERNELS(double)
}  // namespace socu
