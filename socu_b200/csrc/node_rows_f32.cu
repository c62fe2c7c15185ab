// float instantiations of the register-row level node.
#include "node_rows.cuh"

namespace socu {
SOCU_NODE_ROWS_KERNELS(float)
}  // namespace socu
