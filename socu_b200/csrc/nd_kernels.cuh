// Per-level kernels of the nested-dissection block-tridiagonal Cholesky.
//
// One factor level l (stride s) is two launches, all deterministic (no
// floating-point atomics, every output block has exactly one writer):
//   node      (k_node_rows, node_rows.cuh) C_i = chol(L_i) in place
//             (socu: potrf K2, block_tridiag_solver.py:197-216) fused with
//             the solves against C_i of the node's vectors:
//               rows of the right slot     -> F = E[o_l+i/s] C_i^{-T}   (K3 trsm_rltn, :219-248)
//               columns of the left slot   -> G = C_i^{-1} E[o_l+(i-s)/s] (K4 trsm_llnn, :251-279)
//               columns of y_i (factor_and_solve) -> y_i <- C_i^{-1} y_i (:108-110)
//   update    (k_update_rows, update_rows.cuh)
//             target j = 2 s u - 1 (owner computes; the reference uses
//             atomics here, K5/K6 :282-342)
//                 L_j -= F_{j-s} F_{j-s}^T + G_{j+s}^T G_{j+s}
//             fill-in for nodes with both neighbours (K7, :345-377)
//                 E[o_{l+1} + t - 1] -= F_t G_t
// Substitution sweeps (K9-K16, :425-736), reading only lower(L_i):
//   forward        levels ascending, one launch per level: each vector pulls
//                  the previous level's coupling updates
//                  y_j -= F_{j-s/2} y_{j-s/2} + G_{j+s/2}^T y_{j+s/2} and the
//                  level's nodes then solve y_i <- C_i^{-1} y_i
//   backward       levels descending: x_i -= F_i^T x_{i+s} + G_i x_{i-s};
//                  x_i <- C_i^{-T} x_i
// (k_sweep_rows, sweep_rows.cuh)
#pragma once

#include "nd_device.cuh"

namespace socu {

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline int min_i(int a, int b) { return a < b ? a : b; }

// leading dimension of a block in shared memory (elements)
__host__ __device__ inline int gemm_ld(int n, int es) { return es == 8 ? ((n + 15) / 16) * 16 + 4 : n + 1; }

// cp.async groups: close the group of copies issued so far / wait until at
// most one group is still in flight
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// info reset before a factor: 0 for every batch entry
static __global__ void k_info_reset(int* info, int B) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < B; b += gridDim.x * blockDim.x) info[b] = 0;
}

// Output blocks of one update level per instance: N / 2s targets (s is a power of two), then the
// fill-in blocks.
__host__ __device__ inline int update_targets(int N, const Level& lv) {
#ifdef __CUDA_ARCH__
  return N >> __ffs(lv.s);
#else
  return N / (2 * lv.s);
#endif
}
__host__ __device__ inline int update_blocks(int N, const Level& lv) { return update_targets(N, lv) + lv.d - 1; }

}  // namespace socu
