// Top levels of the substitution sweeps in one cluster-resident kernel.
//
// k_top walks the upper levels (1-16 vectors each) inside one thread-block
// cluster per system: forward levels fwd_lo .. K-1 (ascending), then backward
// levels K-1 .. bwd_lo (descending), task t of a level on cluster block t mod C,
// with a cluster barrier (arrive.release / wait.acquire) between two levels.
// The arithmetic is the per-level kernels' own (sweep_rows_body; the vectors
// are read through L2, where other blocks of the cluster wrote them), so the
// results are bit-identical to theirs.
//
// Opt-in (SOCU_TOP_SWEEP=1): the per-level launches of a CUDA graph with
// programmatic dependent launch are faster, since a level's launch and block
// loads overlap the kernel before it.
//
// The cluster barrier is the hardware barrier: every block of a cluster runs
// the same sequence of barriers (one per level but the last, whether or not
// it has a task there), so none can wait for a block that left.
#pragma once

#include "sweep_rows.cuh"

namespace socu {

constexpr int kTopMaxLevels = 12;

// Levels of one k_top launch.  fl[i]: forward level fwd_lo + i; bl[i]: backward level bwd_lo + i.
struct TopLevels {
  Level fl[kTopMaxLevels];
  Level bl[kTopMaxLevels];
  int fwd_lo, fwd_n;   // forward levels fwd_lo .. fwd_lo + fwd_n - 1 (fwd_n = 0: none)
  int bwd_lo, bwd_n;   // backward levels bwd_lo + bwd_n - 1 .. bwd_lo (bwd_n = 0: none)
};

__device__ __forceinline__ unsigned cluster_ctarank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}

__device__ __forceinline__ unsigned cluster_nctarank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
  return r;
}

template <typename T, int NT, bool INV>
__global__ void __launch_bounds__(32 * NT) k_top(Problem<T> p, const __grid_constant__ TopLevels tl) {
  const int C = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
  const int b = blockIdx.x / C;
  if (!p.active(b)) return;   // the whole cluster (one instance) leaves together
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_wait();
  pdl_trigger();
  for (int li = 0; li < tl.fwd_n; ++li) {
    const Level& L = tl.fl[li];
    for (int t = rank; t < sweep_tasks<kModeForward>(p.N, L); t += C) {
      __syncthreads();
      sweep_rows_body<T, NT, false, kModeForward, INV, true, false>(BlockGroup{}, p, L, b, t, smem_raw, kWaitNone);
    }
    if (li + 1 < tl.fwd_n || tl.bwd_n > 0) {
      cluster_arrive();
      cluster_wait();
    }
  }
  for (int li = tl.bwd_n - 1; li >= 0; --li) {
    const Level& L = tl.bl[li];
    for (int t = rank; t < L.d; t += C) {
      __syncthreads();
      sweep_rows_body<T, NT, false, kModeBackward, INV, true, false>(BlockGroup{}, p, L, b, t, smem_raw, kWaitNone);
    }
    if (li > 0) {
      cluster_arrive();
      cluster_wait();
    }
  }
}

// k_top exists for blocks up to 64, in three sizes
__host__ __device__ inline int top_nt(int n) { return n <= 16 ? 2 : (n <= 32 ? 4 : 8); }
__host__ __device__ inline long long smem_top_bytes(int n, bool inv) { return smem_sweep_rows_bytes(8 * top_nt(n), inv); }

// Sweep kernels by op, block size and inverse-carrying factors (sweeps_f32.cu,
// sweeps_f64.cu: one translation unit per type).
template <typename T>
using SweepFn = void (*)(Problem<T>, Level, int, int);
template <typename T>
using TopFn = void (*)(Problem<T>, TopLevels);
template <typename T>
SweepFn<T> sweep_kernel(SweepMode mode, int n, bool full, bool inv);
template <typename T>
TopFn<T> top_sweep_kernel(int n, bool inv);

template <typename T, int NT, bool FULL>
inline SweepFn<T> sweep_kernel_nt(SweepMode mode, bool inv) {
  if (mode == kModePull) return k_sweep_rows<T, NT, FULL, kModePull, true>;
  if constexpr (NT <= 8) {   // factors carry inverses up to n = 64
    if (inv) {
      if (mode == kModeForward) return k_sweep_rows<T, NT, FULL, kModeForward, true>;
      return k_sweep_rows<T, NT, FULL, kModeBackward, true>;
    }
  }
  if (mode == kModeForward) return k_sweep_rows<T, NT, FULL, kModeForward, false>;
  return k_sweep_rows<T, NT, FULL, kModeBackward, false>;
}

#define SOCU_SWEEP_KERNELS(T)                                                              \
  template <>                                                                              \
  SweepFn<T> sweep_kernel<T>(SweepMode mode, int n, bool full, bool inv) {                 \
    switch (rows_nt(n)) {                                                                  \
      case 1: return full ? sweep_kernel_nt<T, 1, true>(mode, inv) : sweep_kernel_nt<T, 1, false>(mode, inv); \
      case 2: return full ? sweep_kernel_nt<T, 2, true>(mode, inv) : sweep_kernel_nt<T, 2, false>(mode, inv); \
      case 3: return full ? sweep_kernel_nt<T, 3, true>(mode, inv) : sweep_kernel_nt<T, 3, false>(mode, inv); \
      case 4: return full ? sweep_kernel_nt<T, 4, true>(mode, inv) : sweep_kernel_nt<T, 4, false>(mode, inv); \
      case 5: return full ? sweep_kernel_nt<T, 5, true>(mode, inv) : sweep_kernel_nt<T, 5, false>(mode, inv); \
      case 6: return full ? sweep_kernel_nt<T, 6, true>(mode, inv) : sweep_kernel_nt<T, 6, false>(mode, inv); \
      case 7: return full ? sweep_kernel_nt<T, 7, true>(mode, inv) : sweep_kernel_nt<T, 7, false>(mode, inv); \
      case 8: return full ? sweep_kernel_nt<T, 8, true>(mode, inv) : sweep_kernel_nt<T, 8, false>(mode, inv); \
      case 10: return full ? sweep_kernel_nt<T, 10, true>(mode, inv) : sweep_kernel_nt<T, 10, false>(mode, inv); \
      case 12: return full ? sweep_kernel_nt<T, 12, true>(mode, inv) : sweep_kernel_nt<T, 12, false>(mode, inv); \
      case 14: return full ? sweep_kernel_nt<T, 14, true>(mode, inv) : sweep_kernel_nt<T, 14, false>(mode, inv); \
      default: return full ? sweep_kernel_nt<T, 16, true>(mode, inv) : sweep_kernel_nt<T, 16, false>(mode, inv); \
    }                                                                                      \
  }                                                                                        \
  template <>                                                                              \
  TopFn<T> top_sweep_kernel<T>(int n, bool inv) {                                          \
    switch (top_nt(n)) {                                                                   \
      case 2: return inv ? k_top<T, 2, true> : k_top<T, 2, false>;                         \
      case 4: return inv ? k_top<T, 4, true> : k_top<T, 4, false>;                         \
      default: return inv ? k_top<T, 8, true> : k_top<T, 8, false>;                        \
    }                                                                                      \
  }

template <> SweepFn<float> sweep_kernel<float>(SweepMode, int, bool, bool);
template <> SweepFn<double> sweep_kernel<double>(SweepMode, int, bool, bool);
template <> TopFn<float> top_sweep_kernel<float>(int, bool);
template <> TopFn<double> top_sweep_kernel<double>(int, bool);

}  // namespace socu
