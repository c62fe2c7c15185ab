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
//   k_fwd          levels ascending, one launch per level: each vector pulls
//                  the previous level's coupling updates
//                  y_j -= F_{j-s/2} y_{j-s/2} + G_{j+s/2}^T y_{j+s/2} and the
//                  level's nodes then solve y_i <- C_i^{-1} y_i
//   k_bwd          levels descending: x_i -= F_i^T x_{i+s} + G_i x_{i-s};
//                  x_i <- C_i^{-T} x_i
#pragma once

#include "nd_device.cuh"
#include "tma.cuh"

namespace socu {

constexpr int kTile = 32;     // output tile / streamed chunk width
constexpr int kMC = 32;       // RHS columns handled per pass in the sweeps

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline int min_i(int a, int b) { return a < b ? a : b; }

// shared-memory sizes (elements) ------------------------------------------------
__host__ __device__ inline int gemm_ld(int n, int es) { return es == 8 ? ((n + 15) / 16) * 16 + 4 : n + 1; }
__host__ __device__ inline int update_ld(int k, int es) { return gemm_ld(k, es); }
// streamed (non-resident) sweeps: Y, Z1, Z2 (n x sweep_ldy) and the chunk buffer
// Cc (n x sweep_ldc >= kTile x (n + 1) for the triangular panels), dv (kTile)
__host__ __device__ inline int sweep_ldy(int mc) { return mc + 4; }
constexpr int kSweepLdc = kTile + 4;   // 4 (mod 16) doubles: conflict-free DMMA fragments

// cp.async groups: close the group of copies issued so far / wait until at
// most one group is still in flight
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
// (two chunk buffers: the next chunk's copies overlap this chunk's product)
__host__ __device__ inline long long smem_sweep_elems(int n, int m) {
  const int mc = min_i(m, kMC);
  const long long cc = 2LL * n * kSweepLdc > (long long)kTile * (n + 1) ? 2LL * n * kSweepLdc
                                                                        : (long long)kTile * (n + 1);
  return 3LL * n * sweep_ldy(mc) + cc + kTile;
}

// ---------------------------------------------------------------------------
// Inverse-first node (n <= kNodeGemmMaxN): factor L_i against the identity
// only, C W = I, so W = C^{-1} comes out of the blocked solve, then every
// other vector set is one dense GEMM with W (tensor cores for double):
//     F = R W^T      (rows of the right slot, R loaded row-major)
//     G = W Lf       (left slot)
//     y = W y        (factor_and_solve)
// R, Lf and the first y chunk are loaded together once the factor is done
// and the three GEMMs run back to back without barriers in between; results
// go from the accumulators straight to global memory.  Shared layout:
// S1 (n x ld: A/C, then R), W (n x ld), S2 (n x ld: Lf), Y (n x ldy).
// INV keeps W^T in the strict upper triangle of L_i.
// ---------------------------------------------------------------------------
constexpr int kNodeGemmMaxN = 64;
__host__ __device__ inline int node_gemm_ldy(int m) { return m > 0 ? even_ld(min_i(m, kMC)) : 0; }
// S1, W, S2 (n x ld), Y (n x ldy)
__host__ __device__ inline long long smem_node_gemm_elems(int n, int m, int es) {
  return 3LL * n * gemm_ld(n, es) + (long long)n * node_gemm_ldy(m);
}

template <typename T, bool WITH_Y, bool INV>
__device__ __forceinline__ void node_gemm_body(const Problem<T>& p, const Level& lv, int b, int t,
                                               unsigned char* smem_raw) {
  constexpr int es = sizeof(T);
  const int n = p.n, s = lv.s, i = s - 1 + 2 * s * t;
  const bool right = i + s < p.N, left = t >= 1;
  const int ld = gemm_ld(n, es);
  const int ldy = node_gemm_ldy(WITH_Y ? p.m : 0);
  T* S1 = reinterpret_cast<T*>(smem_raw);
  T* W = S1 + n * ld;
  T* S2 = W + n * ld;
  T* Y = S2 + n * ld;
  T* Li = p.Lb(b, i);
  T* R = right ? p.Eb(b, lv.oc + 2 * t) : nullptr;
  T* Lf = left ? p.Eb(b, lv.oc + 2 * t - 1) : nullptr;
  T* yi = WITH_Y ? p.Xb(b, i) : nullptr;

  async_load(S1, ld, Li, n, n, n);
  if (left) async_load(S2, ld, Lf, n, n, n);   // prefetch: S2 is untouched by the factor
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int r = e / n, c = e - r * n;
    W[r * ld + c] = r == c ? T(1) : T(0);
  }
  cp_async_wait_all();
  __syncthreads();
  // lower(S1) = C, W = C^{-1} (zeros above)
  cta_chol_solve<T, true>(S1, ld, n, W, ld, n);
  check_factor(p, b, i, S1, ld);
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int r = e / n, c = e - r * n;
    Li[e] = c <= r ? S1[r * ld + c] : (INV ? W[c * ld + r] : T(0));
  }
  const int mc0 = WITH_Y ? min_i(kMC, p.m) : 0;
  __syncthreads();
  if (right) async_load(S1, ld, R, n, n, n);
  if (WITH_Y) async_load(Y, ldy, yi, n, mc0, p.m);
  cp_async_wait_all();
  __syncthreads();
  // F[r][c] = sum_k R[r][k] W[c][k]
  if (right)
    cta_gemm<T, false, true>(n, n, n, S1, ld, W, ld, [&](int r, int c, T v) { R[(long long)r * n + c] = v; });
  // G[r][c] = sum_k W[r][k] Lf[k][c]
  if (left)
    cta_gemm<T, false, false>(n, n, n, W, ld, S2, ld, [&](int r, int c, T v) { Lf[(long long)r * n + c] = v; });
  if (WITH_Y) {
    for (int c0 = 0; c0 < p.m; c0 += kMC) {
      const int mc = min_i(kMC, p.m - c0);
      if (c0 > 0) {
        __syncthreads();
        async_load(Y, ldy, yi + c0, n, mc, p.m);
        cp_async_wait_all();
        __syncthreads();
      }
      cta_gemm<T, false, false>(n, mc, n, W, ld, Y, ldy,
                                [&](int r, int c, T v) { yi[(long long)r * p.m + c0 + c] = v; });
    }
  }
}

// info reset before a factor: 0 for every batch entry
static __global__ void k_info_reset(int* info, int B) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < B; b += gridDim.x * blockDim.x) info[b] = 0;
}

// ---------------------------------------------------------------------------
// k_update
// ---------------------------------------------------------------------------
// Whole-block update for n <= kNodeGemmMaxN: task u-1 < U updates target
// j = 2su-1 completely (all lower tiles, K = 2n), task U + t-1 forms the whole
// fill-in block of node t.  One CTA per block keeps every warp busy.
__host__ __device__ inline int update_blocks(int N, const Level& lv) { return N / (2 * lv.s) + lv.d - 1; }
// n <= 64 updates run on DMMA for both types; float rows padded to 4 (mod 32)
// words so the fragment loads hit distinct banks
__host__ __device__ inline int update_full_ld(int k, int es) { return es == 8 ? update_ld(k, es) : ((k + 3) & ~3) + 4; }
__host__ __device__ inline long long smem_update_full_elems(int n, int es) {
  const long long a = (long long)n * update_full_ld(2 * n, es);
  const long long f = 2LL * n * update_full_ld(n, es);
  return a > f ? a : f;
}

template <typename T>
__device__ __forceinline__ void update_full_body(const Problem<T>& p, const Level& lv, int b, int task,
                                                 unsigned char* smem_raw) {
  constexpr int es = sizeof(T);
  const int n = p.n, N = p.N, s = lv.s;
  const int U = N / (2 * s);
  T* Ab = reinterpret_cast<T*>(smem_raw);
  if (task < U) {
    const int u = task + 1;
    const int j = 2 * s * u - 1;
    const T* F = p.Eb(b, lv.oc + 2 * (u - 1));
    const bool hasG = j + s < N;
    const T* G = hasG ? p.Eb(b, lv.oc + 2 * u - 1) : nullptr;
    const int K = hasG ? 2 * n : n;
    const int lda = update_full_ld(2 * n, es);
    // Ab[r][k] = F[r][k], Ab[r][n+k] = G[k][r]
    async_load(Ab, lda, F, n, n, n);
    if (hasG) async_load_t(Ab + n, lda, G, n, n, n);
    cp_async_wait_all();
    __syncthreads();
    T* Lj = p.Lb(b, j);
    // DMMA for both types (float operands widened: one rounding per entry)
    warp_gemm_dmma<T, false, true, true>(n, n, K, Ab, lda, Ab, lda, [&](int r, int c, double v) {
      T* o = Lj + (long long)r * n + c;
      *o = (T)((double)*o - v);
    });
  } else {
    const int t = task - U + 1;
    const int i = s - 1 + 2 * s * t;
    if (i + s >= N) return;
    const T* F = p.Eb(b, lv.oc + 2 * t);
    const T* G = p.Eb(b, lv.oc + 2 * t - 1);
    T* X = p.Eb(b, lv.on + t - 1);
    const int ld = update_full_ld(n, es);
    T* Bb = Ab + n * ld;
    async_load(Ab, ld, F, n, n, n);
    async_load(Bb, ld, G, n, n, n);
    cp_async_wait_all();
    __syncthreads();
    warp_gemm_dmma<T, false, false>(n, n, n, Ab, ld, Bb, ld, [&](int r, int c, double v) {
      T* o = X + (long long)r * n + c;
      *o = (T)((double)*o - v);
    });
  }
}

// ---------------------------------------------------------------------------
// Sweeps.  Shared layout: Y, Z1, Z2 (n x (mc+1) each), Cc (n x (kTile+1)), dv (kTile)
// ---------------------------------------------------------------------------

// Y -= op(M1) Z1 + op(M2) Z2 with M1, M2 n x n global blocks (a null M skips
// its product), streamed through two Cc buffers in kTile chunks of the
// contraction index: the copies of chunk c + 1 are in flight while chunk c's
// product runs.  TRx: op(M)[r][k] = M[k][r].  Each chunk's product runs on the
// FP64 tensor cores (DMMA warp tiles of 16 x 32; float operands widened in
// registers, FP64 sums, one rounding per entry and chunk): with n > 64 and
// many right-hand sides these products, not the block loads, bound the sweep.
template <typename T, bool TR1, bool TR2>
__device__ void sweep_accumulate2(T* Y, const T* Z1, const T* __restrict__ M1, const T* Z2,
                                  const T* __restrict__ M2, int ldy, int mc, int n, T* Cc) {
  constexpr int ldc = kSweepLdc;
  const int per = (n + kTile - 1) / kTile;
  const int c1 = M1 ? per : 0, total = c1 + (M2 ? per : 0);
  if (total == 0) return;
  auto stage = [&](int c) {
    T* dst = Cc + (c & 1) * n * ldc;
    const bool first = c < c1;
    const T* M = first ? M1 : M2;
    const bool tr = first ? TR1 : TR2;
    const int k0 = (first ? c : c - c1) * kTile, kw = min_i(kTile, n - k0);
    if (tr)
      async_load_t(dst, ldc, M + (long long)k0 * n, kw, n, n);   // dst[r][kk] = M[k0+kk][r]
    else
      async_load(dst, ldc, M + k0, n, kw, n);                   // dst[r][kk] = M[r][k0+kk]
    cp_async_commit();
  };
  __syncthreads();
  stage(0);
  for (int c = 0; c < total; ++c) {
    if (c + 1 < total) stage(c + 1);
    else cp_async_commit();
    cp_async_wait_one();
    __syncthreads();
    const bool first = c < c1;
    const int k0 = (first ? c : c - c1) * kTile, kw = min_i(kTile, n - k0);
    const T* Z = first ? Z1 : Z2;
    warp_gemm_dmma<T, false, false>(n, mc, kw, Cc + (c & 1) * n * ldc, ldc, Z + k0 * ldy, ldy,
                                    [&](int r, int cc, double v) {
                                      T* o = Y + r * ldy + cc;
                                      *o = (T)((double)*o - v);
                                    });
    __syncthreads();
  }
}

// Y <- C^{-1} Y (lower C = lower(Lb)), blocked by kTile rows: a warp takes
// four columns at once (lane = row of the panel), so the panel elements are
// loaded once for four columns and the four substitution chains interleave.
constexpr int kSolveCols = 4;
template <typename T>
__device__ void sweep_lower_solve(T* Y, int ldy, int mc, const T* __restrict__ Lb, int n, T* Cc, T* dv) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int ldc = n + 1;  // Cc holds >= kTile * (n + 1) elements
  for (int K = 0; K < n; K += kTile) {
    const int kb = min_i(kTile, n - K);
    __syncthreads();
    async_load(Cc, ldc, Lb + (long long)K * n, kb, K + kb, n);   // rows [K,K+kb), cols [0,K+kb)
    cp_async_wait_all();
    __syncthreads();
    if (threadIdx.x < kb) dv[threadIdx.x] = T(1) / Cc[threadIdx.x * ldc + K + threadIdx.x];
    __syncthreads();
    for (int cb = warp; cb < mc; cb += nw * kSolveCols) {
      int col[kSolveCols];
      bool cv[kSolveCols];
#pragma unroll
      for (int q = 0; q < kSolveCols; ++q) {
        col[q] = cb + q * nw;
        cv[q] = col[q] < mc;
        if (!cv[q]) col[q] = cb;
      }
      T v[kSolveCols];
#pragma unroll
      for (int q = 0; q < kSolveCols; ++q) v[q] = lane < kb ? Y[(K + lane) * ldy + col[q]] : T(0);
      if (lane < kb) {
        for (int k = 0; k < K; ++k) {
          const T cm = Cc[lane * ldc + k];
#pragma unroll
          for (int q = 0; q < kSolveCols; ++q) v[q] = fma(-cm, Y[k * ldy + col[q]], v[q]);
        }
      }
      for (int j = 0; j < kb; ++j) {
        const T cj = (lane > j && lane < kb) ? Cc[lane * ldc + K + j] : T(0);
#pragma unroll
        for (int q = 0; q < kSolveCols; ++q) {
          const T yj = __shfl_sync(kFull, v[q], j) * dv[j];
          v[q] = lane == j ? yj : fma(-cj, yj, v[q]);
        }
      }
      if (lane < kb) {
#pragma unroll
        for (int q = 0; q < kSolveCols; ++q)
          if (cv[q]) Y[(K + lane) * ldy + col[q]] = v[q];
      }
    }
  }
  __syncthreads();
}

// Y <- C^{-T} Y (lower C = lower(Lb)), blocks from the bottom, four columns per warp.
template <typename T>
__device__ void sweep_upper_solve(T* Y, int ldy, int mc, const T* __restrict__ Lb, int n, T* Cc, T* dv) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  constexpr int ldc = kTile + 1;
  const int last = ((n - 1) / kTile) * kTile;
  for (int K = last; K >= 0; K -= kTile) {
    const int kb = min_i(kTile, n - K);
    __syncthreads();
    // column panel: rows [K, n), columns [K, K+kb): Cc[(k-K)][r] = C[k][K+r]
    async_load(Cc, ldc, Lb + (long long)K * n + K, n - K, kb, n);
    cp_async_wait_all();
    __syncthreads();
    if (threadIdx.x < kb) dv[threadIdx.x] = T(1) / Cc[threadIdx.x * ldc + threadIdx.x];
    __syncthreads();
    for (int cb = warp; cb < mc; cb += nw * kSolveCols) {
      int col[kSolveCols];
      bool cv[kSolveCols];
#pragma unroll
      for (int q = 0; q < kSolveCols; ++q) {
        col[q] = cb + q * nw;
        cv[q] = col[q] < mc;
        if (!cv[q]) col[q] = cb;
      }
      T v[kSolveCols];
#pragma unroll
      for (int q = 0; q < kSolveCols; ++q) v[q] = lane < kb ? Y[(K + lane) * ldy + col[q]] : T(0);
      if (lane < kb) {
        for (int k = K + kb; k < n; ++k) {
          const T cm = Cc[(k - K) * ldc + lane];
#pragma unroll
          for (int q = 0; q < kSolveCols; ++q) v[q] = fma(-cm, Y[k * ldy + col[q]], v[q]);
        }
      }
      for (int j = kb - 1; j >= 0; --j) {
        const T cj = lane < j ? Cc[j * ldc + lane] : T(0);
#pragma unroll
        for (int q = 0; q < kSolveCols; ++q) {
          const T xj = __shfl_sync(kFull, v[q], j) * dv[j];
          v[q] = lane == j ? xj : fma(-cj, xj, v[q]);
        }
      }
      if (lane < kb) {
#pragma unroll
        for (int q = 0; q < kSolveCols; ++q)
          if (cv[q]) Y[(K + lane) * ldy + col[q]] = v[q];
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Resident sweep helpers: the whole factor block and both coupling blocks of
// a node sit in shared memory (one load round), Y/Z are n x mc column chunks.
// Leading dimensions are even so every load can be vectorised.
// ---------------------------------------------------------------------------
// vector leading dimension of the resident sweeps: rows start on 16 bytes and
// every 8-column pass can read 8 elements past its first column
__host__ __device__ inline int res_ldy(int mc) { return ((mc + 3) / 4) * 4 + 4; }
// block leading dimension of the resident sweeps: rows start on 16 bytes (one
// 16-byte copy per 4 floats / 2 doubles) and 4 threads x 8 rows of a warp hit
// distinct banks in the row-major reads
__host__ __device__ inline int res_ldm(int n) { return ((n + 3) & ~3) + 4; }
// elements of one resident-sweep region, rounded so the next region starts on
// 128 bytes (TMA destinations)
__host__ __device__ inline long long res_round(long long elems, int es) {
  const long long q = 128 / es;
  return ((elems + q - 1) / q) * q;
}
// three vector regions, three block regions, dv (n) and two mbarriers; the
// 4-byte rounding is the larger, so the count covers both element sizes
__host__ __device__ inline long long smem_sweep_res_elems(int n, int m) {
  const int mc = min_i(m, kMC);
  return 3LL * res_round((long long)n * res_ldy(mc), 4) + 3LL * res_round((long long)n * res_ldm(n), 4) + n + 8;
}

// TMA use of one resident-sweep CTA: block and vector loads by the validity of
// their maps and a 128-byte aligned shared base (the same in every thread);
// initialises the two mbarriers (all threads call).
struct ResTma {
  bool blocks, vecs;
};
__device__ __forceinline__ ResTma res_tma_begin(const SweepMaps* tm, unsigned char* raw, uint64_t* bar) {
  ResTma r{false, false};
  if (tm == nullptr || (smem_addr(raw) & 127u) != 0) return r;
  r.blocks = tm->blocks != 0;
  r.vecs = tm->vecs != 0;
  if (r.blocks || r.vecs) {
    if (threadIdx.x == 0) {
      tc::mbar_init(bar, 1);
      tc::mbar_init(bar + 1, 1);
    }
    __syncthreads();
  }
  return r;
}

// Wait for this chunk's TMA copies: the blocks (first chunk) and the vectors;
// false (in every thread) if a wait ran out.
__device__ __forceinline__ bool res_tma_wait(const ResTma& tu, bool blocks_pending, uint64_t* bar, int chunk) {
  const bool okb = (tu.blocks && blocks_pending) ? tma::wait(bar, 0) : true;
  const bool okv = tu.vecs ? tma::wait(bar + 1, (unsigned)chunk & 1u) : true;
  return okb && okv;
}

// CW consecutive elements from 16-byte-aligned shared memory (8-byte for CW = 2 floats)
template <typename T, int CW>
__device__ __forceinline__ void load_cols(const T* p, T (&v)[CW]) {
  if constexpr (CW == 1) {
    v[0] = p[0];
  } else if constexpr (sizeof(T) == 4 && CW == 2) {
    const float2 a = *reinterpret_cast<const float2*>(p);
    v[0] = a.x; v[1] = a.y;
  } else if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int h = 0; h < CW / 4; ++h) {
      const float4 a = *reinterpret_cast<const float4*>(p + 4 * h);
      v[4 * h] = a.x; v[4 * h + 1] = a.y; v[4 * h + 2] = a.z; v[4 * h + 3] = a.w;
    }
  } else {
#pragma unroll
    for (int h = 0; h < CW / 2; ++h) {
      const double2 a = *reinterpret_cast<const double2*>(p + 2 * h);
      v[2 * h] = a.x; v[2 * h + 1] = a.y;
    }
  }
}

// Resident block times resident vectors, n <= 64 rows, up to kMC columns:
//   MODE 0: Yout -= M Z            M(r,k) = M[r*ldm + k]
//   MODE 1: Yout -= M^T Z          M(r,k) = M[k*ldm + r]
//   MODE 2: Yout = W^T Z           W^T(r,k) = M[r*ldm + k] for k > r, diagonal dv[r]
//   MODE 3: Yout = W Z             W(r,k) = M[k*ldm + r] for k < r, diagonal dv[r]
// (modes 2/3 read the inverse W = C^{-1} that an inverse-carrying factor keeps
// in its strict upper triangle).  Four consecutive threads share a row and
// split its contraction; each holds CW output columns in registers (CW = 8,
// 4, 2 or 1 by the column count), reads Z rows with vector loads (rows are
// 16-byte aligned, ldy from res_ldy) and the four partial rows are combined
// with two shuffles.
template <typename T, int MODE, int CW>
__device__ __forceinline__ void res_rowdot(T* Yout, const T* Z, int ldy, int mc, const T* M, int ldm, const T* dv,
                                           int n) {
  const int q = threadIdx.x & 3;
  const int nr = ((n + 7) / 8) * 8;   // whole warps iterate together (shuffles)
  for (int c0 = 0; c0 < mc; c0 += CW) {
    for (int rb = threadIdx.x >> 2; rb < nr; rb += blockDim.x >> 2) {
      const int r = rb < n ? rb : n - 1;
      T acc[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) acc[j] = T(0);
      const int k0 = MODE == 2 ? r + 1 : 0, k1 = MODE == 3 ? r : n;
#pragma unroll 4
      for (int k = k0 + q; k < k1; k += 4) {
        const T mv = (MODE == 0 || MODE == 2) ? M[r * ldm + k] : M[k * ldm + r];
        T z[CW];
        load_cols<T, CW>(Z + k * ldy + c0, z);
#pragma unroll
        for (int j = 0; j < CW; ++j) acc[j] = fma(mv, z[j], acc[j]);
      }
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        acc[j] += __shfl_xor_sync(kFull, acc[j], 1);
        acc[j] += __shfl_xor_sync(kFull, acc[j], 2);
      }
      if (rb < n) {
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          if ((j & 3) != q || c0 + j >= mc) continue;
          if (MODE <= 1)
            Yout[r * ldy + c0 + j] -= acc[j];
          else
            Yout[r * ldy + c0 + j] = dv[r] * Z[r * ldy + c0 + j] + acc[j];
        }
      }
    }
  }
}

// Both coupling products of a sweep node in one pass:
//   Y -= A1 Z1 + A2 Z2,   A(r,k) = M[k*ldm + r] if transposed else M[r*ldm + k];
// a null M skips its product.  Same thread layout as res_rowdot.
template <typename T, int CW, bool TR1, bool TR2>
__device__ __forceinline__ void res_rowdot_pair(T* Y, const T* Z1, const T* M1, const T* Z2, const T* M2, int ldy,
                                                int mc, int ldm, int n) {
  const int q = threadIdx.x & 3;
  const int nr = ((n + 7) / 8) * 8;
  const bool h1 = M1 != nullptr, h2 = M2 != nullptr;
  for (int c0 = 0; c0 < mc; c0 += CW) {
    for (int rb = threadIdx.x >> 2; rb < nr; rb += blockDim.x >> 2) {
      const int r = rb < n ? rb : n - 1;
      T acc[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) acc[j] = T(0);
#pragma unroll 4
      for (int k = q; k < n; k += 4) {
        if (h1) {
          const T mv = TR1 ? M1[k * ldm + r] : M1[r * ldm + k];
          T z[CW];
          load_cols<T, CW>(Z1 + k * ldy + c0, z);
#pragma unroll
          for (int j = 0; j < CW; ++j) acc[j] = fma(mv, z[j], acc[j]);
        }
        if (h2) {
          const T mv = TR2 ? M2[k * ldm + r] : M2[r * ldm + k];
          T z[CW];
          load_cols<T, CW>(Z2 + k * ldy + c0, z);
#pragma unroll
          for (int j = 0; j < CW; ++j) acc[j] = fma(mv, z[j], acc[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        acc[j] += __shfl_xor_sync(kFull, acc[j], 1);
        acc[j] += __shfl_xor_sync(kFull, acc[j], 2);
      }
      if (rb < n) {
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          if ((j & 3) != q || c0 + j >= mc) continue;
          Y[r * ldy + c0 + j] -= acc[j];
        }
      }
    }
  }
}

template <typename T, bool TR1, bool TR2>
__device__ __forceinline__ void res_matvec_pair(T* Y, const T* Z1, const T* M1, const T* Z2, const T* M2, int ldy,
                                                int mc, int ldm, int n) {
  if (mc >= 8)
    res_rowdot_pair<T, 8, TR1, TR2>(Y, Z1, M1, Z2, M2, ldy, mc, ldm, n);
  else if (mc >= 4)
    res_rowdot_pair<T, 4, TR1, TR2>(Y, Z1, M1, Z2, M2, ldy, mc, ldm, n);
  else if (mc >= 2)
    res_rowdot_pair<T, 2, TR1, TR2>(Y, Z1, M1, Z2, M2, ldy, mc, ldm, n);
  else
    res_rowdot_pair<T, 1, TR1, TR2>(Y, Z1, M1, Z2, M2, ldy, mc, ldm, n);
}

template <typename T, int MODE>
__device__ __forceinline__ void res_matvec(T* Yout, const T* Z, int ldy, int mc, const T* M, int ldm, const T* dv,
                                           int n) {
  if (mc >= 8)
    res_rowdot<T, MODE, 8>(Yout, Z, ldy, mc, M, ldm, dv, n);
  else if (mc >= 4)
    res_rowdot<T, MODE, 4>(Yout, Z, ldy, mc, M, ldm, dv, n);
  else if (mc >= 2)
    res_rowdot<T, MODE, 2>(Yout, Z, ldy, mc, M, ldm, dv, n);
  else
    res_rowdot<T, MODE, 1>(Yout, Z, ldy, mc, M, ldm, dv, n);
}

// ---------------------------------------------------------------------------
// Products of the resident inverse sweeps on FP64 tensor cores (mma.m8n8k4
// .f64), for float and double blocks: operands are widened to double in
// registers, so products are exact and sums are FP64; the result is rounded
// to T once.  A(r,k) = TR ? M[k*ld + r] : M[r*ld + k].
//   MODE 0: Out -= A1 Z1 + A2 Z2     (a null A skips its product)
//   MODE 2: Out  = dv .* Z1 + A1 Z1, A1 strictly upper (k > r)
//   MODE 3: Out  = dv .* Z1 + A1 Z1, A1 strictly lower (k < r)
// Out never aliases Z1 or Z2.  Warp task = one 8 x 8 output tile, all k-steps,
// two accumulators per product (alternate k-steps).  Fragment layout: a0 =
// A[g][t], b0 = B[t][g], {c0, c1} = C[g][2t + {0, 1}] (g = lane / 4, t = lane % 4).
// ---------------------------------------------------------------------------
// Sweep products on inverse-carrying factors: FP64 sweeps always take the
// tensor-core products (faster at every level); FP32 sweeps only in launches
// wider than one wave of resident sweep CTAs, which are throughput-bound
// (measured at N=1024, n=64: bottom level 17.0 -> 15.7 us), while the
// dependent DMMA chain costs ~0.6 us per node on the 1-256-CTA levels and in
// the persistent ragged CTAs, where the SIMT products are faster.  The host
// decides per launch (Level::tc, from the launch width and the device's SM
// count, or from a tuned setting).
template <typename T>
__device__ __forceinline__ bool sweep_uses_dmma(const Level& lv) {
  return sizeof(T) == 8 || lv.tc != 0;
}

template <typename T, int MODE, bool TR>
__device__ __forceinline__ double dmma_a(const T* A, int ld, int n, int r, int k) {
  bool ok = r < n && k < n;
  if (MODE == 2) ok = ok && k > r;
  if (MODE == 3) ok = ok && k < r;
  const int rr = r < n ? r : 0, kk = k < n ? k : 0;
  const T v = TR ? A[kk * ld + rr] : A[rr * ld + kk];
  return ok ? (double)v : 0.0;
}

template <typename T, int MODE, bool TR1, bool TR2>
__device__ void dmma_product(T* Out, const T* Z1, const T* A1, int ld1, const T* Z2, const T* A2, int ld2, int ldy,
                             int mc, const T* dv, int n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rt = (n + 7) >> 3, ct = (mc + 7) >> 3, kt = (n + 3) >> 2;
  const bool h1 = A1 != nullptr, h2 = MODE == 0 && A2 != nullptr;
  for (int task = warp; task < rt * ct; task += nw) {
    const int r0 = (task / ct) * 8, c0 = (task % ct) * 8;
    const int ra = r0 + g, cb = c0 + g;
    const bool cv = cb < mc;
    const int cc = cv ? cb : 0;
    double acc[4][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    int kb0 = 0, kb1 = kt;
    if (MODE == 2) kb0 = (r0 + 1) >> 2;                             // first k-step with some k > r
    if (MODE == 3) kb1 = min_i(kt, (r0 + 7 + 3) >> 2);              // past the last with some k < r
    for (int kb = kb0; kb < kb1; kb += 2) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {   // two k-steps, one accumulator each
        const int k = (kb + h) * 4 + t;
        const bool kv = kb + h < kb1 && k < n;
        const int kk = kv ? k : 0;
        if (h1) {
          const double a = kv ? dmma_a<T, MODE, TR1>(A1, ld1, n, ra, kk) : 0.0;
          const double b = (kv && cv) ? (double)Z1[kk * ldy + cc] : 0.0;
          dmma_8x8x4(acc[h][0], acc[h][1], a, b);
        }
        if (h2) {
          const double a = kv ? dmma_a<T, MODE, TR2>(A2, ld2, n, ra, kk) : 0.0;
          const double b = (kv && cv) ? (double)Z2[kk * ldy + cc] : 0.0;
          dmma_8x8x4(acc[2 + h][0], acc[2 + h][1], a, b);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = r0 + g, c = c0 + 2 * t + e;
      if (r < n && c < mc) {
        const double v = (acc[0][e] + acc[1][e]) + (acc[2][e] + acc[3][e]);
        T* out = Out + r * ldy + c;
        if (MODE == 0)
          *out = (T)((double)*out - v);
        else
          *out = (T)((double)dv[r] * (double)Z1[r * ldy + c] + v);
      }
    }
  }
}

// Y <- C^{-1} Y (UPPER: Y <- C^{-T} Y), C = lower(Cs) resident, dv[r] = 1/C[r][r].
// Right-looking by 8-row blocks: one thread per column solves the block
// against the 8x8 diagonal block held in registers, then every (row, column)
// of the remaining rows takes an 8-term update.
template <typename T, bool UPPER>
__device__ void res_tri_solve(T* Y, int ldy, int mc, const T* Cs, int ldc, const T* dv, int n) {
  constexpr int BK = 8;
  const int nblk = (n + BK - 1) / BK;
  for (int bi = 0; bi < nblk; ++bi) {
    const int K = UPPER ? (nblk - 1 - bi) * BK : bi * BK;
    const int kb = min_i(BK, n - K);
    for (int c = threadIdx.x; c < mc; c += blockDim.x) {
      T x[BK];
#pragma unroll
      for (int j = 0; j < BK; ++j) x[j] = j < kb ? Y[(K + j) * ldy + c] : T(0);
      if (!UPPER) {
#pragma unroll
        for (int j = 0; j < BK; ++j) {
          if (j < kb) {
#pragma unroll
            for (int i = 0; i < j; ++i) x[j] = fma(-Cs[(K + j) * ldc + K + i], x[i], x[j]);
            x[j] *= dv[K + j];
          }
        }
      } else {
#pragma unroll
        for (int j = BK - 1; j >= 0; --j) {
          if (j < kb) {
#pragma unroll
            for (int i = j + 1; i < BK; ++i)
              if (i < kb) x[j] = fma(-Cs[(K + i) * ldc + K + j], x[i], x[j]);
            x[j] *= dv[K + j];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < BK; ++j)
        if (j < kb) Y[(K + j) * ldy + c] = x[j];
    }
    __syncthreads();
    // remaining rows: below the block (forward) or above it (backward)
    const int r0 = UPPER ? 0 : K + kb;
    const int nr = UPPER ? K : n - K - kb;
    for (int o = threadIdx.x; o < nr * mc; o += blockDim.x) {
      const int r = r0 + o / mc, c = o - (o / mc) * mc;
      T acc = T(0);
#pragma unroll
      for (int j = 0; j < BK; ++j)
        if (j < kb) acc = fma(UPPER ? Cs[(K + j) * ldc + r] : Cs[r * ldc + K + j], Y[(K + j) * ldy + c], acc);
      Y[r * ldy + c] -= acc;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// k_fwd (level l): pull the level-(l-1) coupling updates and solve.
//   l == 0: task t -> node i = 2t:  y_i <- C_i^{-1} y_i
//   l >= 1: task u-1, target j = s*u - 1 of the level-(l-1) updates:
//           y_j -= F y_{j-s/2} + G^T y_{j+s/2}   (slots o_{l-1}+2u-2, +2u-1)
//           and for odd u (j is a level-l node) y_j <- C_j^{-1} y_j.
// Every vector has one writer per launch (K launches per forward sweep).
// RES: factor and coupling blocks resident in shared memory.
// ---------------------------------------------------------------------------
// PULL_ONLY (fused factor_and_solve): apply the updates, never solve.
// INV (resident only): the factor carries its inverse (k_node<INV>), the
// triangular solve becomes a matvec.
// Tasks of one forward level per instance.
__host__ __device__ inline int fwd_tasks(int N, const Level& lv) { return lv.s == 1 ? lv.d : N / lv.s; }

template <typename T, bool RES, bool PULL_ONLY, bool INV>
__device__ __forceinline__ void fwd_body(const Problem<T>& p, const Level& lv, int b, int task,
                                         unsigned char* smem_raw, const SweepMaps* tm = nullptr) {
  const int s = lv.s, N = p.N, n = p.n;
  const int h = s / 2;
  int j, slot = 0;
  bool pull, solve;
  const T *F = nullptr, *G = nullptr;
  if (s == 1) {
    j = 2 * task;
    pull = false;
    solve = true;
  } else {
    const int u = task + 1;
    j = s * u - 1;
    pull = true;
    solve = !PULL_ONLY && (u & 1) != 0;
    slot = lv.op + 2 * u - 2;
    F = p.Eb(b, slot);
    if (j + h < N) G = p.Eb(b, slot + 1);
  }
  const int mcmax = min_i(p.m, kMC), ldy = RES ? res_ldy(mcmax) : sweep_ldy(mcmax);
  // RES: Y, Z1, Z2 (n x ldy), C, F, G (n x ldm), dv (n), two mbarriers, regions on
  // 128 bytes; else Y, Z1, Z2, Cc (smem_sweep_elems), dv
  const long long vy = RES ? res_round((long long)n * ldy, sizeof(T)) : (long long)n * ldy;
  T* Y = reinterpret_cast<T*>(smem_raw);
  T* Z1 = Y + vy;
  T* Z2 = Z1 + vy;
  T* Ms = Z2 + vy;
  const int ldm = res_ldm(n);
  const long long vm = res_round((long long)n * ldm, sizeof(T));
  T* Cs = Ms;
  T* Fs = Cs + vm;
  T* Gs = Fs + vm;
  T* dv = RES ? Gs + vm : Ms + (smem_sweep_elems(n, p.m) - 3LL * n * ldy - kTile);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + ((reinterpret_cast<unsigned char*>(dv + n) - smem_raw + 7) & ~7LL));
  T* yj = p.Xb(b, j);
  const T* Lj = p.Lb(b, j);
  const ResTma tu = RES ? res_tma_begin(tm, smem_raw, bar) : ResTma{false, false};
  const int nblk = RES ? (solve ? 1 : 0) + (F ? 1 : 0) + (G ? 1 : 0) : 0;
  if (!lv.pre) pdl_wait();
  if (RES) {
    if (tu.blocks) {
      if (threadIdx.x == 0 && nblk > 0) {
        tma::expect_tx(bar, (uint32_t)(nblk * n * ldm * sizeof(T)));
        if (solve) tma::load_4d(Cs, &tm->L, 0, 0, j, b, bar);
        if (F) tma::load_4d(Fs, &tm->E, 0, 0, slot, b, bar);
        if (G) tma::load_4d(Gs, &tm->E, 0, 0, slot + 1, b, bar);
      }
    } else {
      if (solve) async_load(Cs, ldm, Lj, n, n, n);
      if (F) async_load(Fs, ldm, F, n, n, n);
      if (G) async_load(Gs, ldm, G, n, n, n);
    }
  }
  if (lv.pre) pdl_wait();
  pdl_trigger();
  for (int c0 = 0, chunk = 0; c0 < p.m; c0 += kMC, ++chunk) {
    const int mc = min_i(kMC, p.m - c0);
    __syncthreads();
    if (tu.vecs) {
      if (threadIdx.x == 0) {
        tma::fence_proxy();
        tma::expect_tx(bar + 1, (uint32_t)((1 + (pull ? 1 : 0) + (G ? 1 : 0)) * n * ldy * sizeof(T)));
        tma::load_4d(Y, &tm->X, c0, 0, j, b, bar + 1);
        if (pull) tma::load_4d(Z1, &tm->X, c0, 0, j - h, b, bar + 1);
        if (G) tma::load_4d(Z2, &tm->X, c0, 0, j + h, b, bar + 1);
      }
    } else {
      async_load(Y, ldy, yj + c0, n, mc, p.m);
      if (pull) async_load(Z1, ldy, p.Xb(b, j - h) + c0, n, mc, p.m);
      if (G) async_load(Z2, ldy, p.Xb(b, j + h) + c0, n, mc, p.m);
    }
    cp_async_wait_all();
    if ((tu.blocks || tu.vecs) && !res_tma_wait(tu, nblk > 0 && chunk == 0, bar, chunk)) return;
    __syncthreads();
    if (RES) {
      if (c0 == 0 && solve)
        for (int r = threadIdx.x; r < n; r += blockDim.x) dv[r] = T(1) / Cs[r * ldm + r];
      // Y -= F y_{j-h} + G^T y_{j+h}
      const bool tc = INV && sweep_uses_dmma<T>(lv);
      if (pull) {
        if (tc)
          dmma_product<T, 0, false, true>(Y, Z1, Fs, ldm, G ? Z2 : nullptr, G ? Gs : nullptr, ldm, ldy, mc, nullptr, n);
        else
          res_matvec_pair<T, false, true>(Y, Z1, Fs, G ? Z2 : nullptr, G ? Gs : nullptr, ldy, mc, ldm, n);
      }
      __syncthreads();
      if (solve) {
        if (INV) {
          if (tc)
            dmma_product<T, 3, true, false>(Z2, Y, Cs, ldm, nullptr, nullptr, 0, ldy, mc, dv, n);   // y = W Y
          else
            res_matvec<T, 3>(Z2, Y, ldy, mc, Cs, ldm, dv, n);
          __syncthreads();
          store_block(yj + c0, p.m, Z2, ldy, n, mc);
          continue;
        }
        res_tri_solve<T, false>(Y, ldy, mc, Cs, ldm, dv, n);
      }
    } else {
      if (pull) sweep_accumulate2<T, false, true>(Y, Z1, F, Z2, G, ldy, mc, n, Ms);
      if (solve) sweep_lower_solve(Y, ldy, mc, Lj, n, Ms, dv);
    }
    store_block(yj + c0, p.m, Y, ldy, n, mc);
  }
}

// ---------------------------------------------------------------------------
// k_bwd (level l, descending): x_i -= F_i^T x_{i+s} + G_i x_{i-s};  x_i <- C_i^{-T} x_i
// ---------------------------------------------------------------------------
template <typename T, bool RES, bool INV>
__device__ __forceinline__ void bwd_body(const Problem<T>& p, const Level& lv, int b, int t,
                                         unsigned char* smem_raw, const SweepMaps* tm = nullptr) {
  const int n = p.n, s = lv.s, N = p.N;
  const int i = s - 1 + 2 * s * t;
  const int mcmax = min_i(p.m, kMC), ldy = RES ? res_ldy(mcmax) : sweep_ldy(mcmax);
  // shared layout as in fwd_body
  const long long vy = RES ? res_round((long long)n * ldy, sizeof(T)) : (long long)n * ldy;
  T* Y = reinterpret_cast<T*>(smem_raw);
  T* Z1 = Y + vy;
  T* Z2 = Z1 + vy;
  T* Ms = Z2 + vy;
  const int ldm = res_ldm(n);
  const long long vm = res_round((long long)n * ldm, sizeof(T));
  T* Cs = Ms;
  T* Fs = Cs + vm;
  T* Gs = Fs + vm;
  T* dv = RES ? Gs + vm : Ms + (smem_sweep_elems(n, p.m) - 3LL * n * ldy - kTile);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + ((reinterpret_cast<unsigned char*>(dv + n) - smem_raw + 7) & ~7LL));
  const bool right = i + s < N, left = i >= s;
  const int slot = lv.oc + 2 * t;
  const T* F = right ? p.Eb(b, slot) : nullptr;
  const T* G = left ? p.Eb(b, slot - 1) : nullptr;
  const T* Li = p.Lb(b, i);
  T* xi = p.Xb(b, i);
  const ResTma tu = RES ? res_tma_begin(tm, smem_raw, bar) : ResTma{false, false};
  if (!lv.pre) pdl_wait();
  if (RES) {
    if (tu.blocks) {
      if (threadIdx.x == 0) {
        tma::expect_tx(bar, (uint32_t)((1 + (right ? 1 : 0) + (left ? 1 : 0)) * n * ldm * sizeof(T)));
        tma::load_4d(Cs, &tm->L, 0, 0, i, b, bar);
        if (right) tma::load_4d(Fs, &tm->E, 0, 0, slot, b, bar);
        if (left) tma::load_4d(Gs, &tm->E, 0, 0, slot - 1, b, bar);
      }
    } else {
      async_load(Cs, ldm, Li, n, n, n);
      if (right) async_load(Fs, ldm, F, n, n, n);
      if (left) async_load(Gs, ldm, G, n, n, n);
    }
  }
  if (lv.pre) pdl_wait();
  pdl_trigger();
  for (int c0 = 0, chunk = 0; c0 < p.m; c0 += kMC, ++chunk) {
    const int mc = min_i(kMC, p.m - c0);
    __syncthreads();
    if (tu.vecs) {
      if (threadIdx.x == 0) {
        tma::fence_proxy();
        tma::expect_tx(bar + 1, (uint32_t)((1 + (right ? 1 : 0) + (left ? 1 : 0)) * n * ldy * sizeof(T)));
        tma::load_4d(Y, &tm->X, c0, 0, i, b, bar + 1);
        if (right) tma::load_4d(Z1, &tm->X, c0, 0, i + s, b, bar + 1);
        if (left) tma::load_4d(Z2, &tm->X, c0, 0, i - s, b, bar + 1);
      }
    } else {
      async_load(Y, ldy, xi + c0, n, mc, p.m);
      if (right) async_load(Z1, ldy, p.Xb(b, i + s) + c0, n, mc, p.m);
      if (left) async_load(Z2, ldy, p.Xb(b, i - s) + c0, n, mc, p.m);
    }
    cp_async_wait_all();
    if ((tu.blocks || tu.vecs) && !res_tma_wait(tu, chunk == 0, bar, chunk)) return;
    __syncthreads();
    if (RES) {
      if (c0 == 0)
        for (int r = threadIdx.x; r < n; r += blockDim.x) dv[r] = T(1) / Cs[r * ldm + r];
      // Y -= F^T x_{i+s} + G x_{i-s}
      const bool tc = INV && sweep_uses_dmma<T>(lv);
      if (right || left) {
        if (tc)
          dmma_product<T, 0, true, false>(Y, right ? Z1 : nullptr, right ? Fs : nullptr, ldm, left ? Z2 : nullptr,
                                          left ? Gs : nullptr, ldm, ldy, mc, nullptr, n);
        else
          res_matvec_pair<T, true, false>(Y, right ? Z1 : nullptr, right ? Fs : nullptr, left ? Z2 : nullptr,
                                          left ? Gs : nullptr, ldy, mc, ldm, n);
      }
      __syncthreads();
      if (INV) {
        if (tc)
          dmma_product<T, 2, false, false>(Z1, Y, Cs, ldm, nullptr, nullptr, 0, ldy, mc, dv, n);   // x = W^T Y
        else
          res_matvec<T, 2>(Z1, Y, ldy, mc, Cs, ldm, dv, n);
        __syncthreads();
        store_block(xi + c0, p.m, Z1, ldy, n, mc);
        continue;
      }
      res_tri_solve<T, true>(Y, ldy, mc, Cs, ldm, dv, n);
    } else {
      sweep_accumulate2<T, true, false>(Y, Z1, F, Z2, G, ldy, mc, n, Ms);
      sweep_upper_solve(Y, ldy, mc, Li, n, Ms, dv);
    }
    store_block(xi + c0, p.m, Y, ldy, n, mc);
  }
}

}  // namespace socu
