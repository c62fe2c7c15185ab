// Level node as rows of 8x8 tiles held in registers (n <= 128), one thread
// block per node (or a thread-block cluster of `splits` blocks on levels with
// fewer nodes than SMs).
//
// The node's Cholesky factor C and everything multiplied by C^{-T} are one
// matrix of row tiles over the same 8-column steps:
//     X = [ L_i ; R ; Lf^T ; y^T ; I ],      X <- X C^{-T}
// whose rows end as C, F = R C^{-T}, G^T = Lf^T C^{-T}, (C^{-1} y)^T and
// W^T = C^{-T}: exactly the blocks the factor stores.  A warp owns a whole row
// tile (8 x n) as FP64 tensor-core accumulators (mma.m8n8k4 .f64, fragment
// {c0, c1} = C[g][2t + {0, 1}], g = lane / 4, t = lane % 4), read from global
// memory straight into registers.  Step k:
//   1. the warp of row k factors its diagonal tile (every lane the whole tile)
//      and publishes C_kk and Inv_k = C_kk^{-1} in shared memory;
//   2. every later row multiplies its tile k by Inv_k^T and corrects the product
//      against C_kk (rows_panel): the final tile P, as exact as a substitution;
//   3. every later row adds P P_j^T to the sums that its tiles j > k are less of.
// The accumulator fragment is the A operand of the next product without any
// shuffle: the contraction index is enumerated as 2t, 2t + 1 (one MMA each),
// and the B operand (a row of Inv_k or of P_j) is then one 16-byte load.
//
// Rows of L_i go through the steps together (phase 1, two barriers per step;
// the warp of row k + 1 has one tile left to update, so it reaches its factor
// while the other warps still update).  The other rows only read what phase 1
// left in shared memory, so each warp takes them one row tile at a time with
// no barrier (phase 2); the first one is loaded when the warp leaves phase 1.
//
// Bound by the latency of phase 1: per step one tile factor (770 cycles FP64,
// 556 float), the panel's three dependent MMA pairs (26 cycles each half) and the
// next diagonal tile's.  The blocks
// of a cluster repeat phase 1 and share out phase 2; the cluster barrier keeps
// one block from overwriting L_i before the others have read it.  Measured,
// all level nodes of one factor_and_solve (event-timed launches), against the
// blocked solve in shared memory that it replaces: N=1024, n=64, m=8 FP64
// 409 -> 231 us, float 373 -> 208 us; N=2048, n=128, m=32 FP64 3308 -> 1203 us
// (201, 178 and 917 us with the inverse's product alone, see rows_panel).
#pragma once

#include "nd_kernels.cuh"

namespace socu {

// 8-column tiles: exact up to 64, then even counts (fewer instantiations)
__host__ __device__ inline int rows_nt(int n) {
  const int t = (n + 7) / 8;
  return t <= 8 ? t : ((t + 1) & ~1);
}
// row stride of the shared factor: 8 (mod 16) doubles, so the 16-byte operand
// loads of a quarter warp (two rows of 64 bytes) cover all banks
__host__ __device__ inline int rows_ld(int nt) { return (nt & 1) ? 8 * nt : 8 * nt + 8; }
__host__ __device__ inline int rows_warps(int nt) { return nt < 4 ? 4 : nt; }
__host__ __device__ inline long long smem_rows_bytes(int n) {
  const int nt = rows_nt(n);
  return 8LL * (8LL * nt * rows_ld(nt) + 128LL * nt);
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }

// Accumulate one MMA.  Not volatile: the compiler may interleave independent ones.
__device__ __forceinline__ void mma_acc(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// named barriers: producers arrive, consumers wait
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_wait(int id, int threads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// 1 / sqrt(d) without a branch: the approximate instruction, then one step of
// Householder's third-order iteration y (1 + e/2 + 3 e^2 / 8), e = 1 - d y^2.
// For normal d.  A subnormal one is flushed by the instruction: infinity comes
// out, and the caller, whose last pivot is then not finite, starts over with the
// library function.
template <typename T, bool FAST>
__device__ __forceinline__ T pivot_rsqrt(T d) {
  if constexpr (FAST && sizeof(T) == 8) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-(d * y), y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
  } else {
    return rsqrt_t(d);
  }
}

// Cholesky factor of the 8x8 tile in S, written over it (lower triangle; the
// caller clears the rest), and its inverse, written to Ivk (8 x 8, lane l the
// column l % 8); returns the last pivot's factor.  Every lane of the warp factors
// the whole tile: the chain is 8 times rsqrt -> multiply -> subtract, about 70
// cycles each in FP64, with no exchange between lanes; the stores go out beside it.
// Measured per tile, without the stores: 770 cycles FP64, 556 float; spread over
// the lanes instead (16 shuffles a column, which issue every 4.3 cycles) 1500 and 790.
template <typename T, bool FAST>
__device__ __forceinline__ T chol8_tile(T* S, double* Ivk) {
  const int lane = threadIdx.x & 31, col = lane & 7;
  T c[8][8], y[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j <= i; j += 2) {
      if constexpr (sizeof(T) == 8) {
        const double2 v = *reinterpret_cast<const double2*>(S + 8 * i + j);
        c[i][j] = v.x;
        c[i][j + 1] = v.y;
      } else {
        const float2 v = *reinterpret_cast<const float2*>(S + 8 * i + j);
        c[i][j] = v.x;
        c[i][j + 1] = v.y;
      }
    }
  __syncwarp();   // every lane has read S
#pragma unroll
  for (int i = 0; i < 8; ++i) y[i] = T(0);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const T d = c[j][j], r = pivot_rsqrt<T, FAST>(d);
#pragma unroll
    for (int i = j; i < 8; ++i) c[i][j] *= r;
    // the root itself, off the chain: one Newton step brings d r within half a unit in the last place
    c[j][j] = fma(T(0.5) * r, fma(-c[j][j], c[j][j], d), c[j][j]);
#pragma unroll
    for (int l = j + 1; l < 8; ++l)
#pragma unroll
      for (int i = l; i < 8; ++i) c[i][l] = fma(-c[i][j], c[l][j], c[i][l]);
    y[j] = j == col ? r : y[j] * r;
#pragma unroll
    for (int i = j + 1; i < 8; ++i) y[i] = fma(-c[i][j], y[j], y[i]);
    Ivk[8 * j + col] = (double)y[j];
    if (lane == 0) {
#pragma unroll
      for (int i = j; i < 8; ++i) S[8 * i + j] = c[i][j];
    }
  }
  return c[7][7];
}

// the factor with the library's reciprocal square root (subnormal pivots)
template <typename T>
__device__ __noinline__ void chol8_redo(T* S, double* Ivk) {
  chol8_tile<T, false>(S, Ivk);
}

// an accumulator fragment as an 8 x 8 tile
template <typename T>
__device__ __forceinline__ void frag_put(T* S, double d0, double d1) {
  const int lane = threadIdx.x & 31;
  if constexpr (sizeof(T) == 8)
    *reinterpret_cast<double2*>(S + 2 * lane) = make_double2(d0, d1);
  else
    *reinterpret_cast<float2*>(S + 2 * lane) = make_float2((float)d0, (float)d1);
}

// Factor the diagonal tile held as an accumulator fragment (d0, d1): C_kk goes to
// S (8 x 8, zeros above the diagonal) and its inverse to Ivk.  All lanes of the
// warp; the caller orders its reads of S and Ivk with __syncwarp or a barrier.
template <typename T>
__device__ __forceinline__ void rows_factor_tile(double d0, double d1, T* S, double* Ivk) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  frag_put(S, d0, d1);
  __syncwarp();
  const T last = chol8_tile<T, true>(S, Ivk);
  // An infinite factor of column 0 to 6 is a NaN in every later pivot (infinity less infinity, or
  // infinity times zero); in column 7 it is the last pivot itself.
  if (sizeof(T) == 8 && !isfinite(last)) {
    __syncwarp();   // S and Ivk are written again
    frag_put(S, d0, d1);
    __syncwarp();
    chol8_redo<T>(S, Ivk);
  }
  if (2 * t > g) S[2 * lane] = T(0);
  if (2 * t + 1 > g) S[2 * lane + 1] = T(0);
}

// The warps that work on one node, output block or vector: a whole thread
// block, or some warps of one (ragged batches), with their barriers.
struct BlockGroup {
  __device__ __forceinline__ int tid() const { return threadIdx.x; }
  __device__ __forceinline__ int threads() const { return blockDim.x; }
  __device__ __forceinline__ int warp() const { return threadIdx.x >> 5; }
  __device__ __forceinline__ int warps() const { return blockDim.x >> 5; }
  __device__ __forceinline__ int bar(int k) const { return k; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
};
struct WarpGroup {
  int first, n, bar0;   // first warp, warps, barriers bar0 .. bar0 + 2
  __device__ __forceinline__ int tid() const { return threadIdx.x - 32 * first; }
  __device__ __forceinline__ int threads() const { return 32 * n; }
  __device__ __forceinline__ int warp() const { return (threadIdx.x >> 5) - first; }
  __device__ __forceinline__ int warps() const { return n; }
  __device__ __forceinline__ int bar(int k) const { return bar0 + k; }
  __device__ __forceinline__ void sync() const {
    if (n == 1)
      __syncwarp();
    else
      bar_wait(bar0, 32 * n);
  }
};

// two consecutive elements, widened; `vec`: the pair is aligned and inside; `pair`: it is aligned
// and, where its first element is inside, all of it
template <typename T>
__device__ __forceinline__ void load_pair(const T* p, bool vec, bool v0, bool v1, double& x0, double& x1,
                                          bool pair = false) {
  if (pair && !vec && !v0) {
    x0 = x1 = 0.0;
  } else if (vec || pair) {
    if constexpr (sizeof(T) == 8) {
      const double2 v = *reinterpret_cast<const double2*>(p);
      x0 = v.x;
      x1 = v.y;
    } else {
      const float2 v = *reinterpret_cast<const float2*>(p);
      x0 = (double)v.x;
      x1 = (double)v.y;
    }
  } else {
    x0 = v0 ? (double)p[0] : 0.0;
    x1 = v1 ? (double)p[1] : 0.0;
  }
}
// two consecutive elements as they are
template <typename T>
__device__ __forceinline__ void load_raw(const T* p, bool vec, bool v0, bool v1, T (&x)[2], bool pair = false) {
  if (pair && !vec && !v0) {
    x[0] = x[1] = T(0);
  } else if (vec || pair) {
    if constexpr (sizeof(T) == 8) {
      const double2 v = *reinterpret_cast<const double2*>(p);
      x[0] = v.x;
      x[1] = v.y;
    } else {
      const float2 v = *reinterpret_cast<const float2*>(p);
      x[0] = v.x;
      x[1] = v.y;
    }
  } else {
    x[0] = v0 ? p[0] : T(0);
    x[1] = v1 ? p[1] : T(0);
  }
}

template <typename T>
__device__ __forceinline__ void store_pair(T* p, bool vec, bool v0, bool v1, double x0, double x1, bool pair = false) {
  if (vec || (pair && v0)) {
    if constexpr (sizeof(T) == 8)
      *reinterpret_cast<double2*>(p) = make_double2(x0, x1);
    else
      *reinterpret_cast<float2*>(p) = make_float2((float)x0, (float)x1);
  } else if (!pair) {
    if (v0) p[0] = (T)x0;
    if (v1) p[1] = (T)x1;
  }
}

// Every row of a block on a pair boundary; and whole 8x8 tiles besides.
template <typename T>
__host__ __device__ __forceinline__ bool rows_paired(const Problem<T>& p, int n) {
  return (n & 1) == 0 && ((reinterpret_cast<uintptr_t>(p.L) | reinterpret_cast<uintptr_t>(p.E)) & (2 * sizeof(T) - 1)) == 0;
}
template <typename T>
__host__ __device__ __forceinline__ bool pairs_ok(const Problem<T>& p, int n) {
  return (n & 7) == 0 && rows_paired(p, n);
}

// A row tile outside L_i: element (r, c) of X, r < lim, at base[r * rs + c * cs].
// kind 0: a row-major block (cs = 1, rs = n); 1: a transposed block (rs = 1);
// 2: rows of the identity (W^T), 3: zeros of the upper triangle of L_i.
template <typename T>
struct RowSrc {
  int kind;
  T* base;      // first element of the row tile
  int ld;       // kind 0: rs; kind 1: cs
  int lim;      // valid rows in the tile
  int k0;       // first step
  bool full;    // whole tiles: no bounds to check (n == 8 nta; not the right-hand sides)
};

// What a panel product reads of one diagonal tile: this lane's elements of Inv_k, of C_kk below the
// diagonal, and the diagonal of its two accumulator columns.
struct DiagFrag {
  double2 iv, cv;
  double d0, d1;
};
template <typename T>
__device__ __forceinline__ DiagFrag diag_frag(const double* Ik, const T* Ck) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  DiagFrag f;
  f.iv = *reinterpret_cast<const double2*>(Ik + 2 * lane);
  load_pair(Ck + 2 * lane, true, true, true, f.cv.x, f.cv.y);
  f.d0 = (double)Ck[18 * t];
  f.d1 = (double)Ck[18 * t + 9];
  if (2 * t == g) f.cv.x = 0.0;
  if (2 * t + 1 == g) f.cv.y = 0.0;
  return f;
}

// X tile row: P = X_k C_kk^{-T}.  The product with the explicit inverse has a residual that grows
// with the tile's condition; one correction, P += (X - P C_kk^T) Inv_k^T, brings it down to that of
// a substitution.  The diagonal's part of the residual is one fused operation, so that what cancels
// is not rounded before, and the correction is summed by itself and added once.  Componentwise
// backward error of C and F at a tile of condition 1e4: over 1000 u without it, a few u with it; true
// error of F at n = 16: 1.5e-16 without, 1.3e-16 corrected in the product's own accumulators, 1.0e-16
// so.  N = 1024, n = 64, m = 8 FP64 368, 396 and 404 us.
__device__ __forceinline__ void rows_panel(double& p0, double& p1, double x0, double x1, const DiagFrag& f) {
  double s0 = 0.0, s1 = 0.0, q0 = 0.0, q1 = 0.0;
  p0 = p1 = 0.0;
  mma_acc(p0, p1, x0, f.iv.x);
  mma_acc(p0, p1, x1, f.iv.y);
  mma_acc(s0, s1, p0, f.cv.x);
  mma_acc(s0, s1, p1, f.cv.y);
  const double r0 = fma(-p0, f.d0, x0) - s0, r1 = fma(-p1, f.d1, x1) - s1;
  mma_acc(q0, q1, r0, f.iv.x);
  mma_acc(q0, q1, r1, f.iv.y);
  p0 += q0;
  p1 += q1;
}

// (identity rows start at their own step: tile k0 is the identity, later tiles zero)
template <typename T, int NT, bool PAIR = false>
__device__ __forceinline__ void rows_load(T (&x)[NT][2], const RowSrc<T>& s, int n, bool vec) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bool rv = g < s.lim;
  if (s.kind == 0) {
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int c = 8 * j + 2 * t;
      load_raw(s.base + (g * s.ld + c), vec && 8 * j < n, rv && c < n, rv && c + 1 < n, x[j], PAIR);
    }
  } else if (s.kind == 1) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * j + 2 * t + e;
        const bool in = s.full ? 8 * j < n : rv && c < n;
        x[j][e] = in ? s.base[c * s.ld + g] : T(0);
      }
  } else {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) x[j][e] = (j == s.k0 && g == 2 * t + e) ? T(1) : T(0);
  }
}

template <typename T, int NT, bool PAIR = false>
__device__ __forceinline__ void rows_store(const double (&acc)[NT][2], const RowSrc<T>& s, int n, bool vec) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bool rv = g < s.lim;
  if (s.kind == 1) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * j + 2 * t + e;
        if (s.full ? 8 * j < n : rv && c < n) s.base[c * s.ld + g] = (T)acc[j][e];
      }
  } else {
    // (rows of the identity: tiles right of the diagonal one, which is written with C_kk)
    const int j0 = s.kind == 2 ? s.k0 + 1 : 0;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int c = 8 * j + 2 * t;
      if (j >= j0)
        store_pair(s.base + (g * s.ld + c), vec && 8 * j < n, rv && c < n, rv && c + 1 < n, acc[j][0], acc[j][1], PAIR);
    }
  }
}

// tiles j0 .. j0 + CH - 1 (below NT) of one row tile += A P_j^T, A = (a0, a1)
template <int NT, int CH>
__device__ __forceinline__ void rows_update(double (&acc)[NT][2], int j0, double a0, double a1, const double* Ck,
                                            int ld) {
  double2 bv[CH];
#pragma unroll
  for (int h = 0; h < CH; ++h)
    if (j0 + h < NT) bv[h] = *reinterpret_cast<const double2*>(Ck + 8 * (j0 + h) * ld);
#pragma unroll
  for (int h = 0; h < CH; ++h)
    if (j0 + h < NT) mma_acc(acc[j0 + h][0], acc[j0 + h][1], a0, bv[h].x);
#pragma unroll
  for (int h = 0; h < CH; ++h)
    if (j0 + h < NT) mma_acc(acc[j0 + h][0], acc[j0 + h][1], a1, bv[h].y);
}

// Sums from zero where the registers hold a row tile twice: X less the sum of the products is rounded
// once at X's size (true error of F at n = 64: 3.0e-16 -> 1.5e-16).  Larger blocks subtract every
// product from X, as a substitution does: at n = 128 the second copy spilt.
__host__ __device__ constexpr bool rows_from_zero(int nt) { return nt <= 8; }

// All steps of one row tile x against the finished factor, results in acc (FROM0: k0 is 0, and no
// branch separates the steps; the tile that the next step starts from comes first).  EXACT: nta is NT.
template <typename T, int NT, bool FROM0, bool EXACT>
__device__ __forceinline__ void rows_solve(double (&acc)[NT][2], const T (&x)[NT][2], int k0, int nta, const double* Cs,
                                           const double* Iv, const T* Ct) {
  constexpr int ld = (NT & 1) ? 8 * NT : 8 * NT + 8;
  constexpr bool ZERO = rows_from_zero(NT);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) acc[j][e] = ZERO ? 0.0 : (double)x[j][e];
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    if ((FROM0 || k >= k0) && (EXACT || k < nta)) {
      const double* Ck = Cs + g * ld + 8 * k + 2 * t;
      double p0, p1;
      rows_panel(p0, p1, ZERO ? (double)x[k][0] - acc[k][0] : acc[k][0], ZERO ? (double)x[k][1] - acc[k][1] : acc[k][1],
                 diag_frag(Iv + 64 * k, Ct + 64 * k));
      const double a0 = ZERO ? p0 : -p0, a1 = ZERO ? p1 : -p1;
      rows_update<NT, 1>(acc, k + 1, a0, a1, Ck, ld);
#pragma unroll
      for (int j = k + 2; j < NT; j += 4) rows_update<NT, 4>(acc, j, a0, a1, Ck, ld);
      acc[k][0] = p0;
      acc[k][1] = p1;
    }
  }
}

// One node.  q, splits: this block's share of the row tiles outside L_i (every
// block of a cluster runs phase 1).  Warp w < n / 8 of the group owns row tile w of L_i.
// FULL: n is 8 NT and pairs are aligned, so sizes and offsets are constants.  PAIR: rows_paired holds.
template <typename T, int NT, bool FULL, bool EXACT, bool PAIR = false, class Group>
__device__ __forceinline__ void node_rows_body(const Group& grp, const Problem<T>& p, const Level& lv, int b, int t,
                                               unsigned char* smem_raw, int q, int splits, bool with_y, bool inv) {
  constexpr int ld = (NT & 1) ? 8 * NT : 8 * NT + 8;
  const int lane = threadIdx.x & 31, row = grp.warp(), W = grp.warps();
  const int g = lane >> 2, tq = lane & 3;
  const int n = FULL ? 8 * NT : p.n, s = lv.s, i = s - 1 + 2 * s * t;
  const int nta = (n + 7) >> 3;
  const bool right = i + s < p.N, left = t >= 1;
  double* Cs = reinterpret_cast<double*>(smem_raw);   // rows of C, 8 NT x ld
  double* Iv = Cs + 8 * NT * ld;                      // Inv_k, 8 x 8 each
  T* Ct = reinterpret_cast<T*>(Iv + 64 * NT);         // C_kk, 8 x 8 each
  T* Li = p.Lb(b, i);
  T* R = right ? p.Eb(b, lv.oc + 2 * t) : nullptr;
  T* Lf = left ? p.Eb(b, lv.oc + 2 * t - 1) : nullptr;
  T* yi = with_y ? p.Xb(b, i) : nullptr;
  // paired accesses: whole tiles, and every row of a block on a pair boundary
  const bool vec = FULL || (NT > 8 && pairs_ok(p, n));   // (up to 64: NT is exact, whole tiles are FULL)
  const int vr = right ? nta : 0, vl = left ? nta : 0, vy = with_y ? (p.m + 7) >> 3 : 0;
  const int vtot = vr + vl + vy + nta;
  auto source = [&](int v) {
    RowSrc<T> o;
    o.ld = n;
    o.k0 = 0;
    o.full = vec;
    if (v < vr) {
      o.kind = 0;
      o.base = R + (long long)8 * v * n;
      o.lim = n - 8 * v;
    } else if (v < vr + vl) {
      const int c = v - vr;
      o.kind = 1;
      o.base = Lf + 8 * c;
      o.lim = n - 8 * c;
    } else if (v < vr + vl + vy) {
      const int c = v - vr - vl;
      o.kind = 1;
      o.base = yi + 8 * c;
      o.full = false;
      o.ld = p.m;
      o.lim = p.m - 8 * c;
    } else {
      const int c = v - vr - vl - vy;
      o.kind = inv ? 2 : 3;
      o.base = Li + (long long)8 * c * n;
      o.lim = n - 8 * c;
      o.k0 = c;
    }
    return o;
  };

  // This warp's row tile of L_i (lower tiles; the padding of the last tile is an identity).  Where
  // the products are summed from zero it waits in its place in shared memory, the diagonal tile in
  // registers; larger blocks have no registers for both and subtract from the tile.
  // (FP64 errors at n = 64: 7.9e-17 in C, against 1.6e-16 when every product is rounded at X's size.)
  constexpr bool ZERO = rows_from_zero(NT);
  const int gr = 8 * row + g;
  double* Xr = Cs + gr * ld + 2 * tq;
  double acc[NT][2], dx0 = 0.0, dx1 = 0.0;
  {
    double x[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      x[j][0] = x[j][1] = 0.0;
      if (row < nta && j <= row) {
        const int c = 8 * j + 2 * tq;
        load_pair(Li + (long long)gr * n + c, vec, gr < n && c < n, gr < n && c + 1 < n, x[j][0], x[j][1], PAIR);
        if (!vec && gr >= n) {
          if (c == gr) x[j][0] = 1.0;
          if (c + 1 == gr) x[j][1] = 1.0;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      acc[j][0] = ZERO ? 0.0 : x[j][0];
      acc[j][1] = ZERO ? 0.0 : x[j][1];
      if (ZERO && row < nta && j < row) *reinterpret_cast<double2*>(Xr + 8 * j) = make_double2(x[j][0], x[j][1]);
      if (ZERO ? j == row : j == 0) {
        dx0 = x[j][0];
        dx1 = x[j][1];
      }
    }
  }
  const int v_first = q + splits * row;
  if (splits > 1) cluster_arrive();   // L_i is in this thread's registers

  // Phase 1.  Barrier 1, step k: Inv_k is published (its warp arrives, later
  // rows wait); barrier 2: the step's panel is published (row k + 1 arrives, as
  // its own tile needs nothing else, later rows wait).  Warps past their row
  // leave the steps and meet the others at the end.
  if (row < nta) {
    double d0 = dx0, d1 = dx1;   // the diagonal tile
#pragma unroll
    for (int k = 0; k < NT - 1; ++k) {
      if (k < row) {
        const int after = nta - 1 - k;   // rows after k
        double2 x = make_double2(0.0, 0.0);
        if (ZERO) x = *reinterpret_cast<const double2*>(Xr + 8 * k);
        bar_wait(grp.bar(1), 32 * (after + 1));
        double p0, p1;
        rows_panel(p0, p1, ZERO ? x.x - acc[k][0] : acc[k][0], ZERO ? x.y - acc[k][1] : acc[k][1],
                   diag_frag(Iv + 64 * k, Ct + 64 * k));
        *reinterpret_cast<double2*>(Xr + 8 * k) = make_double2(p0, p1);
        const double a0 = ZERO ? p0 : -p0, a1 = ZERO ? p1 : -p1;
        if (row == k + 1) {
          if (after > 1) bar_arrive(grp.bar(2), 32 * after);
          double s0 = acc[k + 1][0], s1 = acc[k + 1][1];
          mma_acc(s0, s1, a0, p0);
          mma_acc(s0, s1, a1, p1);
          d0 = ZERO ? dx0 - s0 : s0;
          d1 = ZERO ? dx1 - s1 : s1;
        } else {
          bar_wait(grp.bar(2), 32 * after);
#pragma unroll
          for (int j = k + 1; j < NT; j += 4)
            if (j <= row) rows_update<NT, 4>(acc, j, a0, a1, Cs + g * ld + 8 * k + 2 * tq, ld);
        }
      }
    }
    rows_factor_tile<T>(d0, d1, Ct + 64 * row, Iv + 64 * row);
    if (row + 1 < nta) bar_arrive(grp.bar(1), 32 * (nta - row));
    if (splits > 1) cluster_wait();   // every block of the cluster has read L_i
    if (q == 0) {
      __syncwarp();
      for (int j = 0; j < row; ++j) {
        const double2 v = *reinterpret_cast<const double2*>(Cs + gr * ld + 8 * j + 2 * tq);
        const int c = 8 * j + 2 * tq;
        store_pair(Li + (long long)gr * n + c, vec, gr < n && c < n, gr < n && c + 1 < n, v.x, v.y, PAIR);
      }
      // diagonal tile: C_kk and, above the diagonal, W^T (or zeros)
      const double* Ik = Iv + 64 * row;
      const double c0 = (double)Ct[64 * row + 2 * lane], c1 = (double)Ct[64 * row + 2 * lane + 1];
      const int c = 8 * row + 2 * tq;
      const double u0 = inv ? Ik[8 * (2 * tq) + g] : 0.0, u1 = inv ? Ik[8 * (2 * tq + 1) + g] : 0.0;
      store_pair(Li + (long long)gr * n + c, vec, gr < n && c < n, gr < n && c + 1 < n, 2 * tq <= g ? c0 : u0,
                 2 * tq + 1 <= g ? c1 : u1, PAIR);
      if (p.info != nullptr) {
        const double dg = (g & 1) ? c1 : c0;   // lanes with t = g / 2 hold the diagonal
        const bool bad = (g >> 1) == tq && gr < n && (!(dg > 0.0) || isinf(dg));
        if (__any_sync(kFull, bad) && lane == 0) record_failure(p.info + b, i);
      }
    }
  } else if (splits > 1) {
    cluster_wait();
  }
  // (the first row tile arrives while later rows finish phase 1)
  T xv[NT][2];
  if (v_first < vtot) rows_load<T, NT, PAIR>(xv, source(v_first), n, vec);
  grp.sync();   // the factor is complete in shared memory

  // phase 2
  for (int v = v_first; v < vtot; v += splits * W) {
    const RowSrc<T> src = source(v);
    if (src.kind == 3) {   // no inverse kept: zeros right of the diagonal tile
      for (int k = src.k0 + 1; k < nta; ++k) {
        const int c = 8 * k + 2 * tq;
        store_pair(src.base + (long long)g * n + c, vec, g < src.lim && c < n, g < src.lim && c + 1 < n, 0.0, 0.0, PAIR);
      }
      continue;
    }
    if (v != v_first) rows_load<T, NT, PAIR>(xv, src, n, vec);
    double av[NT][2];
    if (src.kind == 2)
      rows_solve<T, NT, false, EXACT>(av, xv, src.k0, nta, Cs, Iv, Ct);
    else
      rows_solve<T, NT, true, EXACT>(av, xv, 0, nta, Cs, Iv, Ct);
    rows_store<T, NT, PAIR>(av, src, n, vec);
  }
}

template <typename T, int NT, bool FULL>
__global__ void __launch_bounds__(32 * (NT < 4 ? 4 : NT), NT <= 4 ? 4 : (NT <= 8 ? 2 : 1))
    k_node_rows(Problem<T> p, Level lv, int splits, int with_y, int inv) {
  const int node = blockIdx.x / splits, q = blockIdx.x - node * splits;
  const int b = node / lv.d, t = node - b * lv.d;
  pdl_wait();
  pdl_trigger();
  if (!p.active(b)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  node_rows_body<T, NT, FULL, FULL || NT <= 8>(BlockGroup{}, p, lv, b, t, smem_raw, q, splits, with_y != 0, inv != 0);
}

template <typename T>
using NodeRowsFn = void (*)(Problem<T>, Level, int, int, int);

// the kernel for block size n; full: n is a whole tile count and pairs_ok (node_rows_f32.cu, node_rows_f64.cu: one
// translation unit per type, so the instantiations compile in parallel)
template <typename T>
NodeRowsFn<T> node_rows_kernel(int n, bool full);

#define SOCU_NODE_ROWS_KERNELS(T)                      \
  template <>                                          \
  NodeRowsFn<T> node_rows_kernel<T>(int n, bool full) { \
    switch (rows_nt(n)) {                              \
      case 1: return full ? k_node_rows<T, 1, true> : k_node_rows<T, 1, false>; \
      case 2: return full ? k_node_rows<T, 2, true> : k_node_rows<T, 2, false>; \
      case 3: return full ? k_node_rows<T, 3, true> : k_node_rows<T, 3, false>; \
      case 4: return full ? k_node_rows<T, 4, true> : k_node_rows<T, 4, false>; \
      case 5: return full ? k_node_rows<T, 5, true> : k_node_rows<T, 5, false>; \
      case 6: return full ? k_node_rows<T, 6, true> : k_node_rows<T, 6, false>; \
      case 7: return full ? k_node_rows<T, 7, true> : k_node_rows<T, 7, false>; \
      case 8: return full ? k_node_rows<T, 8, true> : k_node_rows<T, 8, false>; \
      case 10: return full ? k_node_rows<T, 10, true> : k_node_rows<T, 10, false>; \
      case 12: return full ? k_node_rows<T, 12, true> : k_node_rows<T, 12, false>; \
      case 14: return full ? k_node_rows<T, 14, true> : k_node_rows<T, 14, false>; \
      default: return full ? k_node_rows<T, 16, true> : k_node_rows<T, 16, false>; \
    }                                                  \
  }

template <> NodeRowsFn<float> node_rows_kernel<float>(int n, bool full);
template <> NodeRowsFn<double> node_rows_kernel<double>(int n, bool full);

}  // namespace socu
