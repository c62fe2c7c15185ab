// Device-side building blocks of the nested-dissection block-tridiagonal
// Cholesky (sm_100a).  Everything here works on one CTA's shared memory.
//
// Storage contract (identical to socu, socu/block_tridiag_solver.py:739-774):
//   L  (B, N, n, n)   diagonal blocks, lower triangle read, factor written
//   E  (B, S, n, n)   off-diagonal storage, S = off_diag_storage_len(N)
//   X  (B, N, n, m)   right-hand sides in, solution out
// Level l has stride s = 2^l and nodes i = s-1 + 2 s t, t < (N+s)/(2s)
// (socu/block_tridiag_solver.py:174).  Slot E[o_l + k] couples node
// p = (k+1)s-1 (columns) with q = p+s (rows).
//
// Factor output: lower(L_i) = C_i (lower Cholesky factor).  The strict upper
// triangle is 0, or holds W_i^T with W_i = C_i^{-1} where a path keeps the
// diagonal inverses (factor_and_solve, the internal float factor of the mixed
// solve).  The reference leaves the upper triangle unspecified and every
// kernel here that is given a factor from outside reads only lower(L_i), so
// factors are interchangeable with socu's.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace socu {

constexpr unsigned kFull = 0xffffffffu;

template <typename T> __device__ __forceinline__ T rsqrt_t(T x);
template <> __device__ __forceinline__ double rsqrt_t<double>(double x) { return rsqrt(x); }
template <> __device__ __forceinline__ float rsqrt_t<float>(float x) { return rsqrtf(x); }

template <typename T>
struct Problem {
  T* L;
  T* E;
  T* X;                  // may be null (factor only)
  const uint8_t* mask;   // may be null: all batch entries active
  int* info;             // may be null: per batch entry, 0 or 1 + the first node whose pivot failed
  int B, N, n, m, S;
  long long sL, sE, sX;  // per-batch strides in elements

  __device__ __forceinline__ T* Lb(int b, int i) const {
    return L + (long long)b * sL + (long long)i * n * n;
  }
  __device__ __forceinline__ T* Eb(int b, int slot) const {
    return E + (long long)b * sE + (long long)slot * n * n;
  }
  __device__ __forceinline__ T* Xb(int b, int i) const {
    return X + (long long)b * sX + (long long)i * n * m;
  }
  __device__ __forceinline__ bool active(int b) const { return mask == nullptr || mask[b] != 0; }
};

// Numerical status of one batch entry: node i failed to factor (a pivot
// <= 0, or a non-finite value).  info keeps the failing node that comes first
// in elimination order -- lowest level ctz(i+1), then lowest index -- so the
// result does not depend on which node of a level reports first.  LAPACK's
// potrf reports the failing column the same way (info > 0); the reference
// reports nothing (socu/blas/potrf.py:97-117 takes the square root of
// whatever pivot it meets).
__device__ __forceinline__ void record_failure(int* info, int i) {
  const int mine = i + 1;
  int cur = *reinterpret_cast<volatile int*>(info);
  while (true) {
    if (cur != 0) {
      const int lc = __ffs(cur) - 1, lm = __ffs(mine) - 1;
      if (lc < lm || (lc == lm && cur <= mine)) return;
    }
    const int prev = atomicCAS(info, cur, mine);
    if (prev == cur) return;
    cur = prev;
  }
}

// After the blocked Cholesky of node i (lower(A) = C, leading dimension lda):
// every diagonal entry must be a positive finite number.  All threads call it.
template <typename T>
__device__ __forceinline__ void check_factor(const Problem<T>& p, int b, int i, const T* A, int lda) {
  if (p.info == nullptr) return;
  bool bad = false;
  for (int r = threadIdx.x; r < p.n; r += blockDim.x) {
    const T d = A[r * lda + r];
    bad = bad || !(d > T(0)) || isinf(d);
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) record_failure(p.info + b, i);
}

// One nested-dissection level (socu/block_tridiag_solver.py:869-914).
struct Level {
  int s;    // stride 2^l
  int d;    // nodes at this level, (N+s)/(2s)
  int oc;   // offset of this level's slots
  int on;   // offset of the next level's slots
  int op;   // offset of the previous level's slots (unused at level 0)
};

// Programmatic dependent launch (sm_90+).  A kernel launched with the
// programmatic-serialization attribute may start while its predecessor in the
// stream is still running; pdl_wait() returns once the predecessor grid has
// completed and its memory is visible, pdl_trigger() lets the successor start
// launching.  Both are no-ops for kernels launched without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// ---------------------------------------------------------------------------
// Asynchronous global -> shared copies (cp.async, element granular so that
// padded shared layouts are allowed).  Issue everything, then wait once.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

template <int BYTES>
__device__ __forceinline__ void cp_async_bytes(void* dst, const void* src) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_addr(dst)), "l"(src), "n"(BYTES) : "memory");
}

template <typename T>
__device__ __forceinline__ void cp_async_elem(T* dst, const T* src) {
  cp_async_bytes<sizeof(T)>(dst, src);
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// widest copy (16, 8 or element bytes) that keeps every row chunk aligned
template <typename T>
__device__ __forceinline__ int copy_width(const T* dst, int ld, const T* src, int cols, long long src_ld) {
  const unsigned long long a = reinterpret_cast<unsigned long long>(src) |
                               (unsigned long long)smem_addr(dst) |
                               (unsigned long long)(cols * sizeof(T)) | (unsigned long long)(ld * sizeof(T)) |
                               (unsigned long long)(src_ld * (long long)sizeof(T));
  return (a & 15) == 0 ? 16 : ((a & 7) == 0 ? 8 : (int)sizeof(T));
}

template <typename T, int BYTES>
__device__ __forceinline__ void async_load_w(int tid, int threads, T* dst, int ld, const T* src, int rows, int cols,
                                             long long src_ld) {
  constexpr int V = BYTES / sizeof(T);
  const int cv = cols / V;
  // element tid, tid + threads, ... of the rows x cv copies, without a division each
  const int dr = threads / cv, dc = threads - dr * cv;
  int r = tid / cv, c = tid - r * cv;
#pragma unroll 2
  while (r < rows) {
    cp_async_bytes<BYTES>(dst + r * ld + c * V, src + (long long)r * src_ld + c * V);
    r += dr;
    c += dc;
    if (c >= cv) {
      c -= cv;
      ++r;
    }
  }
}

// dst[r*ld + c] = src[r*src_ld + c] by `threads` threads; vectorised when alignment allows
template <typename T>
__device__ __forceinline__ void async_load_by(int tid, int threads, T* dst, int ld, const T* src, int rows, int cols,
                                              long long src_ld) {
  const int w = copy_width(dst, ld, src, cols, src_ld);
  if (w == 16)
    async_load_w<T, 16>(tid, threads, dst, ld, src, rows, cols, src_ld);
  else if (w == 8)
    async_load_w<T, 8>(tid, threads, dst, ld, src, rows, cols, src_ld);
  else
    async_load_w<T, sizeof(T)>(tid, threads, dst, ld, src, rows, cols, src_ld);
}
template <typename T>
__device__ __forceinline__ void async_load(T* dst, int ld, const T* src, int rows, int cols, long long src_ld) {
  async_load_by(threadIdx.x, blockDim.x, dst, ld, src, rows, cols, src_ld);
}

// FP64 tensor-core product of 8x8x4 (mma.m8n8k4 .f64).  Fragments (PTX ISA): A a0 = A[g][t],
// B b0 = B[t][g], C {c0, c1} = C[g][2t + {0, 1}] with g = lane / 4, t = lane % 4.
__device__ __forceinline__ void dmma_8x8x4(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// ---------------------------------------------------------------------------
// Trailing update of one 8-column step of cta_chol_solve, both parts in one
// tile loop (rows R0..n-1, P = A[R0.., K..K+kb) the solved panel):
//   A22[r][c] -= sum_k P[r][k] P[c][k]        (c <= r)
//   V[r][c]   -= sum_k P[r][k] V[K+k][c]      (c < nv)
// The accumulators start from the target values and the panel operand is
// negated, so a tile ends in a plain store.  FP64: DMMA warp tiles of 16 x 32
// (fragment layout of mma.m8n8k4 .f64: a0 = A[g][t], b0 = B[t][g],
// {c0, c1} = C[g][2t + {0, 1}], g = lane/4, t = lane%4).  FP32: 4 x 4 SIMT
// micro-tiles per thread.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void rank_update_simt(T* A, int lda, T* V, int ldv, int n, int K, int kb, int R0, int nv) {
  constexpr int BK = 8;
  const int M = n - R0;
  const int tm = (M + 3) / 4;
  const int tnA = (M + 3) / 4, tnV = (nv + 3) / 4;
  const int nA = tm * tnA, total = nA + tm * tnV;
  const T* P = A + R0 * lda + K;
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const bool isA = idx < nA;
    const int tt = isA ? idx : idx - nA;
    const int tn = isA ? tnA : tnV;
    const int r0 = (tt / tn) * 4, c0 = (tt % tn) * 4;
    if (isA && c0 > r0 + 3) continue;
    T* C = isA ? A + R0 * lda + R0 : V + R0 * ldv;
    const int ldc = isA ? lda : ldv;
    const int N = isA ? M : nv;
    T acc[4][4];
    int ra[4], cb[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) ra[i] = min(r0 + i, M - 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) cb[j] = min(c0 + j, N - 1);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = C[ra[i] * ldc + cb[j]];
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      if (k < kb) {
        T a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = P[ra[i] * lda + k];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = isA ? P[cb[j] * lda + k] : V[(K + k) * ldv + cb[j]];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fma(-a[i], b[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = r0 + i, c = c0 + j;
        if (r < M && c < N && (!isA || c <= r)) C[r * ldc + c] = acc[i][j];
      }
  }
}

// ---------------------------------------------------------------------------
// CTA: blocked right-looking Cholesky of the n x n block in A fused with the
// solve C V = V for nv vectors (columns of V), by 8-column blocks.
//   1. every thread loads the diagonal block into registers and factors it
//      redundantly: no communication on the critical chain;
//   2. one thread per item solves against that block: each row of the panel
//      below it (A21 <- A21 C11^{-T}) and each vector segment
//      (V1 <- C11^{-1} V1) -- the same forward substitution;
//   3. trailing updates A22 -= P P^T (lower) and V2 -= P V1 with
//      P = the solved panel (tensor cores for double).
// On exit lower(A) = C.  Two barriers per block.
// ---------------------------------------------------------------------------
// IDENTITY: V starts as the n x n identity (nv = n), so it ends as C^{-1}.
// Rows [K, K+kb) of column c are still zero for c >= K+kb, which leaves those
// columns out of the item solves and of the trailing update.
template <typename T, bool IDENTITY = false>
__device__ void cta_chol_solve(T* A, int lda, int n, T* V, int ldv, int nv) {
  // diagonal block width: the whole block lives in every thread's registers
  // and is factored redundantly by every thread (work grows as BK^3 x threads)
  constexpr int BK = 8;
  const int nv_all = nv;
  for (int K = 0; K < n; K += BK) {
    const int kb = min(BK, n - K);
    const int R0 = K + kb, rows = n - R0;
    if (IDENTITY) nv = min(nv_all, R0);
    // 1. diagonal block in registers (identity-padded past kb), only in the
    //    threads that own an item (thread 0 always: it writes the block back)
    T c[BK][BK], rsv[BK];
    const bool act = threadIdx.x < max(rows + nv, 1);
    if (act) {
#pragma unroll
    for (int i = 0; i < BK; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j)
        c[i][j] = (i < kb) ? A[(K + i) * lda + K + j] : (i == j ? T(1) : T(0));
#pragma unroll
    for (int j = 0; j < BK; ++j) {
      const T r = rsqrt_t(c[j][j]);
      rsv[j] = r;
      c[j][j] *= r;
#pragma unroll
      for (int i = j + 1; i < BK; ++i) c[i][j] *= r;
#pragma unroll
      for (int i = j + 1; i < BK; ++i)
#pragma unroll
        for (int l = j + 1; l <= i; ++l) c[i][l] = fma(-c[i][j], c[l][j], c[i][l]);
    }
    // 2. forward substitution of every item against the diagonal block
    for (int it = threadIdx.x; it < rows + nv; it += blockDim.x) {
      T* base;
      int stride;
      if (it < rows) {
        base = A + (R0 + it) * lda + K;   // panel row: contiguous columns
        stride = 1;
      } else {
        base = V + K * ldv + (it - rows); // vector segment: rows of V
        stride = ldv;
      }
      T x[BK];
#pragma unroll
      for (int j = 0; j < BK; ++j) x[j] = j < kb ? base[j * stride] : T(0);
#pragma unroll
      for (int j = 0; j < BK; ++j) {
#pragma unroll
        for (int i = 0; i < j; ++i) x[j] = fma(-x[i], c[j][i], x[j]);
        x[j] *= rsv[j];
      }
#pragma unroll
      for (int j = 0; j < BK; ++j)
        if (j < kb) base[j * stride] = x[j];
    }
    }
    __syncthreads();
    // 3. write the factored diagonal block (one thread, static register
    //    indices), then the trailing updates
    if (threadIdx.x == 0) {
#pragma unroll
      for (int i = 0; i < BK; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j)
          if (i < kb) A[(K + i) * lda + K + j] = c[i][j];
    }
    if (R0 < n) {
      rank_update_simt<T>(A, lda, V, ldv, n, K, kb, R0, nv);
    }
    __syncthreads();
  }
}

}  // namespace socu
