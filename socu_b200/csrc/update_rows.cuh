// Schur update of one separator level (n <= 128) on FP64 tensor cores.
//
//   target j = 2su - 1:  L_j -= F F^T + G^T G   (lower triangle; F left, G right of j)
//   fill-in of node t:   E[o_{l+1} + t - 1] -= F_t G_t
//
// (the reference adds both with atomics, socu/block_tridiag_solver.py:282-377;
// here every output block has one writer).  Float operands are widened in
// registers: exact products, FP64 sums, one rounding per entry.
//
// A warp owns a row of 8x8 output tiles as mma.m8n8k4 .f64 accumulators, summed
// from zero and subtracted from the output block once (starting them from the
// block instead doubled the FP64 factor's error, 5e-16 -> 1e-15).  F and G stream through shared memory in
// chunks of 32 of the contraction index, both always row-major as they lie in
// memory (16-byte copies): rows of F are read as pairs along the contraction
// (index 2t, 2t + 1, one MMA each, as in node_rows.cuh), rows of G down the
// contraction, and the two row strides put each kind of fragment load on
// distinct banks.  Two chunks are in flight, so up to n = 64 everything is
// requested at once.
//
// `splits` thread blocks share an output block on narrow levels: block q takes
// row tiles q, q + splits, ..., and `splits` warps share a row's tiles.  Every
// tile keeps its contraction order, so the bits do not depend on the split.
#pragma once

#include "sweep_rows.cuh"

namespace socu {

constexpr int kUpdKC = 32;                 // contraction chunk
constexpr int kUpdLdF = kUpdKC + 8;        // rows of F: 8 (mod 16) doubles / 8 (mod 32) floats
// rows of G (8 nt columns): 2 (mod 8) doubles / 4 (mod 16) floats
__host__ __device__ constexpr int upd_ldg(int nt, int es) {
  return es == 8 ? 8 * nt + 2 : ((nt & 1) ? 8 * nt + 12 : 8 * nt + 4);
}
__host__ __device__ constexpr int upd_stage_elems(int nt, int es) { return 8 * nt * kUpdLdF + kUpdKC * upd_ldg(nt, es); }
__host__ __device__ inline int upd_chunks(int n) { return (n + kUpdKC - 1) / kUpdKC; }
__host__ __device__ inline long long smem_update_rows_bytes(int n, int es) {
  return (long long)(upd_chunks(n) < 2 ? 1 : 2) * upd_stage_elems(rows_nt(n), es) * es;
}
// warps of a block: `splits` per row tile it owns
__host__ __device__ inline int update_rows_warps(int n, int splits) {
  return splits * (((n + 7) / 8 + splits - 1) / splits);
}

// One k-step (8 of the contraction index) of a row's tiles, four at a time.
// Target: += a F_j^T (+ h G_j); fill-in: += a G_j.  fk, gk: this lane's
// elements of row tile / column tile 0.  Tiles past jmax repeat the last one
// (split rows) or read whatever the buffer holds; their sums are dropped.
template <typename T, int NT, bool SPLIT, bool TARGET, bool HAS_G>
__device__ __forceinline__ void upd_step(double (&acc)[NT][2], const T* fk, const T* gk, int part, int splits,
                                         int jmax, double a0, double a1, double h0, double h1) {
  constexpr int ldg = upd_ldg(NT, sizeof(T)), CH = SPLIT ? 2 : 4;
#pragma unroll
  for (int jj = 0; jj < NT; jj += CH) {
    if ((SPLIT ? part + splits * jj : jj) > jmax) break;
    double x[CH][2];
    if (TARGET) {
#pragma unroll
      for (int h = 0; h < CH; ++h)
        if (jj + h < NT) {
          const int j = SPLIT ? min_i(part + splits * (jj + h), jmax) : jj + h;
          load_pair(fk + 8 * j * kUpdLdF, true, true, true, x[h][0], x[h][1]);
        }
#pragma unroll
      for (int h = 0; h < CH; ++h)
        if (jj + h < NT) mma_acc(acc[jj + h][0], acc[jj + h][1], a0, x[h][0]);
#pragma unroll
      for (int h = 0; h < CH; ++h)
        if (jj + h < NT) mma_acc(acc[jj + h][0], acc[jj + h][1], a1, x[h][1]);
    }
    if (HAS_G) {
      const double b0 = TARGET ? h0 : a0, b1 = TARGET ? h1 : a1;
#pragma unroll
      for (int h = 0; h < CH; ++h)
        if (jj + h < NT) {
          const int j = SPLIT ? min_i(part + splits * (jj + h), jmax) : jj + h;
          x[h][0] = (double)gk[8 * j];
          x[h][1] = (double)gk[ldg + 8 * j];
        }
#pragma unroll
      for (int h = 0; h < CH; ++h)
        if (jj + h < NT) mma_acc(acc[jj + h][0], acc[jj + h][1], b0, x[h][0]);
#pragma unroll
      for (int h = 0; h < CH; ++h)
        if (jj + h < NT) mma_acc(acc[jj + h][0], acc[jj + h][1], b1, x[h][1]);
    }
  }
}

// One output block, `task` in [0, update_blocks).
template <typename T, int NT, bool FULL, bool SPLIT, bool PAIR = false, class Group>
__device__ __forceinline__ void update_rows_body(const Group& grp, const Problem<T>& p, const Level& lv, int b, int task,
                                                 unsigned char* smem_raw, int q, int splits) {
  constexpr int es = sizeof(T), ldg = upd_ldg(NT, es);
  constexpr bool kAhead = NT <= 8;   // (registers: larger blocks read the output block at the end)
  const int lane = threadIdx.x & 31, warp = grp.warp(), W = grp.warps();
  const int g = lane >> 2, t = lane & 3;
  const int n = FULL ? 8 * NT : p.n, N = p.N, s = lv.s, nta = (n + 7) >> 3;
  const int U = update_targets(N, lv);
  const bool target = task < U;
  const T *F, *G;
  T* Out;
  if (target) {
    const int u = task + 1, j = 2 * s * u - 1;
    F = p.Eb(b, lv.oc + 2 * (u - 1));
    G = j + s < N ? p.Eb(b, lv.oc + 2 * u - 1) : nullptr;
    Out = p.Lb(b, j);
  } else {
    const int f = task - U + 1, i = s - 1 + 2 * s * f;
    if (i + s >= N) return;
    F = p.Eb(b, lv.oc + 2 * f);
    G = p.Eb(b, lv.oc + 2 * f - 1);
    Out = p.Eb(b, lv.on + f - 1);
  }
  const bool vec = FULL || (NT > 8 && pairs_ok(p, n));
  const int part = warp % splits, step = splits * (W / splits);
  const int first = q + splits * (warp / splits);       // this warp's first row tile
  const int last = q + splits * ((nta - 1 - q) / splits);  // the block's last row tile
  // rows of F and columns of G that the block reads
  const int lim = target ? min_i(n, 8 * (last + 1)) : n;
  T* buf = reinterpret_cast<T*>(smem_raw);
  const int chunks = upd_chunks(n);
  auto stage = [&](int c) {
    T* Fs = buf + (c & 1) * upd_stage_elems(NT, es);
    T* Gs = Fs + 8 * NT * kUpdLdF;
    const int k0 = c * kUpdKC, kw = min_i(kUpdKC, n - k0);
    if (target || splits == 1) {
      async_load_by(grp.tid(), grp.threads(), Fs, kUpdLdF, F + k0, lim, kw, n);
    } else {
      for (int i = q; i < nta; i += splits)
        async_load_by(grp.tid(), grp.threads(), Fs + 8 * i * kUpdLdF, kUpdLdF, F + (long long)8 * i * n + k0, min_i(8, n - 8 * i), kw, n);
    }
    if (G) async_load_by(grp.tid(), grp.threads(), Gs, ldg, G + (long long)k0 * n, kw, lim, n);
    const int kp = (kw + 7) & ~7;   // zeros up to a whole k-step
    if (kp > kw) {
      for (int e = grp.tid(); e < 8 * nta * (kp - kw); e += grp.threads())
        Fs[(e / (kp - kw)) * kUpdLdF + kw + e % (kp - kw)] = T(0);
      if (G)
        for (int e = grp.tid(); e < 8 * nta * (kp - kw); e += grp.threads())
          Gs[(kw + e / (8 * nta)) * ldg + e % (8 * nta)] = T(0);
    }
    cp_async_commit();
  };
  int requested = 0;   // chunks
  bool staged = false;   // all chunks have arrived (n <= 64: later rows need no barrier)
  for (int i = first; i < nta || !staged; i += step) {
    const bool on = i < nta;
    const int jmax = target ? i : nta - 1;   // last tile of the row
    const int gr = 8 * i + g;
    double acc[NT][2];
    T out[kAhead ? NT : 1][2];   // the output block's entries, requested before the products
#pragma unroll
    for (int jj = 0; jj < NT; ++jj) {
      acc[jj][0] = acc[jj][1] = 0.0;
      const int j = part + splits * jj, c = 8 * j + 2 * t;
      if (kAhead && on && j <= jmax)
        load_raw(Out + (long long)gr * n + c, vec, gr < n && c < n, gr < n && c + 1 < n, out[kAhead ? jj : 0], PAIR);
    }
    for (int c = 0; c < chunks; ++c) {
      if (!staged) {
        // two chunks ahead (one call: the staging code is large, and the steps
        // around it should stay in the instruction cache)
        while (requested < chunks && requested < c + 2) {
          if (requested > 1) grp.sync();   // its buffer is free again
          stage(requested++);
        }
        if (c + 1 < chunks)
          cp_async_wait_one();
        else
          cp_async_wait_all();
        grp.sync();
      }
      if (on) {
        const T* Fs = buf + (c & 1) * upd_stage_elems(NT, es);
        const T* Gs = Fs + 8 * NT * kUpdLdF;
        const int ks = (min_i(kUpdKC, n - c * kUpdKC) + 7) >> 3;
        const T* fk = Fs + g * kUpdLdF + 2 * t;   // F rows: pairs along the contraction
        const T* gk = Gs + 2 * t * ldg + g;       // G rows: down the contraction
#pragma unroll 1
        for (int kk = 0; kk < ks; ++kk, fk += 8, gk += 8 * ldg) {
          double a0, a1, h0 = 0.0, h1 = 0.0;
          load_pair(fk + 8 * i * kUpdLdF, true, true, true, a0, a1);
          if (target && G) {
            h0 = (double)gk[8 * i];
            h1 = (double)gk[ldg + 8 * i];
          }
          if (!target)
            upd_step<T, NT, SPLIT, false, true>(acc, fk, gk, part, splits, jmax, a0, a1, h0, h1);
          else if (G)
            upd_step<T, NT, SPLIT, true, true>(acc, fk, gk, part, splits, jmax, a0, a1, h0, h1);
          else
            upd_step<T, NT, SPLIT, true, false>(acc, fk, gk, part, splits, jmax, a0, a1, h0, h1);
        }
      }
    }
    staged = true;
    if (on) {
#pragma unroll
      for (int jj = 0; jj < NT; ++jj) {
        const int j = part + splits * jj, c = 8 * j + 2 * t;
        if (j <= jmax) {
          const bool diag = target && j == i;   // only the lower triangle of a target is written
          T o[2];
          if (kAhead) {
            o[0] = out[kAhead ? jj : 0][0];
            o[1] = out[kAhead ? jj : 0][1];
          } else {
            load_raw(Out + (long long)gr * n + c, vec, gr < n && c < n, gr < n && c + 1 < n, o);
          }
          store_pair(Out + (long long)gr * n + c, vec && !diag, gr < n && c < n && (!diag || c <= gr),
                     gr < n && c + 1 < n && (!diag || c + 1 <= gr), (double)o[0] - acc[jj][0],
                     (double)o[1] - acc[jj][1], PAIR && !diag);
        }
      }
    }
  }
}

// The first `upd` blocks update; any others are the forward pull that factor_and_solve needs of the
// same nodes, `chunks` blocks of `cols` right-hand sides to a vector of level `next`.
template <typename T, int NT, bool FULL>
__global__ void __launch_bounds__(NT <= 8 ? 256 : 512, NT <= 8 ? 2 : 1)
    k_update_rows(Problem<T> p, Level lv, int splits, int upd, Level next, int chunks, int cols) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if ((int)blockIdx.x >= upd) {
    const int v = (blockIdx.x - upd) / chunks, q = blockIdx.x - upd - v * chunks;
    const int per_b = sweep_tasks<kModePull>(p.N, next), b = v / per_b;
    if (p.active(b))
      sweep_rows_body<T, NT, FULL, kModePull, true, true>(BlockGroup{}, p, next, b, v - b * per_b, smem_raw, kWaitNone,
                                                          q * cols, cols);
    return;
  }
  const int block = blockIdx.x / splits, q = blockIdx.x - block * splits;
  const int per_b = update_blocks(p.N, lv);
  const int b = block / per_b, task = block - b * per_b;
  if (!p.active(b)) return;
  if (splits > 1)
    update_rows_body<T, NT, FULL, true>(BlockGroup{}, p, lv, b, task, smem_raw, q, splits);
  else
    update_rows_body<T, NT, FULL, false>(BlockGroup{}, p, lv, b, task, smem_raw, 0, 1);
}

template <typename T>
using UpdateRowsFn = void (*)(Problem<T>, Level, int, int, Level, int, int);

template <typename T>
UpdateRowsFn<T> update_rows_kernel(int n, bool full);

#define SOCU_UPDATE_ROWS_KERNELS(T)                    \
  template <>                                          \
  UpdateRowsFn<T> update_rows_kernel<T>(int n, bool full) { \
    switch (rows_nt(n)) {                              \
      case 1: return full ? k_update_rows<T, 1, true> : k_update_rows<T, 1, false>; \
      case 2: return full ? k_update_rows<T, 2, true> : k_update_rows<T, 2, false>; \
      case 3: return full ? k_update_rows<T, 3, true> : k_update_rows<T, 3, false>; \
      case 4: return full ? k_update_rows<T, 4, true> : k_update_rows<T, 4, false>; \
      case 5: return full ? k_update_rows<T, 5, true> : k_update_rows<T, 5, false>; \
      case 6: return full ? k_update_rows<T, 6, true> : k_update_rows<T, 6, false>; \
      case 7: return full ? k_update_rows<T, 7, true> : k_update_rows<T, 7, false>; \
      case 8: return full ? k_update_rows<T, 8, true> : k_update_rows<T, 8, false>; \
      case 10: return full ? k_update_rows<T, 10, true> : k_update_rows<T, 10, false>; \
      case 12: return full ? k_update_rows<T, 12, true> : k_update_rows<T, 12, false>; \
      case 14: return full ? k_update_rows<T, 14, true> : k_update_rows<T, 14, false>; \
      default: return full ? k_update_rows<T, 16, true> : k_update_rows<T, 16, false>; \
    }                                                  \
  }

template <> UpdateRowsFn<float> update_rows_kernel<float>(int n, bool full);
template <> UpdateRowsFn<double> update_rows_kernel<double>(int n, bool full);

}  // namespace socu
