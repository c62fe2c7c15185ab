// Substitution sweeps (n <= 128): one thread block per vector, one warp per
// 8-row tile of it, products on FP64 tensor cores (mma.m8n8k4 .f64; float
// factors and vectors are widened, one rounding per result).
//
//   forward (level l >= 1):  y_j -= F y_{j-s/2} + G^T y_{j+s/2}, then at the
//                            level's own nodes  y_j <- C_j^{-1} y_j
//   forward (level 0):       y_i <- C_i^{-1} y_i
//   backward:                x_i -= F^T x_{i+s} + G x_{i-s};  x_i <- C_i^{-T} x_i
//   pull:                    the coupling part of a forward level alone
// (socu/block_tridiag_solver.py:425-736)
//
// A sweep reads every block once and no element of a block is needed by two
// warps, so the blocks are not staged: each lane loads its MMA operands from
// global memory straight into registers (row-major blocks as pairs along the
// contraction, transposed ones down it; both fill whole 32-byte sectors) and,
// up to n = 64, holds a whole row tile of all three blocks before the vectors
// of the previous level are needed.  Only the vectors go through shared memory.
//
// On a factor that carries W = C^{-1} (INV) the solve is one more product.
// Otherwise it is a substitution by 8-row tiles: the warps take turns; in FP64 a
// lane solves a column against the tile, for floats the tile's FP64 inverse is an operand.
#pragma once

#include "node_rows.cuh"

namespace socu {

enum SweepMode { kModeForward = 0, kModeBackward = 1, kModePull = 2 };
// how the kernel meets the one before it (programmatic dependent launch)
enum SweepWait {
  kWaitNone = 0,    // called inside another kernel
  kWaitFirst = 1,   // the blocks themselves come from the previous kernel
  kWaitVectors = 2  // the blocks were complete before: only the vectors are waited for
};
// columns per pass: 8 up to n = 64, where the blocks stay in registers between passes, else 32
__host__ __device__ constexpr int sweep_cols(int nt) { return nt <= 8 ? 8 : 32; }
// stride of a staged vector row: 2 (mod 8) doubles, so the two rows of an operand pair and the
// next three pairs of a half warp are on distinct banks
__host__ __device__ constexpr int sweep_ldz(int nt) { return sweep_cols(nt) + 2; }
__host__ __device__ inline long long smem_sweep_rows_bytes(int n, bool inv) {
  const int nt = rows_nt(n);
  return 8LL * (3LL * 8 * nt * sweep_ldz(nt) + (inv ? 0 : 64LL * nt));
}

// two consecutive elements through L2 (another block may have written them in this kernel's lifetime)
template <typename T>
__device__ __forceinline__ void ldcg_pair(const T* p, bool vec, bool v0, bool v1, double& x0, double& x1) {
  if (vec) {
    if constexpr (sizeof(T) == 8) {
      const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
      x0 = v.x;
      x1 = v.y;
    } else {
      const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
      x0 = (double)v.x;
      x1 = (double)v.y;
    }
  } else {
    x0 = v0 ? (double)__ldcg(p) : 0.0;
    x1 = v1 ? (double)__ldcg(p + 1) : 0.0;
  }
}

// MMA operand of an n x n block, row tile i, column tile kk: elements (r, c), (r, c + 1) with
// r = 8i + g, c = 8kk + 2t; TR: of the block's transpose.  vec: the tile is whole (and pairs are aligned);
// pair: rows_paired.
template <typename T, bool TR>
__device__ __forceinline__ void block_frag(const T* M, int n, int i, int kk, bool vec, T& a0, T& a1,
                                           bool pair = false) {
  const int lane = threadIdx.x & 31, r = 8 * i + (lane >> 2), c = 8 * kk + 2 * (lane & 3);
  if (TR) {
    const T* q = M + (c * n + r);   // (n <= 128: offsets inside a block fit 32 bits)
    a0 = vec || (r < n && c < n) ? q[0] : T(0);
    a1 = vec || (r < n && c + 1 < n) ? q[n] : T(0);
  } else if (pair && !vec && !(r < n && c < n)) {
    a0 = a1 = T(0);
  } else if (vec || pair) {
    if constexpr (sizeof(T) == 8) {
      const double2 v = *reinterpret_cast<const double2*>(M + (r * n + c));
      a0 = v.x;
      a1 = v.y;
    } else {
      const float2 v = *reinterpret_cast<const float2*>(M + (r * n + c));
      a0 = v.x;
      a1 = v.y;
    }
  } else {
    a0 = (r < n && c < n) ? M[r * n + c] : T(0);
    a1 = (r < n && c + 1 < n) ? M[r * n + c + 1] : T(0);
  }
}

// Operand of the solve, row tile i, column tile kk (0 outside its strict triangle).
//   INV forward: W (strictly upper L transposed), backward: W^T; their diagonal, 1 / C[r][r], is
//   a factor of its own (solve_diag).
//   Else forward: C left of the diagonal tile, backward: C^T right of it.
template <typename T, bool BWD, bool INV>
__device__ __forceinline__ void solve_frag(const T* L, int n, int i, int kk, bool vec, T& a0, T& a1, bool pair) {
  a0 = a1 = T(0);
  if (BWD ? kk < i : kk > i) return;
  if (kk != i) {
    block_frag<T, INV != BWD>(L, n, i, kk, vec, a0, a1, pair);
    return;
  }
  if (!INV) return;
  const int lane = threadIdx.x & 31, r = 8 * i + (lane >> 2), c = 8 * i + 2 * (lane & 3);
  T a[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int k = c + e;
    a[e] = r < n && k < n && (BWD ? k > r : k < r) ? (BWD ? L[r * n + k] : L[k * n + r]) : T(0);
  }
  a0 = a[0];
  a1 = a[1];
}
// diagonal of C in this lane's row of row tile i
template <typename T>
__device__ __forceinline__ T solve_diag(const T* L, int n, int i) {
  const int r = 8 * i + ((threadIdx.x & 31) >> 2);
  return r < n ? L[r * n + r] : T(1);
}

// One vector, its columns col0 .. col0 + cols (a multiple of 8).  ONE: the block has a warp per
// row tile (else the warps loop over them and the blocks are read as they are used).
template <typename T, int NT, bool FULL, int MODE, bool INV, bool ONE, bool EXACT = (NT <= 8), bool PAIR = false,
          class Group>
__device__ __forceinline__ void sweep_rows_body(const Group& grp, const Problem<T>& p, const Level& lv, int b, int task,
                                                unsigned char* smem_raw, int wait, int col0 = 0,
                                                int cols = 1 << 30) {
  constexpr bool BWD = MODE == kModeBackward, KEEP = ONE && NT <= 8;
  constexpr int XC = sweep_cols(NT), CG = XC / 8, ldz = sweep_ldz(NT), NK = KEEP ? NT : 1;
  static_assert(INV || ONE, "the substitution needs a warp per row tile");
  const int lane = threadIdx.x & 31, warp = grp.warp(), W = grp.warps();
  const int g = lane >> 2, t = lane & 3;
  const int n = FULL ? 8 * NT : p.n, m = p.m, N = p.N, s = lv.s, nta = (n + 7) >> 3;
  // the vector, the row-major block P with its vector and the transposed block Q with its
  int j, jp = 0, jq = 0;
  bool solve = MODE != kModePull;
  const T *P = nullptr, *Q = nullptr;
  if (BWD) {
    j = s - 1 + 2 * s * task;
    jp = j - s;
    jq = j + s;
    if (j >= s) P = p.Eb(b, lv.oc + 2 * task - 1);
    if (j + s < N) Q = p.Eb(b, lv.oc + 2 * task);
  } else if (s == 1) {
    j = 2 * task;
  } else {
    const int u = task + 1, h = s / 2;
    j = s * u - 1;
    jp = j - h;
    jq = j + h;
    P = p.Eb(b, lv.op + 2 * u - 2);
    if (jq < N) Q = p.Eb(b, lv.op + 2 * u - 1);
    solve = MODE == kModeForward && (u & 1) != 0;
  }
  const T* L = p.Lb(b, j);
  T* yj = p.Xb(b, j);
  const bool vec = FULL || (!EXACT && pairs_ok(p, n));
  const bool vecx = (m & 1) == 0 && (reinterpret_cast<uintptr_t>(p.X) & (2 * sizeof(T) - 1)) == 0;
  double* Zp = reinterpret_cast<double*>(smem_raw);
  double* Zq = Zp + 8 * NT * ldz;
  double* Rs = Zq + 8 * NT * ldz;
  double* Iv = Rs + 8 * NT * ldz;

  if (wait == kWaitFirst) pdl_wait();
  // fs: the solve's operands, by column tile (INV) or by step of the substitution; larger
  // blocks read them four steps at a time as they are used
  T fp[NK][2], fq[NK][2], fs[KEEP ? NT : 4][2], dc = T(1);
  auto load_solve = [&](int e0) {
#pragma unroll
    for (int e = 0; e < (KEEP ? NT : 4); ++e) {
      const int kk = INV || !BWD ? e0 + e : nta - 1 - e0 - e;
      T f0 = T(0), f1 = T(0);
      if (kk >= 0 && kk < nta) solve_frag<T, BWD, INV>(L, n, warp, kk, vec, f0, f1, PAIR);
      fs[e][0] = f0;
      fs[e][1] = f1;
    }
  };
  if (KEEP && warp < nta) {
#pragma unroll
    for (int kk = 0; kk < NT; ++kk) {
      if (P) block_frag<T, false>(P, n, warp, kk, vec && kk < nta, fp[KEEP ? kk : 0][0], fp[KEEP ? kk : 0][1], PAIR);
      if (Q) block_frag<T, true>(Q, n, warp, kk, vec && kk < nta, fq[KEEP ? kk : 0][0], fq[KEEP ? kk : 0][1]);
    }
    if (solve) {
      load_solve(0);
      if (INV) dc = solve_diag(L, n, warp);
    }
  }
  if (!KEEP && solve)   // the solve's block is read after the products: into L2 meanwhile
    for (int e = grp.tid() * (128 / (int)sizeof(T)); e < n * n; e += grp.threads() * (128 / (int)sizeof(T)))
      asm volatile("prefetch.global.L2 [%0];\n" ::"l"(L + e));
  // The diagonal tile, for its own warp.  FP64: the tile with its pivots' reciprocals (forward: its
  // transpose; padding: an identity), against which a lane solves a column.  Float: its inverse in
  // FP64, exact beyond float's rounding, as an operand (i0, i1; transposed for the backward sweep).
  constexpr bool SUBST = sizeof(T) == 8;
  double* D = Iv + 64 * warp;
  double i0 = 0.0, i1 = 0.0;
  if (!INV && solve && warp < nta) {
    T d0, d1;
    block_frag<T, false>(L, n, warp, warp, vec, d0, d1, PAIR);
    const int r = 8 * warp + g, c = 8 * warp + 2 * t;
    const double v0 = r >= n && r == c ? 1.0 : (double)d0, v1 = r >= n && r == c + 1 ? 1.0 : (double)d1;
    if (SUBST) {
      D[BWD ? 8 * g + 2 * t : 16 * t + g] = r == c ? 1.0 / v0 : v0;
      D[BWD ? 8 * g + 2 * t + 1 : 16 * t + 8 + g] = r == c + 1 ? 1.0 / v1 : v1;
    } else {
      // every lane: column lane % 8 of C_kk^{-1}
      D[2 * lane] = v0;
      D[2 * lane + 1] = v1;
      __syncwarp();
      double y[8], rd[8];
#pragma unroll
      for (int a = 0; a < 8; ++a) rd[a] = 1.0 / D[9 * a];
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        double v = a == (lane & 7) ? 1.0 : 0.0;
#pragma unroll
        for (int c = 0; c < a; ++c) v = fma(-D[8 * a + c], y[c], v);
        y[a] = v * rd[a];
      }
      __syncwarp();
#pragma unroll
      for (int a = 0; a < 8; ++a) D[8 * a + (lane & 7)] = y[a];
      __syncwarp();
      i0 = BWD ? D[8 * (2 * t) + g] : D[8 * g + 2 * t];
      i1 = BWD ? D[8 * (2 * t + 1) + g] : D[8 * g + 2 * t + 1];
    }
    __syncwarp();
  }
  if (wait == kWaitVectors) pdl_wait();
  if (wait == kWaitFirst || wait == kWaitVectors) pdl_trigger();

  const int cend = cols < m - col0 ? col0 + cols : m;
  for (int c0 = col0; c0 < cend; c0 += XC) {
    const int mc = min_i(XC, cend - c0), groups = (mc + 7) >> 3;
    if (c0 > col0) grp.sync();
    // neighbours' vectors, zeros outside (KEEP's products run over all NT tiles: a zero operand
    // does not cancel a NaN that an earlier kernel left in shared memory)
    if (P || Q) {
      const int w = CG == 1 ? 8 : 8 * groups;   // (a constant up to n = 64: no division)
      for (int e = grp.tid(); e < 8 * (KEEP ? NT : nta) * w; e += grp.threads()) {
        const int k = e / w, c = e - k * w;
        const bool in = k < n && c < mc;
        const long long o = (long long)k * m + c0 + c;
        if (P) Zp[k * ldz + c] = in ? (double)__ldcg(p.Xb(b, jp) + o) : 0.0;
        if (Q) Zq[k * ldz + c] = in ? (double)__ldcg(p.Xb(b, jq) + o) : 0.0;
      }
    }
    double ys[ONE ? CG : 1][2];
    if (ONE && CG == 1 && warp < nta) {   // (with four column groups the registers are short: after the products)
      const int r = 8 * warp + g, c = c0 + 2 * t;
      ldcg_pair(yj + (long long)r * m + c, vecx && r < n && c < m, r < n && c < m, r < n && c + 1 < m, ys[0][0], ys[0][1]);
    }
    grp.sync();
    for (int i = warp; i < nta; i += ONE ? 8 * NT : W) {
      // one column group: a chain of MMAs per block; four groups are four chains as they are
      double ap[CG][2], aq[1][2] = {{0.0, 0.0}};
#pragma unroll
      for (int q = 0; q < CG; ++q) ap[q][0] = ap[q][1] = 0.0;
      auto products = [&](int kk, T f0, T f1, T h0, T h1) {
        const int zo = (8 * kk + 2 * t) * ldz + g;
#pragma unroll
        for (int q = 0; q < CG; ++q) {
          if (CG == 1 || q < groups) {
            if (P) {
              mma_acc(ap[q][0], ap[q][1], (double)f0, Zp[zo + 8 * q]);
              mma_acc(ap[q][0], ap[q][1], (double)f1, Zp[zo + ldz + 8 * q]);
            }
            if (Q) {
              double(&ac)[2] = CG == 1 ? aq[0] : ap[q];
              mma_acc(ac[0], ac[1], (double)h0, Zq[zo + 8 * q]);
              mma_acc(ac[0], ac[1], (double)h1, Zq[zo + ldz + 8 * q]);
            }
          }
        }
      };
      if (KEEP) {
        if (P || Q)
#pragma unroll
          for (int kk = 0; kk < NT; ++kk)
            products(kk, fp[KEEP ? kk : 0][0], fp[KEEP ? kk : 0][1], fq[KEEP ? kk : 0][0], fq[KEEP ? kk : 0][1]);
      } else if (P || Q) {
        // batches of operands, the next one requested before this one's products
        constexpr int BK = 4;
        T fb[BK][4];
        auto fetch = [&](T (&f)[BK][4], int k0) {
#pragma unroll
          for (int h = 0; h < BK; ++h) {
            f[h][0] = f[h][1] = f[h][2] = f[h][3] = T(0);
            if (k0 + h < nta) {
              if (P) block_frag<T, false>(P, n, i, k0 + h, vec, f[h][0], f[h][1], PAIR);
              if (Q) block_frag<T, true>(Q, n, i, k0 + h, vec, f[h][2], f[h][3]);
            }
          }
        };
        fetch(fb, 0);
        for (int k0 = 0; k0 < nta; k0 += BK) {
          T cur[BK][4];
#pragma unroll
          for (int h = 0; h < BK; ++h)
#pragma unroll
            for (int e = 0; e < 4; ++e) cur[h][e] = fb[h][e];
          if (k0 + BK < nta) fetch(fb, k0 + BK);
#pragma unroll
          for (int h = 0; h < BK; ++h)
            if (k0 + h < nta) products(k0 + h, cur[h][0], cur[h][1], cur[h][2], cur[h][3]);
        }
      }
#pragma unroll
      for (int q = 0; q < CG; ++q) {
        if (CG > 1 && q >= groups) break;
        const int r = 8 * i + g, c = c0 + 8 * q + 2 * t;
        const bool ok0 = r < n && c < m, ok1 = r < n && c + 1 < m;
        double y0, y1;
        if (ONE && CG == 1) {
          y0 = ys[0][0];
          y1 = ys[0][1];
        } else {
          ldcg_pair(yj + (long long)r * m + c, vecx && ok0, ok0, ok1, y0, y1);
        }
        y0 -= ap[q][0] + (CG == 1 ? aq[0][0] : 0.0);
        y1 -= ap[q][1] + (CG == 1 ? aq[0][1] : 0.0);
        if (!FULL && r >= n) y0 = y1 = 0.0;   // (padding: zero times an infinity is not)
        if (!solve) {
          store_pair(yj + (long long)r * m + c, vecx && ok0, ok0, ok1, y0, y1);
        } else {
          if (ONE) {
            ys[ONE ? q : 0][0] = y0;
            ys[ONE ? q : 0][1] = y1;
          }
          if (INV) {
            Rs[r * ldz + 8 * q + 2 * t] = y0;
            Rs[r * ldz + 8 * q + 2 * t + 1] = y1;
          }
        }
      }
    }
    if (!solve) continue;
    if (INV) {
      grp.sync();
      for (int i = warp; i < nta; i += ONE ? 8 * NT : W) {
        double ax[CG][2], ay[CG][2];
#pragma unroll
        for (int q = 0; q < CG; ++q) ax[q][0] = ax[q][1] = ay[q][0] = ay[q][1] = 0.0;
        T fr[ONE ? 1 : NT][2];   // (all requested before the first is used)
        if (!ONE) dc = solve_diag(L, n, i);
        if (!ONE)
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) {
            T f0 = T(0), f1 = T(0);
            if (kk < nta) solve_frag<T, BWD, INV>(L, n, i, kk, vec, f0, f1, PAIR);
            fr[ONE ? 0 : kk][0] = f0;
            fr[ONE ? 0 : kk][1] = f1;
          }
#pragma unroll
        for (int kk = 0; kk < NT; ++kk) {
          if (BWD ? kk >= i && kk < nta : kk <= i) {   // (the triangle only: zero times an infinity is not zero)
            const T f0 = ONE ? fs[KEEP ? kk : 0][0] : fr[ONE ? 0 : kk][0];
            const T f1 = ONE ? fs[KEEP ? kk : 0][1] : fr[ONE ? 0 : kk][1];
            const int zo = (8 * kk + 2 * t) * ldz + g;
#pragma unroll
            for (int q = 0; q < CG; ++q)
              if (CG == 1 || q < groups) {
                mma_acc(ax[q][0], ax[q][1], (double)f0, Rs[zo + 8 * q]);
                mma_acc(ay[q][0], ay[q][1], (double)f1, Rs[zo + ldz + 8 * q]);
              }
          }
        }
#pragma unroll
        for (int q = 0; q < CG; ++q) {
          if (CG > 1 && q >= groups) break;
          const int r = 8 * i + g, c = c0 + 8 * q + 2 * t;
          const double* Rr = Rs + r * ldz + 8 * q + 2 * t;   // (this lane's own)
          const double rd = 1.0 / (double)dc;
          store_pair(yj + (long long)r * m + c, vecx && r < n && c < m, r < n && c < m, r < n && c + 1 < m,
                     fma(rd, Rr[0], ax[q][0] + ay[q][0]), fma(rd, Rr[1], ax[q][1] + ay[q][1]));
        }
      }
    } else {
      // substitution: step st solves row tile kk, later row tiles subtract it.  Four steps are
      // unrolled at a time, the next four's operands requested before them (all steps unrolled
      // did not fit the instruction cache at n = 128: 3 us a step).
      constexpr int U = KEEP ? NT : 4;
      double sum[ONE ? CG : 1][2];   // products with the rows solved so far, summed from zero
#pragma unroll
      for (int q = 0; q < (ONE ? CG : 1); ++q) sum[q][0] = sum[q][1] = 0.0;
      if (!KEEP && warp < nta) load_solve(0);
#pragma unroll 1
      for (int s0 = 0; s0 < nta; s0 += U) {
        T cur[U][2];
#pragma unroll
        for (int h = 0; h < U; ++h) {
          cur[h][0] = fs[h][0];
          cur[h][1] = fs[h][1];
        }
        if (!KEEP && s0 + U < nta && warp < nta) load_solve(s0 + U);
#pragma unroll
        for (int h = 0; h < U; ++h) {
          const int st = s0 + h, kk = BWD ? nta - 1 - st : st;
          if (st < nta) {
            if (warp == kk) {
              double* Rk = Rs + 8 * kk * ldz;
#pragma unroll
              for (int q = 0; q < CG; ++q) {
                if (CG > 1 && q >= groups) break;
                Rk[g * ldz + 8 * q + 2 * t] = ys[ONE ? q : 0][0] - sum[ONE ? q : 0][0];
                Rk[g * ldz + 8 * q + 2 * t + 1] = ys[ONE ? q : 0][1] - sum[ONE ? q : 0][1];
              }
              __syncwarp();
              if (SUBST) {
                if (lane < 8 * groups) {
                  double z[8];
#pragma unroll
                  for (int a = 0; a < 8; ++a) z[a] = Rk[a * ldz + lane];
#pragma unroll
                  for (int e = 0; e < 8; ++e) {
                    const int a = BWD ? 7 - e : e;
                    z[a] *= D[9 * a];
                    Rk[a * ldz + lane] = z[a];
#pragma unroll
                    for (int h = 0; h < 8; h += 2) {
                      const double2 c = *reinterpret_cast<const double2*>(D + 8 * a + h);
                      if (BWD ? h < a : h > a) z[h] = fma(-c.x, z[a], z[h]);
                      if (BWD ? h + 1 < a : h + 1 > a) z[h + 1] = fma(-c.y, z[a], z[h + 1]);
                    }
                  }
                }
              } else {
                double x[ONE ? CG : 1][2];
#pragma unroll
                for (int q = 0; q < CG; ++q) {
                  if (CG > 1 && q >= groups) break;
                  double(&xq)[2] = x[ONE ? q : 0];
                  xq[0] = xq[1] = 0.0;
                  mma_acc(xq[0], xq[1], i0, Rk[2 * t * ldz + 8 * q + g]);
                  mma_acc(xq[0], xq[1], i1, Rk[(2 * t + 1) * ldz + 8 * q + g]);
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < CG; ++q) {
                  if (CG > 1 && q >= groups) break;
                  Rk[g * ldz + 8 * q + 2 * t] = x[ONE ? q : 0][0];
                  Rk[g * ldz + 8 * q + 2 * t + 1] = x[ONE ? q : 0][1];
                }
              }
            }
            grp.sync();
            if ((BWD ? warp < kk : warp > kk) && warp < nta) {
#pragma unroll
              for (int q = 0; q < CG; ++q) {
                if (CG > 1 && q >= groups) break;
                const int zo = (8 * kk + 2 * t) * ldz + 8 * q + g;
                mma_acc(sum[ONE ? q : 0][0], sum[ONE ? q : 0][1], (double)cur[h][0], Rs[zo]);
                mma_acc(sum[ONE ? q : 0][0], sum[ONE ? q : 0][1], (double)cur[h][1], Rs[zo + ldz]);
              }
            }
          }
        }
      }
      if (warp < nta) {
#pragma unroll
        for (int q = 0; q < CG; ++q) {
          if (CG > 1 && q >= groups) break;
          const int r = 8 * warp + g, c = c0 + 8 * q + 2 * t;
          store_pair(yj + (long long)r * m + c, vecx && r < n && c < m, r < n && c < m, r < n && c + 1 < m,
                     Rs[r * ldz + 8 * q + 2 * t], Rs[r * ldz + 8 * q + 2 * t + 1]);
        }
      }
    }
  }
}

// vectors of one level per instance
template <int MODE>
__host__ __device__ inline int sweep_tasks(int N, const Level& lv) {
#ifdef __CUDA_ARCH__
  return MODE == kModeBackward || lv.s == 1 ? lv.d : N >> (__ffs(lv.s) - 1);
#else
  return MODE == kModeBackward || lv.s == 1 ? lv.d : N / lv.s;
#endif
}

// Blocks per SM that the registers are cut for.  Blocks of up to 24 rows hold few operands, and wide
// levels want warps: 28 an SM (21 at three tiles, where 75 registers spilt) against 16.  FP64 solve on
// factors with inverses, 33 x (N = 882, n = 10, m = 1): 211 -> 145 us, 100 x (N = 512, m = 1) at n = 12
// 324 -> 233, at n = 20 583 -> 502.  At three tiles the substitution needs more registers (24 x (N = 63,
// n = 17, m = 3): 51 us with 16 warps, 58 with 21).
__host__ __device__ constexpr int sweep_blocks(int nt, bool inv) {
  return nt <= 2 ? 28 / nt : (inv && nt == 3 ? 7 : (nt <= 8 ? 16 / nt : 1));
}

// cols: columns per block; on narrow levels several blocks (along y) share a vector's right-hand sides
template <typename T, int NT, bool FULL, int MODE, bool INV>
__global__ void __launch_bounds__(32 * NT, sweep_blocks(NT, INV))
    k_sweep_rows(Problem<T> p, Level lv, int wait, int cols) {
  const int per_b = sweep_tasks<MODE>(p.N, lv);
  const int b = blockIdx.x / per_b;
  if (!p.active(b)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  sweep_rows_body<T, NT, FULL, MODE, INV, true>(BlockGroup{}, p, lv, b, blockIdx.x - b * per_b, smem_raw, wait, blockIdx.y * cols, cols);
}

}  // namespace socu
