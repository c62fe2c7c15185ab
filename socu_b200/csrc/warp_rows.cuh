// Level node and Schur update by a single warp (n <= 64).
//
// The bodies of node_rows.cuh and update_rows.cuh spread a node over a thread
// block to shorten its chain; where thousands of nodes are ready at once (ragged
// batches) the chain does not matter and the warps that wait on it do: a block
// of eight warps at 128 registers leaves room for two nodes per SM.  One warp per
// node needs no barrier, and twelve fit.  Same tiles, same products.
#pragma once

#include "sweep_rows.cuh"
#include "update_rows.cuh"

namespace socu {

// Shared memory of one warp (bytes): the lower tiles of C as 8x8 blocks of
// doubles (off-diagonal tile (i, j) at i (i - 1) / 2 + j, then the inverses of the
// diagonal tiles) and the diagonal tiles themselves.  A fragment is 16 bytes at 2 * lane.
__host__ __device__ constexpr int warp_node_tiles(int nt) { return nt * (nt + 1) / 2; }
__host__ __device__ inline long long smem_warp_node_bytes(int nt) { return 512LL * (warp_node_tiles(nt) + nt); }

__device__ __forceinline__ double2 tile_frag(const double* tile) {
  return *reinterpret_cast<const double2*>(tile + 2 * (threadIdx.x & 31));
}
__device__ __forceinline__ void tile_put(double* tile, double x0, double x1) {
  *reinterpret_cast<double2*>(tile + 2 * (threadIdx.x & 31)) = make_double2(x0, x1);
}

// `count` elements from p into L2
template <typename T>
__device__ __forceinline__ void warp_prefetch(const T* p, int count) {
  constexpr int line = 128 / (int)sizeof(T);
  for (int e = (threadIdx.x & 31) * line; e < count; e += 32 * line)
    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p + e));
}

// All steps of R row tiles against the finished factor: they share every operand load.
template <typename T, int NT, int R>
__device__ __forceinline__ void warp_rows_solve(double (&acc)[R][NT][2], const T (&x)[R][NT][2], int k0, int nta,
                                                const double* Ls, const double* Iv, const T* Ct) {
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[r][j][0] = acc[r][j][1] = 0.0;
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    if (k >= k0 && k < nta) {
      const DiagFrag f = diag_frag(Iv + 64 * k, Ct + 64 * k);
      double p[R][2];
#pragma unroll
      for (int r = 0; r < R; ++r)
        rows_panel(p[r][0], p[r][1], (double)x[r][k][0] - acc[r][k][0], (double)x[r][k][1] - acc[r][k][1], f);
#pragma unroll
      for (int j = k + 1; j < NT; ++j) {
        if (j < nta) {
          const double2 bv = tile_frag(Ls + 64 * (j * (j - 1) / 2 + k));
#pragma unroll
          for (int r = 0; r < R; ++r) mma_acc(acc[r][j][0], acc[r][j][1], p[r][0], bv.x);
#pragma unroll
          for (int r = 0; r < R; ++r) mma_acc(acc[r][j][0], acc[r][j][1], p[r][1], bv.y);
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        acc[r][k][0] = p[r][0];
        acc[r][k][1] = p[r][1];
      }
    }
  }
}

// One node (with its right-hand sides, keeping the inverse): as node_rows_body.
// The factor is left-looking: column k of tiles is L_i's column less the products
// of the columns before it, so only one column is in registers at a time.
template <typename T, int NT, bool FULL, bool PAIR>
__device__ __forceinline__ void node_warp_body(const Problem<T>& p, const Level& lv, int b, int t,
                                               unsigned char* smem_raw) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
  const int n = FULL ? 8 * NT : p.n, s = lv.s, i = s - 1 + 2 * s * t, nta = (n + 7) >> 3;
  const bool right = i + s < p.N, left = t >= 1;
  double* Ls = reinterpret_cast<double*>(smem_raw);
  double* Iv = Ls + 64 * (NT * (NT - 1) / 2);
  T* Ct = reinterpret_cast<T*>(Iv + 64 * NT);
  T* Li = p.Lb(b, i);
  constexpr bool vec = FULL;
  // the coupling blocks, needed after the factor: into L2 meanwhile
  T* R = right ? p.Eb(b, lv.oc + 2 * t) : nullptr;
  T* Lf = left ? p.Eb(b, lv.oc + 2 * t - 1) : nullptr;
  if (right) warp_prefetch(R, n * n);
  if (left) warp_prefetch(Lf, n * n);
  // L_i's lower tiles (diagonal ones in the inverses' places; the padding is an identity),
  // all requested before the first is used
  {
    T x[warp_node_tiles(NT)][2];
#pragma unroll
    for (int r = 0; r < NT; ++r)
#pragma unroll
      for (int j = 0; j <= r; ++j) {
        const int gr = 8 * r + g, c = 8 * j + 2 * tq, e = r * (r + 1) / 2 + j;
        x[e][0] = x[e][1] = T(0);
        if (r < nta) load_raw(Li + (gr * n + c), vec, gr < n && c < n, gr < n && c + 1 < n, x[e], PAIR);
        if (!FULL && gr >= n) {
          if (c == gr) x[e][0] = T(1);
          if (c + 1 == gr) x[e][1] = T(1);
        }
      }
#pragma unroll
    for (int r = 0; r < NT; ++r)
#pragma unroll
      for (int j = 0; j <= r; ++j)
        if (r < nta) {
          const int e = r * (r + 1) / 2 + j;
          tile_put(j == r ? Iv + 64 * r : Ls + 64 * (r * (r - 1) / 2 + j), (double)x[e][0], (double)x[e][1]);
        }
  }
  // (tiles are read as the fragments they were written as, each lane its own; only the
  // diagonal tiles, factored by the whole warp, need the warp in step)
#pragma unroll 1
  for (int k = 0; k < nta; ++k) {
    double acc[NT][2];   // products of tiles (k + r, k), summed from zero (as in node_rows_body)
#pragma unroll
    for (int r = 0; r < NT; ++r) acc[r][0] = acc[r][1] = 0.0;
#pragma unroll 1
    for (int j = 0; j < k; ++j) {
      const double2 bv = tile_frag(Ls + 64 * (k * (k - 1) / 2 + j));
#pragma unroll
      for (int r = 0; r < NT; ++r)
        if (k + r < nta) {
          const double2 av = r == 0 ? bv : tile_frag(Ls + 64 * ((k + r) * (k + r - 1) / 2 + j));
          mma_acc(acc[r][0], acc[r][1], av.x, bv.x);
          mma_acc(acc[r][0], acc[r][1], av.y, bv.y);
        }
    }
#pragma unroll
    for (int r = 0; r < NT; ++r)
      if (k + r < nta) {
        const double2 v = tile_frag(r == 0 ? Iv + 64 * k : Ls + 64 * ((k + r) * (k + r - 1) / 2 + k));
        acc[r][0] = v.x - acc[r][0];
        acc[r][1] = v.y - acc[r][1];
      }
    __syncwarp();
    rows_factor_tile<T>(acc[0][0], acc[0][1], Ct + 64 * k, Iv + 64 * k);
    __syncwarp();
    const DiagFrag f = diag_frag(Iv + 64 * k, Ct + 64 * k);
#pragma unroll
    for (int r = 1; r < NT; ++r)
      if (k + r < nta) {
        double p0, p1;
        rows_panel(p0, p1, acc[r][0], acc[r][1], f);
        tile_put(Ls + 64 * ((k + r) * (k + r - 1) / 2 + k), p0, p1);
        const int gr = 8 * (k + r) + g, c = 8 * k + 2 * tq;
        store_pair(Li + (long long)gr * n + c, vec, gr < n && c < n, gr < n && c + 1 < n, p0, p1, PAIR);
      }
    // diagonal tile: C_kk and, above the diagonal, W^T
    const int gr = 8 * k + g, c = 8 * k + 2 * tq;
    const double c0 = 2 * tq == g ? f.d0 : f.cv.x, c1 = 2 * tq + 1 == g ? f.d1 : f.cv.y;
    store_pair(Li + (long long)gr * n + c, vec, gr < n && c < n, gr < n && c + 1 < n,
               2 * tq <= g ? c0 : Iv[64 * k + 8 * (2 * tq) + g], 2 * tq + 1 <= g ? c1 : Iv[64 * k + 8 * (2 * tq + 1) + g],
               PAIR);
    __syncwarp();
  }
  // rows of the right slot, columns of the left slot and of y, two tiles at a time
  const int vr = right ? nta : 0, vl = left ? nta : 0, vy = (p.m + 7) >> 3;
  T* yi = p.Xb(b, i);
  auto source = [&](int v) {
    RowSrc<T> o;
    o.ld = n;
    o.k0 = 0;
    o.kind = 1;
    o.full = vec;
    if (v < vr) {
      o.kind = 0;
      o.base = R + (long long)8 * v * n;
      o.lim = n - 8 * v;
    } else if (v < vr + vl) {
      o.base = Lf + 8 * (v - vr);
      o.lim = n - 8 * (v - vr);
    } else {
      o.base = yi + 8 * (v - vr - vl);
      o.ld = p.m;
      o.full = false;
      o.lim = v < vr + vl + vy ? p.m - 8 * (v - vr - vl) : 0;   // (no row: a second tile that is not there)
    }
    return o;
  };
#pragma unroll 1
  for (int v = 0; v < vr + vl + vy; v += 2) {
    const RowSrc<T> s0 = source(v), s1 = source(v + 1);
    T x[2][NT][2];
    double acc[2][NT][2];
    rows_load<T, NT, PAIR>(x[0], s0, n, vec);
    rows_load<T, NT, PAIR>(x[1], s1, n, vec);
    warp_rows_solve<T, NT, 2>(acc, x, 0, nta, Ls, Iv, Ct);
    rows_store<T, NT, PAIR>(acc[0], s0, n, vec);
    rows_store<T, NT, PAIR>(acc[1], s1, n, vec);
  }
  // rows of the identity: W^T right of the diagonal tiles (the last row tile has none)
#pragma unroll 1
  for (int c = 0; c + 1 < nta; ++c) {
    RowSrc<T> o;
    o.kind = 2;
    o.full = vec;
    o.base = Li + (long long)8 * c * n;
    o.ld = n;
    o.lim = n - 8 * c;
    o.k0 = c;
    T x[1][NT][2];
    double acc[1][NT][2];
    rows_load<T, NT, PAIR>(x[0], o, n, vec);
    warp_rows_solve<T, NT, 1>(acc, x, c, nta, Ls, Iv, Ct);
    rows_store<T, NT, PAIR>(acc[0], o, n, vec);
  }
}

// One output block: as update_rows_body, operands straight from global memory,
// two row tiles of the output at a time (each operand feeds both).
template <typename T, int NT, bool FULL, bool PAIR>
__device__ __forceinline__ void update_warp_body(const Problem<T>& p, const Level& lv, int b, int task) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n = FULL ? 8 * NT : p.n, N = p.N, s = lv.s, nta = (n + 7) >> 3, U = update_targets(N, lv);
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
  constexpr bool vec = FULL;
  warp_prefetch(Out, n * n);
#pragma unroll 1
  for (int i = 0; i < nta; i += 2) {
    const int jmax = target ? min_i(i + 1, nta - 1) : nta - 1;   // last tile of the two rows
    double acc[2][NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[0][j][0] = acc[0][j][1] = acc[1][j][0] = acc[1][j][1] = 0.0;
    // steps: F's part of a target, then G's; a fill-in (F G) has one part.  (Requesting the next
    // step's operands ahead made one size faster by 5 % and a mix of sizes slower by 12 %: code.)
    const int p0 = target ? 0 : 1, parts = target && G != nullptr ? 2 : 1, steps = nta * parts;
#pragma unroll 1
    for (int it = 0; it < steps; ++it) {
      const int kk = parts == 2 ? it >> 1 : it, part = parts == 2 ? it & 1 : p0;
      const bool tr = part == 1 && target;   // the row operand: G^T
      T a[2][2], x[NT][2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (tr)
          block_frag<T, true>(G, n, i + r, kk, vec && i + r < nta, a[r][0], a[r][1], PAIR);
        else
          block_frag<T, false>(F, n, i + r, kk, vec && i + r < nta, a[r][0], a[r][1], PAIR);
      }
#pragma unroll
      for (int j = 0; j < NT; ++j)
        if (j <= jmax) {
          if (part == 1)
            block_frag<T, true>(G, n, j, kk, vec, x[j][0], x[j][1], PAIR);
          else
            block_frag<T, false>(F, n, j, kk, vec, x[j][0], x[j][1], PAIR);
        }
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int j = 0; j < NT; ++j)
          if (j <= jmax) {
            mma_acc(acc[0][j][0], acc[0][j][1], (double)a[0][e], (double)x[j][e]);
            mma_acc(acc[1][j][0], acc[1][j][1], (double)a[1][e], (double)x[j][e]);
          }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int gr = 8 * (i + r) + g;
      T o[NT][2];
#pragma unroll
      for (int j = 0; j < NT; ++j)
        if (j <= jmax) {
          const int c = 8 * j + 2 * t;
          load_raw(Out + (long long)gr * n + c, vec && i + r < nta, gr < n && c < n, gr < n && c + 1 < n, o[j], PAIR);
        }
#pragma unroll
      for (int j = 0; j < NT; ++j)
        if (j <= jmax && (!target || j <= i + r)) {
          const int c = 8 * j + 2 * t;
          const bool diag = target && j == i + r;   // only the lower triangle of a target is written
          store_pair(Out + (long long)gr * n + c, vec && i + r < nta && !diag, gr < n && c < n && (!diag || c <= gr),
                     gr < n && c + 1 < n && (!diag || c + 1 <= gr), (double)o[j][0] - acc[r][j][0],
                     (double)o[j][1] - acc[r][j][1], PAIR && !diag);
        }
    }
  }
}

}  // namespace socu
