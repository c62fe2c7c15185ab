// Ragged batches: many independent block-tridiagonal systems of different
// horizon N, block size n and right-hand-side count m, solved by ONE
// persistent launch that pulls (instance, phase, chunk) tasks from a device
// work queue.
//
// Every instance walks a fixed sequence of phases; a phase is a set of units
// (level nodes, update targets, sweep nodes, residual row panels), cut into
// chunks of `upc` units.  The units of one phase are independent; a phase may
// start only when the previous phase of the same instance has finished:
//
//   plain factor_and_solve (T = float or double), K separator levels:
//     NODE 0, UPD 0, NODE 1, UPD 1, ..., NODE K-1, BWD K-1, ..., BWD 0
//   mixed refinement (T = float factor of an FP64 problem):
//     INIT, then the plain phases on the float copy with y = b (the first
//     round fused into the factor), XUPD (x += delta), RES (FP64 residual and
//     eta); every further round is FWD 0..K-1, BWD K-1..0, XUPD, RES, until
//     eta <= tol, max_iter rounds, or a non-finite eta.
//
// NODE/UPD/FWD/BWD/INIT/RES run the same device bodies as the per-level kernels
// of the uniform batch, or their one-warp forms (warp_rows.cuh, sweep_rows.cuh,
// refine.cuh), so each output block has one writer and the results do not
// depend on the task order.
//
// Workers.  In a large batch every warp is a worker of its own (twelve per SM):
// with thousands of units ready, units in flight count and not the time of one.
// In a small batch the levels of its largest systems, one after another, are
// the time: there a thread block of eight warps is the worker, and a unit gets a
// warp per 8-row tile (smaller blocks run side by side, rg_group_warps).  The
// host chooses (rg_use_blocks).  UPD of the plain
// path also applies the fused forward pull of the next level (the uniform
// factor_and_solve launches it separately).
//
// Queue protocol (lane 0 of a worker acts for it):
//   pop:      k = atomicAdd(head, 1); wait until slot[k] holds a task, or all
//             instances are done (then exit); a wait that sees no queue
//             progress for timeout_ns (%globaltimer) records an error and exits.
//   complete: fence; if atomicSub(rem[inst], 1) == 1 the phase is over: fence,
//             set rem for the next phase, push its chunks 1..c-1 and keep
//             chunk 0 for this worker (an instance's critical path never waits
//             in the queue).  The last phase increments `done`.
// Tasks never wait on one another, only on the queue, so the protocol cannot
// deadlock whether or not every worker is resident.
#pragma once

#include "refine.cuh"
#include "warp_rows.cuh"

namespace socu {

struct RgInst {
  long long oL, oE, oX;   // element offsets of the instance in the packed L, E and x arrays
  int N, n, m, S;
  int K;                  // separator levels
  int upc;                // units per chunk
};

enum RgMode { kRgPlain = 0, kRgRefine = 1 };
enum RgKind { kRgNode = 0, kRgUpd, kRgBwd, kRgFwd, kRgInit, kRgXupd, kRgRes };

struct RgPhase {
  int kind, level, units, upc;
};

constexpr unsigned long long kRgValid = 1ull << 63;
constexpr unsigned long long kRgExit = ~0ull;
constexpr int kRgInstBits = 24, kRgPhaseBits = 16, kRgChunkBits = 23;

__host__ __device__ inline unsigned long long rg_encode(int inst, int ph, int chunk) {
  return kRgValid | ((unsigned long long)inst << (kRgPhaseBits + kRgChunkBits)) |
         ((unsigned long long)ph << kRgChunkBits) | (unsigned long long)chunk;
}
__host__ __device__ inline void rg_decode(unsigned long long t, int& inst, int& ph, int& chunk) {
  chunk = (int)(t & ((1ull << kRgChunkBits) - 1));
  ph = (int)((t >> kRgChunkBits) & ((1ull << kRgPhaseBits) - 1));
  inst = (int)((t >> (kRgPhaseBits + kRgChunkBits)) & ((1ull << kRgInstBits) - 1));
}

// Level l of the separator schedule of a horizon-N system
// (socu/block_tridiag_solver.py:869-914).
__host__ __device__ inline Level rg_level(int N, int l) {
  // (strides are powers of two: shifts, as every worker computes this for every chunk)
  int prev = 0, curr = 0, nxt = N - 1;
  for (int k = 1; k <= l; ++k) {
    prev = curr;
    curr = nxt;
    nxt += (N >> k) - 1;
  }
  Level lv;
  lv.s = 1 << l;
  lv.d = (N + lv.s) >> (l + 1);
  lv.oc = curr;
  lv.on = nxt;
  lv.op = prev;
  return lv;
}

// Phases of the plain path; the refinement path is unbounded (decided on the device).
__host__ __device__ inline int rg_plain_phases(int K) { return 3 * K - 1; }
// Phases of the refinement path with `rounds` refinement rounds.
__host__ __device__ inline int rg_refine_phases(int K, int rounds) { return 3 * K + 2 + (rounds - 1) * (2 * K + 2); }

__host__ __device__ inline RgPhase rg_phase(const RgInst& I, int mode, int ph) {
  const int K = I.K;
  RgPhase r;
  r.upc = I.upc;
  int f = ph;
  if (mode == kRgRefine) {
    if (ph == 0) {
      r.kind = kRgInit;
      r.level = 0;
      r.units = I.N > I.S ? I.N : I.S;
      r.upc = 2 * I.upc;
      return r;
    }
    f = ph - 1;
  }
  if (f < 2 * K - 1) {
    r.level = f >> 1;
    const Level lv = rg_level(I.N, r.level);
    if ((f & 1) == 0) {
      r.kind = kRgNode;
      r.units = lv.d;
    } else {
      r.kind = kRgUpd;
      r.units = I.N >> (r.level + 1);
    }
    return r;
  }
  f -= 2 * K - 1;
  if (mode == kRgPlain || f < K) {
    r.kind = kRgBwd;
    r.level = K - 1 - f;
    r.units = rg_level(I.N, r.level).d;
    return r;
  }
  // refinement: XUPD and RES of the first round, then whole rounds
  f -= K;
  const int q = f < 2 ? 2 * K + f : (f - 2) % (2 * K + 2);
  if (q < K) {
    r.kind = kRgFwd;
    r.level = q;
    r.units = sweep_tasks<kModeForward>(I.N, rg_level(I.N, q));
  } else if (q < 2 * K) {
    r.kind = kRgBwd;
    r.level = 2 * K - 1 - q;
    r.units = rg_level(I.N, r.level).d;
  } else if (q == 2 * K) {
    r.kind = kRgXupd;
    r.level = 0;
    r.units = I.N;
    r.upc = 16;    // 16 blocks per chunk: a short elementwise pass
  } else {
    r.kind = kRgRes;
    r.level = 0;
    r.units = I.N;   // block rows
  }
  return r;
}

__host__ __device__ inline int rg_chunks(const RgPhase& P) { return (P.units + P.upc - 1) / P.upc; }

struct RgQueue {
  unsigned long long* slot;   // capacity entries; 0 = empty
  unsigned int* head;         // next slot to pop
  unsigned int* tail;         // next slot to push
  unsigned int* done;         // finished instances
  int* rem;                   // per instance: unfinished chunks of its current phase
  int* error;                 // 1: a queue wait gave up; 2: the queue overflowed
  const unsigned long long* init;   // first-phase chunks of every instance, in priority order
  unsigned int n_init;
  unsigned int capacity;
};

template <typename T>
struct RgArgs {
  const RgInst* inst;
  int count;
  T* L;   // packed diagonal blocks (factored in place; float copy when refining)
  T* E;   // packed off-diagonal storage
  T* X;   // packed right-hand sides / solutions (float correction when refining)
  // refinement only
  const double* L64;
  const double* E64;
  const double* b64;
  double* x64;
  RefineState* st;
  double* eta;
  int* iters;
  double tol;
  int max_iter;
  RgQueue q;
  long long timeout_ns;       // bound of one queue wait
  int worker_bytes;           // shared memory of one warp worker
};

__device__ __forceinline__ unsigned long long rg_clock() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned long long rg_load_slot(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned int rg_load_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Lane 0: next task for this worker, or kRgExit.
template <typename T>
__device__ unsigned long long rg_pop(const RgArgs<T>& a) {
  const unsigned int k = atomicAdd(a.q.head, 1u);
  if (k >= a.q.capacity) {
    // more pops than slots: only possible once every task has been handed out
    if (rg_load_u32(a.q.done) < (unsigned)a.count) atomicExch(a.q.error, 2);
    return kRgExit;
  }
  // the bound runs from the last sign of progress (a push or a finished
  // instance), so only a queue that stopped moving gives up
  unsigned long long t0 = rg_clock();
  unsigned int seen_tail = rg_load_u32(a.q.tail), seen_done = rg_load_u32(a.q.done);
  unsigned int ns = 32;
  while (true) {
    const unsigned long long v = rg_load_slot(a.q.slot + k);
    if (v & kRgValid) {
      __threadfence();
      return v;
    }
    const unsigned int done = rg_load_u32(a.q.done), tail = rg_load_u32(a.q.tail);
    if (done >= (unsigned)a.count) return kRgExit;
    const unsigned long long now = rg_clock();
    if (done != seen_done || tail != seen_tail) {
      seen_done = done;
      seen_tail = tail;
      t0 = now;
    } else if ((long long)(now - t0) > a.timeout_ns) {
      atomicExch(a.q.error, 1);
      return kRgExit;
    }
    __nanosleep(ns);
    if (ns < 1024) ns *= 2;
  }
}

// Per-instance view of the packed arrays.
template <typename T>
__device__ __forceinline__ Problem<T> rg_problem(const RgArgs<T>& a, const RgInst& I, int m) {
  Problem<T> p;
  p.L = a.L + I.oL;
  p.E = a.E + I.oE;
  p.X = a.X + I.oX;
  p.mask = nullptr;
  p.info = nullptr;
  p.B = 1;
  p.N = I.N;
  p.n = I.n;
  p.m = m;
  p.S = I.S;
  p.sL = p.sE = p.sX = 0;
  return p;
}

template <typename T>
__device__ __forceinline__ RefineArgs rg_refine_args(const RgArgs<T>& a, const RgInst& I, int ii) {
  RefineArgs r;
  r.L = a.L64 + I.oL;
  r.E = a.E64 + I.oE;
  r.b = a.b64 + I.oX;
  r.x = a.x64 + I.oX;
  r.mask = nullptr;
  r.L32 = reinterpret_cast<float*>(a.L) + I.oL;
  r.E32 = reinterpret_cast<float*>(a.E) + I.oE;
  r.R32 = reinterpret_cast<float*>(a.X) + I.oX;
  r.active = nullptr;
  r.st = a.st + ii;
  r.eta = nullptr;
  r.iters = nullptr;
  r.any_active = nullptr;
  r.rout = nullptr;
  r.B = 1;
  r.N = I.N;
  r.n = I.n;
  r.m = I.m;
  r.S = I.S;
  r.tol = a.tol;
  r.max_iter = a.max_iter;
  r.check_in_residual = 0;
  return r;
}

// Tile counts the bodies are built for: every one, as a body for more tiles than the block has tests
// every step, which keeps the steps from overlapping.
__host__ __device__ inline int rg_nt(int n) { return (n + 7) / 8; }
// Block workers: warps per unit, one per 8-row tile, as a power of two.
__host__ __device__ inline int rg_group_warps(int n) { return n <= 8 ? 1 : (n <= 16 ? 2 : (n <= 32 ? 4 : 8)); }
// Shared memory of one unit (bytes) for blocks of size n.
__host__ __device__ inline long long rg_unit_bytes(int n, int es, bool refine, bool blocks) {
  const int nt = rg_nt(n);
  long long v = blocks ? smem_rows_bytes(8 * nt) : smem_warp_node_bytes(nt);
  const long long w = smem_sweep_rows_bytes(8 * nt, true), u = blocks ? smem_update_rows_bytes(8 * nt, es) : 0;
  if (w > v) v = w;
  if (u > v) v = u;
  if (refine) {
    const long long i = 8 * smem_ref_init_elems(n, blocks ? rg_group_warps(n) : 1);
    if (i > v) v = i;
  }
  return (v + 127) & ~127LL;
}
// Shared memory of a thread block: four warp workers, or one block worker's units.
constexpr int kRgWorkers = 4, kRgBlockWarps = 8;
__host__ __device__ inline long long rg_block_bytes(int n, int es, bool refine, bool blocks) {
  const long long v = rg_unit_bytes(n, es, refine, blocks);
  return v * (blocks ? kRgBlockWarps / rg_group_warps(n) : kRgWorkers);
}
// Block or warp workers.  Blocks of size n alone want this many nodes per SM before single warps beat
// thread blocks (measured at 32 to 512 systems of N ~ U{8..256}, FP64, float and refined, the crossings
// of the three within a third of each other): many where a power of two of warps has no idle one (one,
// two and four tiles; eight never), few where it has (three, five and six tiles); half as many more where
// the last tile is not whole.
__host__ inline double rg_warp_nodes(int n) {
  constexpr double kNodes[] = {360, 180, 80, 110, 50, 55, 150, 1e9};
  return kNodes[rg_nt(n) - 1] * (n % 8 == 0 ? 1.0 : 1.4);
}
// `load` sums nodes / rg_warp_nodes over the batch; `sizes` counts its different bodies (tile count, whole
// or not): the warps of an SM run different ones at a time, which the instruction cache does not hold.
// Crossings in systems, measured and by this rule: {24, 40} 55, 116; {12, 36} 150 to 300, 207;
// {8, 16, 32, 48} 220 to 450, 356; {8, 16, ..., 64} 512 and more, 566.
// Times at 256 systems, warp / block workers: n = 40 3.1 / 6.2 ms FP64, 5.8 / 11.5 refined; n = 64
// 9.0 / 8.4 ms float; n ~ U{4..64} 14.7 / 5.6 ms float.
__host__ inline bool rg_use_blocks(double load, int sizes, int sms) {
  return load < sms * sqrt(sizes * sqrt((double)sizes));
}

// One unit of a level phase (one copy of each per tile count and kind of rows:
// whole tiles, rows on pair boundaries (warps only: blocks gained nothing), neither; the kernel calls them).
template <typename T, int NT, bool FULL, bool PAIR, bool BLOCKS>
__device__ __noinline__ void rg_node_unit(const Problem<T>& p, const Level& lv, int u, unsigned char* smem,
                                          WarpGroup grp) {
  if constexpr (BLOCKS)
    node_rows_body<T, NT, FULL, true, PAIR>(grp, p, lv, 0, u, smem, 0, 1, true, true);
  else
    node_warp_body<T, NT, FULL, PAIR>(p, lv, 0, u, smem);
}
template <typename T, int NT, bool FULL, bool PAIR, bool BLOCKS>
__device__ __noinline__ void rg_update_unit(const Problem<T>& p, const Level& lv, int task, unsigned char* smem,
                                            WarpGroup grp) {
  if constexpr (BLOCKS)
    update_rows_body<T, NT, FULL, false, PAIR>(grp, p, lv, 0, task, smem, 0, 1);
  else
    update_warp_body<T, NT, FULL, PAIR>(p, lv, 0, task);
}
template <typename T, int NT, bool FULL, bool PAIR, bool BLOCKS, int MODE>
__device__ __noinline__ void rg_sweep_unit(const Problem<T>& p, const Level& lv, int u, unsigned char* smem,
                                           WarpGroup grp) {
  sweep_rows_body<T, NT, FULL, MODE, true, BLOCKS, true, PAIR>(grp, p, lv, 0, u, smem, kWaitNone);
}

template <typename T, int MODE, int NT, bool FULL, bool PAIR, bool BLOCKS>
__device__ __forceinline__ void rg_level_unit(const Problem<T>& p, int kind, int level, const Level& lv, int u,
                                              unsigned char* smem, const WarpGroup& grp) {
  if (kind == kRgNode) {
    rg_node_unit<T, NT, FULL, PAIR, BLOCKS>(p, lv, u, smem, grp);
  } else if (kind == kRgUpd) {
    rg_update_unit<T, NT, FULL, PAIR, BLOCKS>(p, lv, u, smem, grp);
    if (u + 1 <= lv.d - 1) {   // fill-in block of node t = u + 1
      grp.sync();
      rg_update_unit<T, NT, FULL, PAIR, BLOCKS>(p, lv, update_targets(p.N, lv) + u, smem, grp);
    }
    // y_j -= F y_{j-s} + G^T y_{j+s} for target j = 2s(u+1) - 1
    grp.sync();
    rg_sweep_unit<T, NT, FULL, PAIR, BLOCKS, kModePull>(p, rg_level(p.N, level + 1), u, smem, grp);
  } else if (kind == kRgBwd) {
    rg_sweep_unit<T, NT, FULL, PAIR, BLOCKS, kModeBackward>(p, lv, u, smem, grp);
  } else {
    if constexpr (MODE != kRgPlain) rg_sweep_unit<T, NT, FULL, PAIR, BLOCKS, kModeForward>(p, lv, u, smem, grp);
  }
}

// Execute one chunk (all threads of the worker).
template <typename T, int MODE, bool BLOCKS>
__device__ void rg_run(const RgArgs<T>& a, int ii, int ph, int chunk, unsigned char* smem) {
  const RgInst I = a.inst[ii];
  const RgPhase P = rg_phase(I, MODE, ph);
  const int u0 = chunk * P.upc;
  const int u1 = min_i(P.units, u0 + P.upc);
  const Level lv = rg_level(I.N, P.level);
  constexpr bool kPlain = MODE == kRgPlain;
  if (P.kind == kRgXupd) {
    if constexpr (!kPlain) {
      const long long per = (long long)I.n * I.m;
      const float* d = reinterpret_cast<const float*>(a.X) + I.oX + u0 * per;
      double* x = a.x64 + I.oX + u0 * per;
      const long long len = (long long)(u1 - u0) * per;
      for (long long e = BLOCKS ? threadIdx.x : threadIdx.x & 31; e < len; e += BLOCKS ? blockDim.x : 32) x[e] += (double)d[e];
    }
    return;
  }
  // units side by side: one, or as many as the block's warps hold
  const int gw = BLOCKS ? rg_group_warps(I.n) : 1, gi = BLOCKS ? (int)(threadIdx.x >> 5) / gw : 0;
  const WarpGroup grp{BLOCKS ? gi * gw : (int)(threadIdx.x >> 5), gw, 1 + 3 * gi};
  if (BLOCKS) smem += gi * rg_unit_bytes(I.n, (int)sizeof(T), !kPlain, true);
  const Problem<T> p = rg_problem(a, I, I.m);
  for (int u = u0 + gi; u < u1; u += BLOCKS ? kRgBlockWarps / gw : 1) {
    grp.sync();
    if (!kPlain && P.kind == kRgInit) {
      if constexpr (!kPlain) ref_init_rows_body<1>(grp, rg_refine_args(a, I, ii), 0, u, smem);
      continue;
    }
    if (!kPlain && P.kind == kRgRes) {
      if constexpr (!kPlain) residual_rows_body<true>(grp, rg_refine_args(a, I, ii), 0, u);
      continue;
    }
    const int nt = rg_nt(I.n);
    const bool pair = rows_paired(p, I.n);
#define SOCU_RG_UNIT(NT)                                                                      \
  case NT:                                                                                    \
    if (pair && I.n == 8 * NT)                                                                \
      rg_level_unit<T, MODE, NT, true, false, BLOCKS>(p, P.kind, P.level, lv, u, smem, grp);  \
    else if (!BLOCKS && pair)                                                                 \
      rg_level_unit<T, MODE, NT, false, !BLOCKS, BLOCKS>(p, P.kind, P.level, lv, u, smem, grp);  \
    else                                                                                      \
      rg_level_unit<T, MODE, NT, false, false, BLOCKS>(p, P.kind, P.level, lv, u, smem, grp); \
    break;
    switch (nt) {
      SOCU_RG_UNIT(1)
      SOCU_RG_UNIT(2)
      SOCU_RG_UNIT(3)
      SOCU_RG_UNIT(4)
      SOCU_RG_UNIT(5)
      SOCU_RG_UNIT(6)
      SOCU_RG_UNIT(7)
      SOCU_RG_UNIT(8)
    }
#undef SOCU_RG_UNIT
  }
}

// Lane 0, after the worker finished a chunk of phase `ph` of instance ii:
// the continuation task (chunk 0 of the next phase) or 0.
template <typename T, int MODE>
__device__ unsigned long long rg_complete(const RgArgs<T>& a, int ii, int ph) {
  __threadfence();
  if (atomicSub(a.q.rem + ii, 1) != 1) return 0ull;
  __threadfence();
  const RgInst I = a.inst[ii];
  int nph = ph + 1;
  if (MODE == kRgRefine && rg_phase(I, MODE, ph).kind == kRgRes) {
    RefineState* s = a.st + ii;
    const double rn = __longlong_as_double((long long)atomicAdd(&s->rnorm, 0ull));
    const double xn = __longlong_as_double((long long)atomicAdd(&s->xnorm, 0ull));
    const double pn = __longlong_as_double((long long)atomicAdd(&s->psi, 0ull));
    const double bn = __longlong_as_double((long long)atomicAdd(&s->bnorm, 0ull));
    const double den = pn * xn + bn;
    const double eta = den > 0.0 ? rn / den : 0.0;
    const int it = a.iters[ii] + 1;
    a.eta[ii] = eta;
    atomicExch(&s->rnorm, 0ull);
    atomicExch(&s->xnorm, 0ull);
    if (!(eta == eta) || isinf(eta)) {
      a.iters[ii] = -it;
      nph = -1;
    } else {
      a.iters[ii] = it;
      if (eta <= a.tol || it >= a.max_iter) nph = -1;
    }
  }
  if (MODE == kRgPlain && nph >= rg_plain_phases(I.K)) nph = -1;
  RgPhase P{};
  if (nph >= 0) {
    P = rg_phase(I, MODE, nph);
    while (P.units <= 0) {   // no phase of a valid schedule is empty; stay safe regardless
      ++nph;
      if (MODE == kRgPlain && nph >= rg_plain_phases(I.K)) {
        nph = -1;
        break;
      }
      P = rg_phase(I, MODE, nph);
    }
  }
  if (nph < 0) {
    __threadfence();
    atomicAdd(a.q.done, 1u);
    return 0ull;
  }
  const int c = rg_chunks(P);
  atomicExch(a.q.rem + ii, c);
  __threadfence();
  if (c > 1) {
    const unsigned int base = atomicAdd(a.q.tail, (unsigned)(c - 1));
    for (int j = 1; j < c; ++j) {
      const unsigned int k = base + (unsigned)(j - 1);
      if (k < a.q.capacity) atomicExch(a.q.slot + k, rg_encode(ii, nph, j));
      else atomicExch(a.q.error, 2);
    }
  }
  return rg_encode(ii, nph, 0);
}

// Queue reset and first-phase chunks; per-instance refinement state.
template <typename T, int MODE>
__global__ void k_rg_start(RgArgs<T> a) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
  for (unsigned int k = gid; k < a.q.n_init; k += gs) a.q.slot[k] = a.q.init[k];
  for (int i = gid; i < a.count; i += gs) {
    const RgInst I = a.inst[i];
    a.q.rem[i] = rg_chunks(rg_phase(I, MODE, 0));
    if (MODE == kRgRefine) {
      a.st[i].psi = 0ull;
      a.st[i].bnorm = 0ull;
      a.st[i].rnorm = 0ull;
      a.st[i].xnorm = 0ull;
      a.eta[i] = __longlong_as_double(0x7ff0000000000000LL);
      a.iters[i] = 0;
    }
  }
  if (gid == 0) {
    *a.q.head = 0u;
    *a.q.tail = a.q.n_init;
    *a.q.done = 0u;
    *a.q.error = 0;
  }
}

// The persistent solver: every worker loops pop -> run -> complete.  Warp
// workers: three blocks of four per SM (168 registers, and the shared memory of
// blocks up to n = 48); block workers: two per SM.
__host__ __device__ constexpr int rg_threads(bool blocks) { return 32 * (blocks ? kRgBlockWarps : kRgWorkers); }
template <typename T, int MODE, bool BLOCKS>
__global__ void __launch_bounds__(rg_threads(BLOCKS), BLOCKS ? 2 : 3) k_ragged(const __grid_constant__ RgArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long s_task;
  unsigned char* smem = BLOCKS ? smem_raw : smem_raw + (threadIdx.x >> 5) * a.worker_bytes;
  const bool lead = BLOCKS ? threadIdx.x == 0 : (threadIdx.x & 31) == 0;
  auto share = [&](unsigned long long v) {   // the lead's value in every thread of the worker
    if (!BLOCKS) {   // (the shuffle orders no memory: what the lead's fence acquired is for every lane)
      v = __shfl_sync(kFull, v, 0);
      __syncwarp();
      return v;
    }
    if (lead) s_task = v;
    __syncthreads();
    v = s_task;
    __syncthreads();
    return v;
  };
  unsigned long long task = 0ull;
  while (true) {
    if (task == 0ull) {
      if (lead) task = rg_pop(a);
      task = share(task);
      if (task == kRgExit) return;
    }
    int ii, ph, chunk;
    rg_decode(task, ii, ph, chunk);
    rg_run<T, MODE, BLOCKS>(a, ii, ph, chunk, smem);
    if (BLOCKS)
      __syncthreads();
    else
      __syncwarp();
    if (lead) task = rg_complete<T, MODE>(a, ii, ph);
    task = share(task);
  }
}

// the kernels (ragged_*.cu: one translation unit each)
template <typename T, int MODE, bool BLOCKS>
void (*ragged_kernel())(RgArgs<T>);
template <> void (*ragged_kernel<double, kRgPlain, false>())(RgArgs<double>);
template <> void (*ragged_kernel<double, kRgPlain, true>())(RgArgs<double>);
template <> void (*ragged_kernel<float, kRgPlain, false>())(RgArgs<float>);
template <> void (*ragged_kernel<float, kRgPlain, true>())(RgArgs<float>);
template <> void (*ragged_kernel<float, kRgRefine, false>())(RgArgs<float>);
template <> void (*ragged_kernel<float, kRgRefine, true>())(RgArgs<float>);

}  // namespace socu
