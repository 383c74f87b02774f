// The implicit solves on row-marching passes (march.cuh), as templates on the operator: restarted GMRES, its
// mixed-precision form and the nested-Newton pressure solve, each one persistent cooperative
// kernel, for a single context or for the members of an ensemble (the _jobs kernels).
//
// GMRES(k) (implicit_operators.cpp:793-919): classical Gram-Schmidt, Givens rotations, left
// preconditioning, tolerance GMREStol * |r0| + GMREStol.  Arnoldi step j is one pass and one
// device-wide pass end: w = sigma_j A v_j - sum_i H[i][j] sigma_i v_i formed row by row (halo
// included), v_{j+1} = w stored unnormalised, A w stored, and the dot products v_i . A w,
// w . A w and w . w that give the next column of H.
//
// The symmetric one-component systems take conjugate gradients instead (below).
//
// What bounds a pass is the traffic of its vectors (j + 3 vectors and the coefficients in, two
// out) once the grid outgrows the L2, the latency of a row's chain of loads and FP64 arithmetic
// on middle grids, and on small grids the pass end.  The tile kernels (kernels_solve.cu), which
// keep the configurations these do not take, stage 32 x 16 tiles in shared memory with two or
// three block barriers per tile and were latency bound at 24-33 % of the issue slots.  Measured
// against them, us per solve: A form 1024^2 429 -> 277, 2048^2 1520 -> 909; B form 768^2 (Krylov
// spaces of 25) 2533 -> 1963, open 700 x 450 900 -> 555, 320^2 296 -> 212; nested Newton 64^2 131 -> 87,
// 700 x 450 348 -> 152, 1024^2 326 -> 151, 2048^2 1189 -> 491, Redlich-Kwong 768^2 689 -> 412; one
// pressure solve of 75 steps on 513 x 400 1609 -> 640.
#pragma once

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <vector>

#include "march.cuh"
#include "march_host.h"

namespace imex {
namespace march {
namespace {

// ------------------------------------------------------------------ one solve's work
template <class TS>
struct Work {
  TS *V, *AV;  // Krylov basis (kmax + 1 vectors) and the A v ring (2 vectors)
  TS *V0, *V0n;  // the basis's first vector, and the buffer of the next cycle's one: a pass that
                 // applies a cycle's update reads V0 on its halo while it writes the next r0
  TS* s[2];      // search-direction images of a conjugate-gradient solve
  double* partial;
  SyncState* sync;
  DevStats* st;
  int kmax, max_restarts, fam;
  int nblk, first;  // the solve's blocks: [first, first + nblk) of the launch
  int per;          // tasks per block
  long long wait_cycles;
  double tol, tol_abs;
  Geom G;
};

// Rows of Krylov vectors on their way to a lane: each lane copies its own columns of the first
// vectors of the basis asynchronously, a whole row of all of them at once and one row ahead of
// its use, so a row costs one memory latency however many vectors it combines and the loads
// hold no registers.  The row stays in the ring until the row it belongs to is completed and
// its dot products are taken, so the passes read each vector from memory once.  Slots: the
// H rows that wait for completion, the current row, the row in flight.
template <class Op, class TS>
struct Ring {
  static constexpr int M = Op::M, C = Op::C;
  static constexpr int kSlots_ = Op::H + 2, kVec = Op::R * (int)(8 / sizeof(TS));
  static constexpr int kReg = Op::R < Op::kDots ? Op::R : Op::kDots;  // dot products that a lane sums in registers
  static constexpr int kBytes = kSlots_ * Op::R * M * C * 32 * 8;  // per warp
  TS* p;  // the lane's first element
  __device__ __forceinline__ TS* at(int it, int i) const { return p + ((it % kSlots_) * kVec + i) * M * C * 32; }
};
__device__ __forceinline__ void copy_async(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits until at most n groups are in flight
template <int n>
__device__ __forceinline__ void copy_wait_but() {
  asm volatile("cp.async.wait_group %0;" ::"n"(n) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <class Op>
struct __align__(16) Smem {
  Shared S;
  unsigned char ring[Op::W][Ring<Op, double>::kBytes];
};
template <class Op, class TS>
__device__ __forceinline__ Ring<Op, TS> ring_of(Smem<Op>& sm) {
  return Ring<Op, TS>{reinterpret_cast<TS*>(sm.ring[threadIdx.x >> 5]) + (threadIdx.x & 31)};
}

enum { GM_CONVERGED = 0, GM_MAXIT = 1, GM_NONFINITE = 2, GM_SYNC = 3, GM_BREAK = 4 };

template <class W>
__device__ __forceinline__ bool lead(const W& g) {
  return threadIdx.x == 0 && (int)blockIdx.x == g.first;
}
template <class W>
__device__ __forceinline__ void record_status(const W& g, int code) {
  if (!lead(g)) return;
  const int s = code == GM_MAXIT ? IMEX_GMRES_MAXIT
                                 : (code == GM_NONFINITE ? IMEX_NONFINITE : (code == GM_SYNC ? IMEX_ERR_SYNC : IMEX_OK));
  if (s != IMEX_OK) atomicMax(&g.st->status, s);
}
// algorithmic bytes of a pass: `vals` vector values of type TS and `cvals` doubles per cell
template <class TS>
__device__ __forceinline__ void count(const Work<TS>& g, Shared& S, int vals, int cvals) {
  if (lead(g)) S.bytes += ((double)vals * sizeof(TS) + (double)cvals * 8.0) * (double)g.G.N;
}
template <class TS>
__device__ __forceinline__ Sync sync_begin(const Work<TS>& g, Shared& S) {
  if (threadIdx.x == 0) {
    S.bytes = 0.0;
    S.cycles = 0;
  }
  Sync y;
  y.s = g.sync;
  y.base = ld_relaxed(&g.sync->epoch);
  y.seq = 0;
  y.limit = g.wait_cycles;
  y.nblk = g.nblk;
  y.rank = (int)blockIdx.x - g.first;
  y.partial = g.partial;
  return y;
}
// the next launch's arrivals start where this one's end
template <class TS>
__device__ __forceinline__ void solve_end(const Work<TS>& g, const Shared& S, const Sync& y, bool ok) {
  if (lead(g)) {
    g.st->alg_bytes[g.fam] += S.bytes;
    g.st->gmres_restarts += S.cycles;
  }
  if (y.rank == 0 && threadIdx.x == 0 && ok && y.seq > 0)
    st_relaxed(&y.s->epoch, y.base + y.seq * (unsigned long long)y.nblk);
}
template <class Op>
__device__ __forceinline__ int coef_planes(const Op& op) {
  if constexpr (std::is_base_of<PressureCoef, Op>::value) return Op::kCoef + (op.jac ? 1 : 0);
  if constexpr (std::is_base_of<FaceCoef, Op>::value) return Op::kCoef + (op.vdiag ? 1 : 0);
  return Op::kCoef;
}

// tasks of this warp: consecutive tasks (vertical neighbours of a strip) go to one block's warps
template <int W, class TS, class F>
__device__ __forceinline__ void for_tasks(const Work<TS>& g, F f) {
  const int t0 = ((int)blockIdx.x - g.first) * g.per;
  const int t1 = t0 + g.per < g.G.ntask ? t0 + g.per : g.G.ntask;
  for (int t = t0 + (int)(threadIdx.x >> 5); t < t1; t += W) f(t);
}
// vector i of the basis
template <class Op, class TS>
__device__ __forceinline__ const TS* basis(const Work<TS>& g, int i) {
  return i == 0 ? g.V0 : g.V + (long long)i * Op::M * g.G.N;
}

// ------------------------------------------------------------------ passes
// the one-component operators with symmetric face weights, solved by conjugate gradients
template <class Op>
constexpr bool kSymmetric = std::is_same<Op, PressureRow<double, false>>::value || std::is_same<Op, EnergyRow<double>>::value;
// the operator of a solve's Krylov passes in arithmetic T
template <class T, class Op>
__device__ __forceinline__ auto krylov_op(const Op& op) {
  if constexpr (kSymmetric<Op>) {
    FaceRow<T> f{};
    f.kx = op.kx;
    f.ky = op.ky;
    f.idg = op.idg;
    if constexpr (std::is_base_of<PressureCoef, Op>::value) {
      f.vdiag = op.jac ? op.vdiag : nullptr;
      f.a = op.a;
    } else {
      f.vdiag = nullptr;
      f.a = op.dxdy;
    }
    return f;
  } else {
    return op.template as<T>();
  }
}
template <class Op>
constexpr bool kScalar = std::is_base_of<PressureCoef, Op>::value || std::is_base_of<EnergyCoef, Op>::value;
// what the first residual pass leaves for the Krylov passes; id = 1 / precP's diagonal
template <class Op>
__device__ __forceinline__ void store_faces(const Op& op, int o, int c, const typename Op::Emit& em, double id) {
  op.idg[o] = id;
  if (!Op::kIsRK) {
    op.kx[o] = em.kx[c];
    op.ky[o] = em.ky[c];
  }
}

// rows of a vector of planes p[m * N + offset]
template <class Op, class PT>
struct RowFill {
  __device__ __forceinline__ void ahead(const int (&)[Op::C]) const {}
  const PT* p;
  long long N;
  struct Buf {
    PT v[Op::M][Op::C];
  };
  __device__ __forceinline__ void issue(int, const int (&off)[Op::C], const int (&)[Op::C], Buf& b) const {
#pragma unroll
    for (int m = 0; m < Op::M; ++m)
#pragma unroll
      for (int c = 0; c < Op::C; ++c) b.v[m][c] = p[m * N + off[c]];
  }
  template <class T>
  __device__ __forceinline__ void finish(int, const int (&)[Op::C], const Buf& b, T (&w)[Op::M][Op::C]) const {
#pragma unroll
    for (int m = 0; m < Op::M; ++m)
#pragma unroll
      for (int c = 0; c < Op::C; ++c) w[m][c] = (T)b.v[m][c];
  }
};
// the first n vectors of the basis in a row: copied through the ring (those that fit), the rest
// read where they are added
template <class Op, class TS>
__device__ __forceinline__ void ring_copy(const Ring<Op, TS>& R, const Work<TS>& g, int it, int n, const int (&off)[Op::C]) {
  constexpr int M = Op::M, C = Op::C;
  const long long N = g.G.N;
  const int nr = n < R.kVec ? n : R.kVec;
  if (nr <= 0) return;
  TS* d = R.at(it, 0);
  const TS* p[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    p[c] = g.V0 + off[c];
#pragma unroll
    for (int m = 0; m < M; ++m) copy_async(d + (m * C + c) * 32, p[c] + m * N);
    p[c] = g.V + M * N + off[c];
  }
  // from the second vector on the planes follow one another
#pragma unroll 3
  for (int i = 1; i < nr; ++i) {
    d += M * C * 32;
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        copy_async(d + (m * C + c) * 32, p[c]);
        p[c] += N;
      }
  }
}
// the vectors past the ring in a row, K of them from i on, in registers
template <class Op, class TS>
struct Rest {
  static constexpr int K = Op::kAhead > 0 ? Op::kAhead : 2;
  TS t[K][Op::M][Op::C];
  __device__ __forceinline__ void load(const Work<TS>& g, int i, int n, const int (&off)[Op::C]) {
    const long long N = g.G.N;
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (i + q < n) {
        const TS* p = basis<Op>(g, i + q);
#pragma unroll
        for (int m = 0; m < Op::M; ++m)
#pragma unroll
          for (int c = 0; c < Op::C; ++c) t[q][m][c] = p[m * N + off[c]];
      }
  }
  __device__ __forceinline__ void add(const double* wt, int i, int n, double (&v)[Op::M][Op::C]) const {
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (i + q < n) {
        const double a = wt[i + q];
#pragma unroll
        for (int m = 0; m < Op::M; ++m)
#pragma unroll
          for (int c = 0; c < Op::C; ++c) v[m][c] = fma(a, (double)t[q][m][c], v[m][c]);
      }
  }
};
// v += sum_{i < n} wt[i] V_i in the row of iteration it
template <class Op, class TS>
__device__ __forceinline__ void ring_add(const Ring<Op, TS>& R, const Work<TS>& g, const double* wt, int it, int n,
                                         const int (&off)[Op::C], double (&v)[Op::M][Op::C]) {
  constexpr int M = Op::M, C = Op::C, kReg = Ring<Op, TS>::kReg, kVec = Ring<Op, TS>::kVec;
  constexpr bool kAhead = Op::kAhead > 0;
  Rest<Op, TS> rest;
  if (kAhead && n > kVec) rest.load(g, kVec, n, off);
  copy_wait();
  const TS* d = R.at(it, 0);
#pragma unroll
  for (int i = 0; i < kReg; ++i)
    if (i < n) {
      const double a = wt[i];
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int c = 0; c < C; ++c) v[m][c] = fma(a, (double)d[((i * M + m) * C + c) * 32], v[m][c]);
    }
  const int nr = n < kVec ? n : kVec;
#pragma unroll 4
  for (int i = kReg; i < nr; ++i) {
    const double a = wt[i];
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c = 0; c < C; ++c) v[m][c] = fma(a, (double)d[((i * M + m) * C + c) * 32], v[m][c]);
  }
  if (kAhead && n > kVec) rest.add(wt, kVec, n, v);
#pragma unroll 1
  for (int i = kVec + (kAhead ? Rest<Op, TS>::K : 0); i < n; i += Rest<Op, TS>::K) {
    rest.load(g, i, n, off);
    rest.add(wt, i, n, v);
  }
}
// rows of an iterate (plus its pending update, plus `more` when an earlier cycle wrote one),
// with the right-hand side b of the completed row (and rho, for the Redlich-Kwong slopes)
template <class Op, class TS, bool kRho = false>
struct IterateFill {
  __device__ __forceinline__ void ahead(const int (&)[Op::C]) const {}
  const Work<TS>& g;
  const Shared& S;
  Ring<Op, TS> R;
  const double *p, *more, *b, *rho;
  const double* scale;  // the update's terms are multiplied by it (conjugate gradients), or null
  int na;               // terms of the pending update
  long long N;
  static constexpr bool kScale = kSymmetric<Op> || std::is_base_of<FaceCoef, Op>::value;
  struct Buf {
    double v[Op::M][Op::C], d[Op::M][Op::C], b[Op::M][Op::C], r[kRho ? Op::C : 1], f[kScale ? Op::C : 1];
  };
  __device__ __forceinline__ void issue(int it, const int (&off)[Op::C], const int (&eo)[Op::C], Buf& u) const {
    ring_copy(R, g, it, na, off);
#pragma unroll
    for (int m = 0; m < Op::M; ++m)
#pragma unroll
      for (int c = 0; c < Op::C; ++c) {
        u.v[m][c] = p[m * N + off[c]];
        u.d[m][c] = more ? more[m * N + off[c]] : 0.0;
        u.b[m][c] = b[m * N + eo[c]];
      }
#pragma unroll
    for (int c = 0; c < Op::C; ++c) {
      if (kRho) u.r[c] = __ldg(rho + eo[c]);
      if (kScale) u.f[c] = scale && na ? scale[off[c]] : 1.0;
    }
  }
  __device__ __forceinline__ void finish(int it, const int (&off)[Op::C], const Buf& u, double (&w)[Op::M][Op::C]) const {
    double d[Op::M][Op::C];
#pragma unroll
    for (int m = 0; m < Op::M; ++m)
#pragma unroll
      for (int c = 0; c < Op::C; ++c) d[m][c] = kScale ? 0.0 : u.d[m][c];
    ring_add(R, g, S.coef, it, na, off, d);
#pragma unroll
    for (int m = 0; m < Op::M; ++m)
#pragma unroll
      for (int c = 0; c < Op::C; ++c) w[m][c] = u.v[m][c] + (kScale ? fma(u.f[c], d[m][c], u.d[m][c]) : d[m][c]);
  }
};

// rows of x with the right-hand side b of the completed row (and rho)
template <class Op, bool kRho = false>
struct RhsFill {
  __device__ __forceinline__ void ahead(const int (&)[Op::C]) const {}
  const double *p, *b, *rho;
  long long N;
  struct Buf {
    double v[Op::M][Op::C], b[Op::M][Op::C], r[kRho ? Op::C : 1];
  };
  __device__ __forceinline__ void issue(int, const int (&off)[Op::C], const int (&eo)[Op::C], Buf& u) const {
#pragma unroll
    for (int m = 0; m < Op::M; ++m)
#pragma unroll
      for (int c = 0; c < Op::C; ++c) {
        u.v[m][c] = p[m * N + off[c]];
        u.b[m][c] = b[m * N + eo[c]];
        if (kRho) u.r[c] = __ldg(rho + eo[c]);
      }
  }
  template <class T>
  __device__ __forceinline__ void finish(int, const int (&)[Op::C], const Buf& u, T (&w)[Op::M][Op::C]) const {
#pragma unroll
    for (int m = 0; m < Op::M; ++m)
#pragma unroll
      for (int c = 0; c < Op::C; ++c) w[m][c] = (T)u.v[m][c];
  }
};

// A v_0 = M^-1 A V0 (unnormalised); S.red[0] = V0 . A V0
template <class Op, class TS>
__device__ __forceinline__ bool pass_av0(const Op& op, const Work<TS>& g, Shared& S, Sync& y) {
  using T = typename Op::T;
  const long long N = g.G.N;
  acc_clear(S);
  double va = 0.0;
  RowFill<Op, TS> fill{g.V0, N};
  auto emit = [&](int, const int (&eo)[Op::C], const bool (&own)[Op::C], const T (&wc)[Op::M][Op::C],
                  T (&out)[Op::M][Op::C], const typename Op::Emit& em, const typename RowFill<Op, TS>::Buf&) {
    op.precond(em, out);
#pragma unroll
    for (int m = 0; m < Op::M; ++m)
#pragma unroll
      for (int c = 0; c < Op::C; ++c)
        if (own[c]) {
          g.AV[m * N + eo[c]] = (TS)out[m][c];
          va += (double)wc[m][c] * (double)out[m][c];
        }
  };
  for_tasks<Op::W>(g, [&](int task) { run_task<Op>(op, g.G, task, fill, emit); });
  va = warp_sum(va);
  if ((threadIdx.x & 31) == 0) S.acc[threadIdx.x >> 5][0] = va;
  count(g, S, 2 * Op::M, coef_planes(op));
  return pass_end<Op::W>(y, S, 1);
}

// adds the lane sums x[0, nI) of vectors i.. to the warp's dot products
__device__ __forceinline__ void add_dots(Shared& S, double (&x)[4], int i, int nI) {
  const int lane = threadIdx.x & 31;
  const double s = warp_sum4(x);
  if ((lane & 7) == 0 && (lane >> 3) < nI) S.acc[threadIdx.x >> 5][i + (lane >> 3)] += s;
}

// w = sigma_j A v_j - sum_i H[i][j] sigma_i v_i
template <class Op, class TS>
struct ArnoldiFill {
  static constexpr int M = Op::M, C = Op::C;
  const Work<TS>& g;
  const Shared& S;
  Ring<Op, TS> R;
  Rest<Op, TS>& dr;
  const TS* AVj;
  int n;  // basis vectors: j + 1
  __device__ __forceinline__ void ahead(const int (&eo)[C]) const {
    if (Op::kAhead > 0 && n > Ring<Op, TS>::kVec) dr.load(g, Ring<Op, TS>::kVec, n, eo);
  }
  struct Buf {
    TS h[M][C];
  };
  __device__ __forceinline__ void issue(int it, const int (&off)[C], const int (&)[C], Buf& b) const {
    const long long N = g.G.N;
    ring_copy(R, g, it, n, off);
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c = 0; c < C; ++c) b.h[m][c] = AVj[m * N + off[c]];
  }
  template <class T>
  __device__ __forceinline__ void finish(int it, const int (&off)[C], const Buf& b, T (&w)[M][C]) const {
    double v[M][C];
    const double s = S.comb[0];
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c = 0; c < C; ++c) v[m][c] = s * (double)b.h[m][c];
    ring_add(R, g, S.comb + 1, it, n, off, v);
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c = 0; c < C; ++c) w[m][c] = (T)v[m][c];
  }
};
// Arnoldi step j (see the top): S.red[i] = v_i . A w (i <= j), [j+1] = w . A w, [j+2] = w . w
template <class Op, class TS>
__device__ __forceinline__ bool pass_arnoldi(const Op& op, const Work<TS>& g, Smem<Op>& sm, Sync& y, int j) {
  using T = typename Op::T;
  constexpr int C = Op::C, M = Op::M;
  Shared& S = sm.S;
  const long long N = g.G.N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  TS* Vn = g.V + (long long)(j + 1) * M * N;
  TS* AVn = g.AV + (long long)((j + 1) & 1) * M * N;
  acc_clear(S);
  double wa = 0.0, ww = 0.0;
  const Ring<Op, TS> R = ring_of<Op, TS>(sm);
  constexpr int kReg = Ring<Op, TS>::kReg;
  double dv[kReg];
#pragma unroll
  for (int i = 0; i < kReg; ++i) dv[i] = 0.0;
  Rest<Op, TS> dr;  // the completed row's vectors past the ring, loaded ahead of the operator
  ArnoldiFill<Op, TS> fill{g, S, R, dr, g.AV + (long long)(j & 1) * M * N, j + 1};
  auto emit = [&](int it, const int (&eo)[C], const bool (&own)[C], const T (&wc)[M][C], T (&out)[M][C],
                  const typename Op::Emit& em, const typename ArnoldiFill<Op, TS>::Buf&) {
    op.precond(em, out);
    double a[M][C];
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        a[m][c] = own[c] ? (double)out[m][c] : 0.0;
        if (own[c]) {
          Vn[m * N + eo[c]] = (TS)wc[m][c];
          AVn[m * N + eo[c]] = (TS)out[m][c];
          wa = fma((double)wc[m][c], a[m][c], wa);
          ww = fma((double)wc[m][c], (double)wc[m][c], ww);
        }
      }
    const int n = j + 1, nr = n < R.kVec ? n : R.kVec;
    const TS* d = R.at(it - Op::H, 0);
#pragma unroll
    for (int i = 0; i < kReg; ++i)
      if (i < n) {
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
          for (int c = 0; c < C; ++c) dv[i] = fma((double)d[((i * M + m) * C + c) * 32], a[m][c], dv[i]);
      }
#pragma unroll 1
    for (int i = kReg; i < nr; i += 4) {
      double x[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (i + q < nr)
#pragma unroll
          for (int m = 0; m < M; ++m)
#pragma unroll
            for (int c = 0; c < C; ++c) x[q] = fma((double)d[(((i + q) * M + m) * C + c) * 32], a[m][c], x[q]);
      add_dots(S, x, i, nr - i);
    }
#pragma unroll 1
    for (int i = nr; i < n; i += Rest<Op, TS>::K) {
      if (i > nr || Op::kAhead == 0) dr.load(g, i, n, eo);
#pragma unroll
      for (int q0 = 0; q0 < Rest<Op, TS>::K; q0 += 4)
        if (i + q0 < n) {
          double x[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (q0 + q < Rest<Op, TS>::K && i + q0 + q < n)
#pragma unroll
              for (int m = 0; m < M; ++m)
#pragma unroll
                for (int c = 0; c < C; ++c) x[q] = fma((double)dr.t[q0 + q < Rest<Op, TS>::K ? q0 + q : 0][m][c], a[m][c], x[q]);
          add_dots(S, x, i + q0, Rest<Op, TS>::K - q0 < n - i - q0 ? Rest<Op, TS>::K - q0 : n - i - q0);
        }
    }
  };
  for_tasks<Op::W>(g, [&](int task) { run_task<Op>(op, g.G, task, fill, emit); });
  double t[4] = {wa, ww, 0.0, 0.0};
  const double s = warp_sum4(t);
#pragma unroll
  for (int i = 0; i < kReg; i += 4)
    if (i <= j) {
      double q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = i + u < kReg ? dv[i + u < kReg ? i + u : 0] : 0.0;
      const double r = warp_sum4(q);
      if ((lane & 7) == 0 && i + (lane >> 3) < kReg) S.acc[warp][i + (lane >> 3)] = r;
    }
  __syncwarp();
  if (lane == 0) S.acc[warp][j + 1] = s;
  if (lane == 8) S.acc[warp][j + 2] = s;
  count(g, S, (j + 4) * M, coef_planes(op));
  return pass_end<Op::W>(y, S, j + 3);
}

// r0 = M^-1 (b - A x) -> V0 (raw: b - A x); S.red[0] = |M^-1 (b - A x)|^2.  kFirst (one-component
// systems): also the planes that the solve's Krylov passes read.
template <bool kFirst, class Op, class TS>
__device__ __forceinline__ bool pass_residual(const Op& op, const Work<TS>& g, Shared& S, Sync& y, const double* x,
                                              const double* b, bool raw = false) {
  using T = typename Op::T;
  constexpr int C = Op::C, M = Op::M;
  const long long N = g.G.N;
  acc_clear(S);
  double rr = 0.0;
  RhsFill<Op> fill{x, b, nullptr, N};
  auto emit = [&](int, const int (&eo)[C], const bool (&own)[C], const T (&)[M][C], T (&out)[M][C],
                  const typename Op::Emit& em, const typename RhsFill<Op>::Buf& u) {
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c = 0; c < C; ++c) out[m][c] = (T)(u.b[m][c] - (double)out[m][c]);
    if constexpr (kFirst && kScalar<Op>) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const double id = 1.0 / (em.vd[c] + em.dg[c]), r = id * (double)out[0][c];
        if (own[c]) {
          store_faces(op, eo[c], c, em, id);
          g.V0[eo[c]] = (TS)(raw ? (double)out[0][c] : r);
          rr = fma(r, r, rr);
        }
      }
    } else {
      op.precond(em, out);
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (own[c]) {
            g.V0[m * N + eo[c]] = (TS)out[m][c];
            rr += (double)out[m][c] * (double)out[m][c];
          }
    }
  };
  for_tasks<Op::W>(g, [&](int task) { run_task<Op>(op, g.G, task, fill, emit); });
  rr = warp_sum(rr);
  if ((threadIdx.x & 31) == 0) S.acc[threadIdx.x >> 5][0] = rr;
  count(g, S, Op::M, 2 * Op::M + coef_planes(op));
  return pass_end<Op::W>(y, S, 1);
}

// ------------------------------------------------------------------ one GMRES cycle
// From V0 = r0 (left-preconditioned residual, norm S.gam[0] > tol): up to kmax Arnoldi steps,
// the Givens update of each column and the back substitution.  Leaves the weights of the
// update sum_i coef_i V_i in S.coef[0, S.nalpha).
template <class Op, class TS>
__device__ __forceinline__ int gmres_cycle(const Op& op, const Work<TS>& g, Smem<Op>& sm, Sync& y, double tol_eff, int& iters) {
  Shared& S = sm.S;
  const int tid = threadIdx.x;
  if (tid == 0) {
    S.sigma[0] = 1.0 / S.gam[0];
    S.nalpha = 0;
  }
  if (lead(g)) S.cycles += 1;
  if (!pass_av0(op, g, S, y)) return GM_SYNC;
  if (tid == 0) {
    const double s0 = S.sigma[0];
    S.hcol[0] = s0 * s0 * S.red[0];
    S.comb[0] = s0;
    S.comb[1] = -S.hcol[0] * s0;
  }
  __syncthreads();
  int jend = -1;
  bool converged = false;
  for (int j = 0; j < g.kmax; ++j) {
    if (!pass_arnoldi(op, g, sm, y, j)) return GM_SYNC;
    ++iters;
    if (tid == 0) {
      // H[j+1][j] = |w|, the rotations of column j (implicit_operators.cpp:857-873)
      const double beta_w = sqrt(S.red[j + 2]);
      double t = S.hcol[0];
      for (int i = 0; i < j; ++i) {
        const double n = S.hcol[i + 1], c = S.cs[i + 1], s = S.sn[i + 1];
        S.H[i][j] = c * t + s * n;
        t = s * t - c * n;
      }
      const double beta = sqrt(t * t + beta_w * beta_w);
      const double s1 = beta_w / beta, c1 = t / beta;
      S.sn[j + 1] = s1;
      S.cs[j + 1] = c1;
      S.H[j][j] = beta;
      const double gj = S.gam[j];
      S.gam[j + 1] = s1 * gj;
      S.gam[j] = c1 * gj;
    } else if (tid >= 32 && tid < 64) {
      // column j + 1 from the pass's dot products: v_i . A v_{j+1}
      const int i = tid - 32;
      const double sw = 1.0 / sqrt(S.red[j + 2]);
      __syncwarp();
      if (i <= j) {
        const double si = S.sigma[i], h = si * S.red[i] * sw;
        S.comb[i + 1] = -h * si;
      }
      if (i == j + 1) {
        S.sigma[i] = sw;
        S.comb[0] = sw;
        S.comb[i + 1] = -(sw * sw * S.red[i]) * sw;
      }
    }
    __syncthreads();
    if (tid <= j) S.hcol[tid] = S.sigma[tid] * S.red[tid] * S.sigma[j + 1];
    if (tid == j + 1) S.hcol[tid] = S.sigma[tid] * S.sigma[tid] * S.red[tid];
    const double gn = S.gam[j + 1];
    jend = j;
    if (!isfinite(gn)) return GM_NONFINITE;
    if (!(gn > tol_eff)) {
      converged = true;
      break;
    }
    __syncthreads();
  }
  __syncthreads();
  if (tid < 32) {  // back substitution (implicit_operators.cpp:882-891), one row per lane
    double yv = tid <= jend ? S.gam[tid] : 0.0;
    const double d = tid <= jend ? S.H[tid][tid] : 1.0;
    for (int k = jend; k >= 0; --k) {
      const double ak = __shfl_sync(0xffffffffu, yv / d, k);
      if (tid < k) yv -= S.H[tid][k] * ak;
      if (tid == k) yv = ak;
    }
    if (tid <= jend) {
      S.coef[tid] = yv * S.sigma[tid];
    }
    if (tid == 0) {
      S.nalpha = jend + 1;
      if ((int)blockIdx.x == g.first) g.st->last_residual = S.gam[jend + 1];
    }
  }
  __syncthreads();
  return converged ? GM_CONVERGED : GM_MAXIT;
}

// x (+)= sum_i coef_i V_i over all values (zero: x is not read)
template <int M, int W, class TS>
__device__ __forceinline__ void apply_update(const Work<TS>& g, Shared& S, double* x, bool zero,
                                             const double* scale = nullptr) {
  const long long N = g.G.N, n = (long long)M * N, stride = (long long)g.nblk * 32 * W;
  const int na = S.nalpha;
  constexpr int U = 4;
  for (long long c0 = ((long long)blockIdx.x - g.first) * 32 * W + threadIdx.x; c0 < n; c0 += U * stride) {
    double v[U], x0[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = c0 + u * stride < n;
      x0[u] = zero || !in ? 0.0 : x[c0 + u * stride];
      v[u] = 0.0;
    }
#pragma unroll 2
    for (int i = 0; i < na; ++i) {
      const TS* p = i == 0 ? g.V0 : g.V + i * n;
      const double a = S.coef[i];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c0 + u * stride < n) v[u] = fma(a, ldv(p + c0 + u * stride), v[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c0 + u * stride < n) x[c0 + u * stride] = fma(scale ? scale[c0 + u * stride] : 1.0, v[u], x0[u]);
  }
  count(g, S, na * M, (zero ? 1 : 2) * M);
}

// A task's rows for passes of one halo row whose planes are copied into per-lane slots of shared
// memory kStage - 1 rows ahead of the one in work (each lane copies and reads its own columns).
// copy(it, c, n): asynchronous copies of cell n, column c, into the slot of iteration it.  The
// caller loops over it < count(): wait(it, on) (row it, the cells on[], is in its slot), reads
// the slot, next(it, copy), then works.
template <int C, int kStage>
struct StagedRows {
  const Geom& G;
  int xo[C], ya, rows;
  bool own[C];
  __device__ __forceinline__ StagedRows(const Geom& g, int task) : G(g) {
    const int strip = task / G.nseg, seg = task - strip * G.nseg, lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int q = lane + 32 * c, x = strip * G.wd + q - 1;
      own[c] = q >= 1 && q < 1 + G.wd && x < G.nx;
      xo[c] = map_x(G, x);
    }
    ya = seg * G.L;
    rows = (ya + G.L < G.ny ? ya + G.L : G.ny) - ya;
  }
  __device__ __forceinline__ int count() const { return rows + 2; }
  template <class Copy>
  __device__ __forceinline__ void issue(int it, Copy& copy) const {
    if (it < rows + 2) {
      const int o = map_y(G, ya - 1 + it) * G.nx;
#pragma unroll
      for (int c = 0; c < C; ++c) copy(it, c, o + xo[c]);
    }
    copy_commit();
  }
  template <class Copy>
  __device__ __forceinline__ void start(Copy& copy) const {
    __syncwarp();  // the slots of the task before are read
#pragma unroll
    for (int it = 0; it < kStage - 1; ++it) issue(it, copy);
  }
  __device__ __forceinline__ void wait(int it, int (&on)[C]) const {
    const int o = map_y(G, ya - 1 + it) * G.nx;
#pragma unroll
    for (int c = 0; c < C; ++c) on[c] = o + xo[c];
    copy_wait_but<kStage - 2>();
  }
  template <class Copy>
  __device__ __forceinline__ void next(int it, Copy& copy) const {
    __syncwarp();  // every lane has read the row before, whose slot the next copies take
    issue(it + kStage - 1, copy);
  }
};

// ------------------------------------------------------------------ conjugate gradients
// The symmetric one-component systems (FaceRow) take preconditioned conjugate gradients in the
// form with one reduction per step (Chronopoulos and Gear, s-step iterative methods for
// symmetric linear systems, 1989):
//   s = w + beta s, r <- r - alpha s, u = M^-1 r, w = A u;  gamma = r.u, delta = w.u, |u|
//   beta = gamma / gamma_old, alpha = gamma / (delta - beta gamma / alpha_old)
// stopped by the same test as GMRES, |M^-1 r| <= tol.  GMRES minimises that norm over the same
// Krylov space, but its step j combines and multiplies j vectors; a step here moves nine planes
// whatever its number.  The residuals are kept as the basis (slot k holds r_k), so the search
// directions p_k = u_k + beta_k p_{k-1} are never stored: the solution sum_k alpha_k p_k is
// M^-1 sum_k c_k r_k with c_k = alpha_k + beta_{k+1} c_{k+1}, formed when the solve ends (or the
// slots are full).  A non-positive curvature hands the solve to GMRES.
template <bool kFirst, class Op, class TS>
__device__ __forceinline__ bool pass_cg(const Op& op, const Work<TS>& g, Smem<Op>& sm, Sync& y, int k, int par,
                                        double alpha, double beta) {
  using T = typename Op::T;
  constexpr int C = Op::C;
  Shared& S = sm.S;
  // rows on their way to the lane (its own columns): kStage - 1 ahead of the one in work
  constexpr int kStage = 4, kRow = 6 * C * 32;
  static_assert(kStage * kRow * 8 <= Ring<Op, double>::kBytes, "the stages live in the ring");
  double* const stage = reinterpret_cast<double*>(sm.ring[threadIdx.x >> 5]);
  auto stage_at = [&](int it) -> double* { return stage + (it & (kStage - 1)) * kRow; };
  const Geom& G = g.G;
  const int lane = threadIdx.x & 31;
  const TS* r0 = basis<Op>(g, k);
  TS* r1 = g.V + (long long)(k + 1) * G.N;
  const TS *w0 = g.AV + (long long)(par ^ 1) * G.N, *s0 = g.s[par ^ 1];
  TS *w1 = g.AV + (long long)par * G.N, *s1 = g.s[par];
  const bool hist = !kFirst && beta != 0.0;
  acc_clear(S);
  double ru = 0.0, wu = 0.0, uu = 0.0;
  for_tasks<Op::W>(g, [&](int task) {
    const int strip = task / G.nseg, seg = task - strip * G.nseg;
    int xo[C];
    bool own[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int q = lane + 32 * c, x = strip * G.wd + q - 1;
      own[c] = q >= 1 && q < 1 + G.wd && x < G.nx;
      xo[c] = map_x(G, x);
    }
    const int ya = seg * G.L, yb = ya + G.L < G.ny ? ya + G.L : G.ny, rows = yb - ya;
    // row `it` into its slot: kx, ky, id as doubles, then r, w, s
    auto issue = [&](int it) {
      if (it < rows + 2) {
        const int o = map_y(G, ya - 1 + it) * G.nx;
        double* d = stage_at(it) + lane;
        TS* t = reinterpret_cast<TS*>(stage_at(it) + 3 * C * 32) + lane;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int n = o + xo[c];
          copy_async(d + c * 32, op.kx + n);
          copy_async(d + (C + c) * 32, op.ky + n);
          copy_async(d + (2 * C + c) * 32, op.idg + n);
          copy_async(t + c * 32, r0 + n);
          if (!kFirst) copy_async(t + (C + c) * 32, w0 + n);
          if (hist) copy_async(t + (2 * C + c) * 32, s0 + n);
        }
      }
      copy_commit();
    };
    typename Op::State st{};
    T vd[C];
    int op_[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      vd[c] = T(0);
      op_[c] = 0;
    }
    __syncwarp();  // the slots of the task before are read
#pragma unroll
    for (int it = 0; it < kStage - 1; ++it) issue(it);
#pragma unroll 1
    for (int it = 0; it < rows + 2; ++it) {
      struct {
        TS r[C], w[C], s[C];
        double id[C];
        typename Op::Row k;
        T vd[C];
      } n;
      const int o = map_y(G, ya - 1 + it) * G.nx;
      int on[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        on[c] = o + xo[c];
        n.vd[c] = op.slope(on[c]);
      }
      copy_wait_but<kStage - 2>();
      {
        const double* d = stage_at(it) + lane;
        const TS* t = reinterpret_cast<const TS*>(stage_at(it) + 3 * C * 32) + lane;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          n.k.kx[c] = (T)d[c * 32];
          n.k.ky[c] = (T)d[(C + c) * 32];
          n.id[c] = d[(2 * C + c) * 32];
          n.r[c] = t[c * 32];
          if (!kFirst) n.w[c] = t[(C + c) * 32];
          if (hist) n.s[c] = t[(2 * C + c) * 32];
        }
      }
      __syncwarp();  // every lane has read the row before, whose slot the next copies take
      issue(it + kStage - 1);
      T u[C], out[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        double r = (double)n.r[c];
        if (!kFirst) {
          const double s = hist ? fma(beta, (double)n.s[c], (double)n.w[c]) : (double)n.w[c];
          r = fma(-alpha, s, r);
          if (it >= 1 && it <= rows && own[c]) {
            r1[on[c]] = (TS)r;
            s1[on[c]] = (TS)s;
          }
        }
        const double ud = n.id[c] * r;
        u[c] = (T)ud;
        if (it >= 1 && it <= rows && own[c]) {
          ru = fma(r, ud, ru);
          uu = fma(ud, ud, uu);
        }
      }
      T uc[C];
#pragma unroll
      for (int c = 0; c < C; ++c) uc[c] = st.x[c];
      op.complete(st, u, n.k, vd, out);
      if (it >= 2) {
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (own[c]) {
            w1[op_[c]] = (TS)out[c];
            wu = fma((double)out[c], (double)uc[c], wu);
          }
      }
#pragma unroll
      for (int c = 0; c < C; ++c) {
        vd[c] = n.vd[c];
        op_[c] = on[c];
      }
    }
  });
  double t[4] = {ru, wu, uu, 0.0};
  const double q = warp_sum4(t);
  if ((lane & 7) == 0 && lane < 24) S.acc[threadIdx.x >> 5][lane >> 3] = q;
  count(g, S, kFirst ? 2 : (hist ? 6 : 5), Op::kCoef + (op.vdiag || op.p ? 1 : 0));
  return pass_end<Op::W>(y, S, 3);
}
// weights of the update: S.coef[i] = c_i of slots 0..k, S.nalpha = k + 1; scale by M^-1 (op.idg)
__device__ __forceinline__ void cg_weights(Shared& S, int k) {
  if (threadIdx.x == 0) {
    double c = S.cga[k];
    S.coef[k] = c;
    for (int i = k - 1; i >= 0; --i) {
      c = fma(S.cgb[i + 1], c, S.cga[i]);
      S.coef[i] = c;
    }
    S.nalpha = k + 1;
  }
  __syncthreads();
}
// From r0 in V0 (not preconditioned).  On return the update M^-1 sum_i coef_i V_i of the last
// slots waits in S; full slots were added to x before (x_live: x already holds a part).
template <class Op, class TS>
__device__ __forceinline__ int cg_solve(const Op& op, const Work<TS>& g, Smem<Op>& sm, Sync& y, double tol_eff, double* x,
                                        bool& x_live, int& iters) {
  Shared& S = sm.S;
  const int tid = threadIdx.x;
  int par = 0, k = 0, cycles = 0;
  __syncthreads();
  if (tid == 0) S.nalpha = 0;
  if (lead(g)) S.cycles += 1;
  if (!pass_cg<true>(op, g, sm, y, 0, par, 0.0, 0.0)) return GM_SYNC;
  double gamma = S.red[0], alpha = gamma / S.red[1], beta = 0.0;
  if (!(gamma > 0.0) || !(alpha > 0.0) || !isfinite(alpha)) return GM_BREAK;
  for (;;) {
    if (tid == 0) {
      S.cga[k] = alpha;
      S.cgb[k] = beta;
    }
    par ^= 1;
    if (!pass_cg<false>(op, g, sm, y, k, par, alpha, beta)) return GM_SYNC;
    ++iters;
    const double gn = S.red[0], delta = S.red[1], res = sqrt(S.red[2]);
    __syncthreads();
    if (lead(g)) g.st->last_residual = res;
    if (!isfinite(res)) return GM_NONFINITE;
    if (!(res > tol_eff)) {
      cg_weights(S, k);
      return GM_CONVERGED;
    }
    const double bn = gn / gamma, den = delta - bn * gn / alpha;
    const bool broke = !(gn > 0.0) || !(den > 0.0) || !isfinite(gn / den);
    const bool full = k + 1 == g.kmax;
    if (broke || (full && ++cycles >= g.max_restarts)) {
      cg_weights(S, k);
      return broke ? GM_BREAK : GM_MAXIT;
    }
    beta = bn;
    alpha = gn / den;
    gamma = gn;
    if (!full) {
      ++k;
      continue;
    }
    // the slots are full: add their part to x, leave p_k / M^-1 in slot 0 and r_{k+1} in slot 1
    cg_weights(S, k);
    if (tid == 0) {  // p_k = M^-1 sum_i e_i r_i
      double e = 1.0;
      S.comb[k] = e;
      for (int i = k - 1; i >= 0; --i) {
        e *= S.cgb[i + 1];
        S.comb[i] = e;
      }
      S.cga[0] = 0.0;
      S.cgb[0] = 0.0;
    }
    if (lead(g)) S.cycles += 1;
    __syncthreads();
    const long long N = g.G.N;
    for (long long c = ((long long)blockIdx.x - g.first) * 32 * Op::W + tid; c < N; c += (long long)g.nblk * 32 * Op::W) {
      double v = 0.0, p = 0.0;
#pragma unroll 4
      for (int i = 0; i <= k; ++i) {
        const double r = ldv(basis<Op>(g, i) + c);
        v = fma(S.coef[i], r, v);
        p = fma(S.comb[i], r, p);
      }
      const TS rn = g.V[(long long)(k + 1) * N + c];
      x[c] = fma(op.idg[c], v, x_live ? x[c] : 0.0);
      g.V0[c] = (TS)p;
      g.V[N + c] = rn;
    }
    count(g, S, k + 4, x_live ? 3 : 2);
    x_live = true;
    if (tid == 0) S.nalpha = 0;
    if (!pass_end<Op::W>(y, S, 1)) return GM_SYNC;
    k = 1;
  }
}

// the job of a block of a batched launch, copied to shared memory once
template <class Job>
struct __align__(16) JobCopy {
  unsigned char b[sizeof(Job)];
};
template <class Job>
__device__ __forceinline__ const Job& copy_job(JobCopy<Job>& s, const Job* j) {
  static_assert(sizeof(Job) % 8 == 0, "copied by words");
  for (unsigned q = threadIdx.x; q < sizeof(Job) / 8; q += blockDim.x)
    reinterpret_cast<unsigned long long*>(s.b)[q] = reinterpret_cast<const unsigned long long*>(j)[q];
  __syncthreads();
  return *reinterpret_cast<const Job*>(s.b);
}

// ------------------------------------------------------------------ GMRES
template <class Op>
struct GmresJob {
  Op op;
  Work<double> g;
  double* x;
  const double* b;
};
template <class Op>
__device__ __forceinline__ int gmres(const Op& op, const Work<double>& g, double* x, const double* b, Smem<Op>& smo, Sync& y) {
  const auto kop = krylov_op<double>(op);
  using KOp = typename std::remove_const<decltype(kop)>::type;
  Smem<KOp>& sm = reinterpret_cast<Smem<KOp>&>(smo);
  Shared& S = sm.S;
  constexpr bool kSym = kSymmetric<Op>;
  double tol_eff = 0.0;
  int iters = 0, code = GM_MAXIT;
  const bool cg = kSym && g.kmax > 1;
  int free = 0;  // cycles that do not count
  for (int outer = 0; outer - free < g.max_restarts; ++outer) {
    bool ok = false;
    if constexpr (!kScalar<Op>) {
      ok = pass_residual<false>(op, g, S, y, x, b);
    } else {
      ok = outer == 0 ? pass_residual<true>(op, g, S, y, x, b, cg) : pass_residual<false>(kop, g, S, y, x, b);
    }
    if (!ok) return GM_SYNC;
    const double r = sqrt(S.red[0]);
    if (outer == 0) tol_eff = g.tol * r + g.tol_abs;
    if (!isfinite(r)) {
      code = GM_NONFINITE;
      break;
    }
    if (r <= tol_eff) {
      if (lead(g)) g.st->last_residual = r;
      code = GM_CONVERGED;
      break;
    }
    bool scaled = false;
    if constexpr (kSym) {
      if (cg && outer == 0) {
        bool live = true;
        code = cg_solve(kop, g, sm, y, tol_eff, x, live, iters);
        scaled = true;
        // where they break down, or need more steps than GMRES may (it minimises the norm that is tested,
        // and can end a few steps before them), GMRES goes on from here with all its restarts
        if (code == GM_BREAK || code == GM_MAXIT) free = 1;
      }
    }
    if (!scaled) {
      if (threadIdx.x == 0) S.gam[0] = r;
      __syncthreads();
      code = gmres_cycle(kop, g, sm, y, tol_eff, iters);
    }
    if (code == GM_SYNC || code == GM_NONFINITE) break;
    if constexpr (kSym) apply_update<Op::M, Op::W>(g, S, x, false, scaled ? op.idg : nullptr);
    else apply_update<Op::M, Op::W>(g, S, x, false);
    if (code == GM_CONVERGED) break;
    if (outer + 1 - free < g.max_restarts && !pass_end<Op::W>(y, S, 1)) return GM_SYNC;  // x is complete before it is read
    code = GM_MAXIT;
  }
  if (lead(g)) g.st->gmres_iters += iters;
  return code;
}
template <class Op>
__device__ __forceinline__ void gmres_body(const GmresJob<Op>& j) {
  extern __shared__ __align__(16) unsigned char dsm[];
  Smem<Op>& sm = *reinterpret_cast<Smem<Op>*>(dsm);
  Op op = j.op;
  op.bind();
  Sync y = sync_begin(j.g, sm.S);
  if (lead(j.g)) j.g.st->gmres_solves += 1;
  const int code = gmres(op, j.g, j.x, j.b, sm, y);
  record_status(j.g, code);
  solve_end(j.g, sm.S, y, code != GM_SYNC);
}
template <class Op>
__global__ void __launch_bounds__(32 * Op::W, 1) k_gmres(const __grid_constant__ GmresJob<Op> j) {
  gmres_body(j);
}
template <class Op>
__global__ void __launch_bounds__(32 * Op::W, 1) k_gmres_jobs(const GmresJob<Op>* jobs, const int* map) {
  __shared__ JobCopy<GmresJob<Op>> s;
  gmres_body(copy_job(s, jobs + map[blockIdx.x]));
}

// ------------------------------------------------------------------ mixed-precision GMRES
// FP64 iterative refinement around FP32 inner cycles: each sweep is one FP64 pass
//   x <- x + (pending inner update), s = b - A x, r0 = M^-1 s stored in FP32, |r0|,
// which stops at |r0| <= tol |r0 of the first sweep| + tol, or at the FP64 rounding floor (an
// inner cycle met its tolerance and yet the residual fell by less than half, or two sweeps in
// a row fell by less than half), and one FP32 GMRES cycle on M^-1 A d = r0, stopped at a relative
// residual of g.tol or after kmax steps (the symmetric systems: conjugate gradients to that
// residual).  x is double buffered between x and xalt.
template <class Op>
struct MixedJob {
  Op op;
  Work<float> g;
  double *x, *xalt;
  const double* b;
  int max_sweeps;
  double tol;
};
template <class Op>
__device__ __forceinline__ bool pass_refine(const Op& op, const Work<float>& g, Smem<Op>& sm, Sync& y, const double* xc,
                                            double* xn, const double* b, const double* scale, bool pending, bool first, bool raw) {
  constexpr int C = Op::C, M = Op::M;
  Shared& S = sm.S;
  const long long N = g.G.N;
  acc_clear(S);
  double rr = 0.0;
  IterateFill<Op, float> fill{g, S, ring_of<Op, float>(sm), xc, nullptr, b, nullptr, scale, pending ? S.nalpha : 0, N};
  auto emit = [&](int, const int (&eo)[C], const bool (&own)[C], const double (&wc)[M][C], double (&out)[M][C],
                  const typename Op::Emit& em, const typename IterateFill<Op, float>::Buf& u) {
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        if (pending && own[c]) xn[m * N + eo[c]] = wc[m][c];
        out[m][c] = u.b[m][c] - out[m][c];
      }
    if constexpr (kScalar<Op>) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const double id = 1.0 / (em.vd[c] + em.dg[c]), r = id * out[0][c];
        if (own[c]) {
          if (first) store_faces(op, eo[c], c, em, id);
          g.V0n[eo[c]] = (float)(raw ? out[0][c] : r);
          rr = fma(r, r, rr);
        }
      }
    } else {
      op.precond(em, out);
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (own[c]) {
            g.V0n[m * N + eo[c]] = (float)out[m][c];
            rr += out[m][c] * out[m][c];
          }
    }
  };
  for_tasks<Op::W>(g, [&](int task) { run_task<Op>(op, g.G, task, fill, emit); });
  rr = warp_sum(rr);
  if ((threadIdx.x & 31) == 0) S.acc[threadIdx.x >> 5][0] = rr;
  count(g, S, M + (pending ? S.nalpha * M : 0), (pending ? 3 : 2) * M + coef_planes(op));
  return pass_end<Op::W>(y, S, 1);
}
template <class Op>
__device__ __forceinline__ int mixed(const Op& op, Work<float> g, double* x, double* xalt, const double* b, int max_sweeps, double tol,
                     Smem<Op>& smd, Sync& y) {
  const auto op32 = krylov_op<float>(op);
  using Op32 = typename std::remove_const<decltype(op32)>::type;
  Smem<Op32>& sm = reinterpret_cast<Smem<Op32>&>(smd);  // the same Shared, a smaller A w buffer
  Shared& S = sm.S;
  double *xc = x, *xn = xalt;
  bool pending = false, inner_ok = false, scaled = false, x_live = true;
  bool cg = kSymmetric<Op> && g.kmax > 1;
  int stalls = 0, iters = 0, code = GM_MAXIT, free = 0;  // free: sweeps that do not count
  double tol_eff = 0.0, prev = INFINITY;
  for (int sweep = 0;; ++sweep) {
    const double* scale = nullptr;
    if constexpr (kSymmetric<Op>) scale = scaled ? op.idg : nullptr;
    if (!pass_refine(op, g, smd, y, xc, xn, b, scale, pending, sweep == 0, cg)) return GM_SYNC;
    float* f = g.V0;
    g.V0 = g.V0n;
    g.V0n = f;
    if (pending) {
      double* t = xc;
      xc = xn;
      xn = t;
      pending = false;
    }
    const double res = sqrt(S.red[0]);
    if (sweep == 0) tol_eff = tol * res + tol;
    if (!isfinite(res)) {
      code = GM_NONFINITE;
      break;
    }
    if (lead(g)) g.st->last_residual = res;
    stalls = res > 0.5 * prev ? stalls + 1 : 0;
    if (res <= tol_eff || (inner_ok && res > 0.5 * prev) || stalls >= 2) {
      code = GM_CONVERGED;
      break;
    }
    prev = res;
    if (sweep - free >= max_sweeps) break;
    if (lead(g)) g.st->refine_sweeps += 1;
    int c2 = GM_MAXIT;
    scaled = cg;
    if constexpr (kSymmetric<Op>) {
      // to the inner tolerance, full slots added to the iterate: cut off after one cycle as GMRES is, the sweeps
      // of an ill-conditioned system gain too little to end within their cap
      if (cg) c2 = cg_solve(op32, g, sm, y, g.tol * res + g.tol_abs, xc, x_live, iters);
    }
    if (!scaled) {
      if (threadIdx.x == 0) S.gam[0] = res;
      __syncthreads();
      c2 = gmres_cycle(op32, g, sm, y, g.tol * res + g.tol_abs, iters);
    }
    if (c2 == GM_SYNC || c2 == GM_NONFINITE) return c2;
    if (c2 == GM_BREAK) {  // not positive definite: GMRES from here on, with all its sweeps
      cg = false;
      prev = INFINITY;
      free = 1;
    }
    inner_ok = c2 == GM_CONVERGED;
    pending = true;
  }
  if (lead(g)) g.st->gmres_iters += iters;
  if (xc != x) {  // the result ends in x
    const long long n = (long long)Op::M * g.G.N;
    for (long long c = ((long long)blockIdx.x - g.first) * 32 * Op::W + threadIdx.x; c < n; c += (long long)g.nblk * 32 * Op::W)
      x[c] = xc[c];
  }
  return code;
}
template <class Op>
__device__ __forceinline__ void mixed_body(const MixedJob<Op>& j) {
  extern __shared__ __align__(16) unsigned char dsm[];
  Smem<Op>& sm = *reinterpret_cast<Smem<Op>*>(dsm);
  Op op = j.op;
  op.bind();
  Sync y = sync_begin(j.g, sm.S);
  if (lead(j.g)) j.g.st->gmres_solves += 1;
  const int code = mixed(op, j.g, j.x, j.xalt, j.b, j.max_sweeps, j.tol, sm, y);
  record_status(j.g, code);
  solve_end(j.g, sm.S, y, code != GM_SYNC);
}
template <class Op>
__global__ void __launch_bounds__(32 * Op::W, 1) k_mixed(const __grid_constant__ MixedJob<Op> j) {
  mixed_body(j);
}
template <class Op>
__global__ void __launch_bounds__(32 * Op::W, 1) k_mixed_jobs(const MixedJob<Op>* jobs, const int* map) {
  __shared__ JobCopy<MixedJob<Op>> s;
  mixed_body(copy_job(s, jobs + map[blockIdx.x]));
}

// ------------------------------------------------------------------ nested Newton
// Pressure_NestedNewton (implicit_operators.cpp:625-738).  A Newton iteration is one residual
// pass and one Jacobian solve whose update the next residual pass applies.  The residual pass
// forms, per cell, the iterate with the pending update, g = L p - a p + V_mod(p) - b, the
// slope V_slope(p), and r0 = -M^-1 g of the Jacobian solve that follows (so that solve starts
// with its A v_0 pass), and reduces |g|^2, |r0|^2, the floored cells and the smallest
// pressure.  The iterate alternates between p and pf so that the second residual pass, the
// last one of a solve without floored cells, leaves the result in p.
// TS = float: the Jacobian systems are solved in FP32 (the Newton loop is their refinement).
struct NewtonArgs {
  double *p, *pf, *g, *dp, *vdiag, *idg2;
  const double *b, *rho;
  DevScalars* sc;
  const unsigned long long* bkeys;  // min b / max V keys from k_pressure_rhs, or null: reduce here
};
template <class TS, bool kRK>
struct NewtonJob {
  PressureRow<double, kRK> op;
  Work<TS> g;
  NewtonArgs na;
};
// V(p) = rho e(rho, p) of the Redlich-Kwong gas and its slope (config.hpp:130-173, 206-239) from
// one inversion T(rho, p).  The slope is the derivative rho e_T / p_T at that T, where the
// reference differences two more inversions at p +- 1e-8; it only enters the Newton's Jacobian.
// The inversion iterates p(T) = K T - A / sqrt(T), K = R / (v - b), A = a / (v (v + b)).
__device__ __forceinline__ double rk_V(const DevParams& P, double rho, double p, double& slope) {
  const double v = 1.0 / rho, vb = v + P.m_b;
  const double K = P.m_R / (v - P.m_b), A = P.m_alfa / (v * vb), U = 1.5 * P.m_alfa / P.m_b * log(v / vb);
  double T_old, T = (v - P.m_b) * (p + P.m_alfa * rho * rho) / P.m_R, rs, df;
  int it = 0;
  do {
    T_old = T;
    rs = 1.0 / sqrt(T_old);
    df = K + 0.5 * A * rs / T_old;
    T = T_old - (K * T_old - A * rs - p) / df;
  } while (fabs(T - T_old) / fabs(T_old) > 1e-14 && ++it < kEosNewtonCap);
  if (it >= kEosNewtonCap) d_eos_flag = 1;
  rs = 1.0 / sqrt(T);
  slope = rho * (P.m_cv - 0.5 * U * rs / T) / (K + 0.5 * A * rs / T);
  return rho * (P.m_cv * T + U * rs);
}
// the residual pass's sums: |g|^2, |r0|^2, floored cells, smallest pressure
struct NewtonSums {
  double gg = 0.0, rr = 0.0, nf = 0.0, mn = INFINITY;
  __device__ __forceinline__ void add(const DevParams& P, double gv, double r0, double pv) {
    gg += gv * gv;
    rr += r0 * r0;
    if (pv < P.p_floor) nf += 1.0;
    mn = fmin(mn, pv);
  }
  template <int W>
  __device__ __forceinline__ bool end(Shared& S, Sync& y) {
    double t[4] = {gg, rr, nf, 0.0};
    const double s = warp_sum4(t);
    mn = warp_min(mn);
    const int lane = threadIdx.x & 31;
    if ((lane & 7) == 0 && lane < 24) S.acc[threadIdx.x >> 5][lane >> 3] = s;
    if (lane == 0) S.acc[threadIdx.x >> 5][3] = mn;
    return pass_end<W>(y, S, 4, 8u);
  }
};
// kFirst: the first residual pass of a Newton solve, which has no pending update and (ideal gas)
// leaves the face weights
template <bool kFirst, class Op, class TS>
__device__ __forceinline__ bool pass_newton(const Op& op, const Work<TS>& g, const NewtonArgs& na, Smem<Op>& sm, Sync& y,
                                            const double* pc, double* pn, double Mbig, const double* scale, double* idg,
                                            bool pending, bool dp_live, bool raw) {
  constexpr int C = Op::C;
  constexpr bool kRK = Op::kIsRK;
  const DevParams& P = op.P;
  Shared& S = sm.S;
  acc_clear(S);
  NewtonSums sum;
  using Fill = typename std::conditional<kFirst, RhsFill<Op, kRK>, IterateFill<Op, TS, kRK>>::type;
  auto emit = [&](int, const int (&eo)[C], const bool (&own)[C], const double (&wc)[1][C], double (&out)[1][C],
                  const typename Op::Emit& em, const typename Fill::Buf& u) {
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (own[c]) {
        const double pv = wc[0][c];
        double V, vs;
        if constexpr (kRK) {
          const bool fl = P.floor_on && !(pv >= P.p_floor);
          V = rk_V(P, u.r[c], fl ? P.p_floor : pv, vs);
          if (fl) {
            V += Mbig * (pv - P.p_floor);
            vs = Mbig;
          }
        } else {  // V_mod and V_slope of the ideal gas (config.hpp:206-239), a = 1 / (gamma - 1)
          const bool fl = P.floor_on && !(pv >= P.p_floor);
          V = fl ? fma(Mbig, pv - P.p_floor, op.a * P.p_floor) : op.a * pv;
          vs = fl ? Mbig : op.a;
        }
        const double gv = out[0][c] - op.a * pv + V - u.b[0][c];
        const double id = 1.0 / (vs + em.dg[c]);
        const double r0 = raw ? -gv * id : (double)(TS)(-gv * id);
        pn[eo[c]] = pv;
        if (!raw) {  // GMRES reads the right-hand side again at a restart, and the slopes
          na.g[eo[c]] = -gv;
          na.vdiag[eo[c]] = vs;
        }
        idg[eo[c]] = id;
        if (kFirst && !kRK) {
          op.kx[eo[c]] = em.kx[c];
          op.ky[eo[c]] = em.ky[c];
        }
        g.V0n[eo[c]] = (TS)(raw ? -gv : r0);
        sum.add(P, gv, r0, pv);
      }
  };
  if constexpr (kFirst) {
    Fill fill{pc, na.b, na.rho, 0};
    for_tasks<Op::W>(g, [&](int task) { run_task<Op>(op, g.G, task, fill, emit); });
  } else {
    Fill fill{g, S, ring_of<Op, TS>(sm), pc, dp_live ? na.dp : nullptr, na.b, na.rho, scale, pending ? S.nalpha : 0, 0};
    for_tasks<Op::W>(g, [&](int task) { run_task<Op>(op, g.G, task, fill, emit); });
  }
  count(g, S, 1 + (pending ? S.nalpha : 0),
        Op::kCoef + (kRK ? 1 : 0) + 4 + (raw ? 0 : 2) + (kFirst && !kRK ? 2 : 0) + (dp_live ? 1 : 0) + (scale ? 1 : 0));
  return sum.template end<Op::W>(S, y);
}
// The later residual passes of the ideal gas, while no cell of the iterate before was floored:
// L p from the face weights that the first pass left (two exchanges between columns instead of
// five, no means of h and e), and the preconditioner's diagonal from its reciprocal there, which
// only a newly floored cell changes.
template <class TS>
__device__ __forceinline__ bool pass_newton_faces(const PressureRow<double, false>& op, const Work<TS>& g,
                                                  const NewtonArgs& na, Smem<FaceRow<double>>& sm, Sync& y,
                                                  const double* pc, double* pn, double Mbig, const double* scale,
                                                  const double* id, double* idn, bool pending, bool dp_live) {
  using Op = FaceRow<double>;
  constexpr int C = Op::C;
  const DevParams& P = op.P;
  Shared& S = sm.S;
  acc_clear(S);
  NewtonSums sum;
  Op f{};
  f.kx = op.kx;
  f.ky = op.ky;
  f.idg = id;
  f.a = op.a;
  IterateFill<Op, TS> fill{g, S, ring_of<Op, TS>(sm), pc, dp_live ? na.dp : nullptr, na.b, na.rho, scale, pending ? S.nalpha : 0, 0};
  auto emit = [&](int, const int (&eo)[C], const bool (&own)[C], const double (&wc)[1][C], double (&out)[1][C],
                  const Op::Emit& em, const typename IterateFill<Op, TS>::Buf& u) {
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (own[c]) {
        const double pv = wc[0][c];
        double gv = out[0][c] - u.b[0][c], id = em.id[c];
        if (P.floor_on && !(pv >= P.p_floor)) {
          gv = out[0][c] - op.a * pv + fma(Mbig, pv - P.p_floor, op.a * P.p_floor) - u.b[0][c];
          id = 1.0 / (Mbig + (1.0 / id - op.a));
        }
        pn[eo[c]] = pv;
        idn[eo[c]] = id;
        g.V0n[eo[c]] = (TS)-gv;
        sum.add(P, gv, -gv * id, pv);
      }
  };
  for_tasks<Op::W>(g, [&](int task) { run_task<Op>(f, g.G, task, fill, emit); });
  count(g, S, 1 + (pending ? S.nalpha : 0), Op::kCoef + 4 + (dp_live ? 1 : 0));
  return sum.template end<Op::W>(S, y);
}
// V_mod and V_slope of the ideal gas where the pressure is below the floor (config.hpp:206-239)
__device__ __forceinline__ double floored_V(const PressureRow<double, false>& op, double Mbig, double pv) {
  return fma(Mbig, pv - op.P.p_floor, op.a * op.P.p_floor);
}
// The two residual passes of the ideal gas for tasks of many rows, with their rows copied ahead
// through the slots of the ring: 1024^2 and 2048^2 gain 6 and 8 % of the Newton solve, tasks of
// a few rows lose to the longer prologue (700 x 450, 4 rows a task, 4 %).
// The first residual pass of the ideal gas: no pending update; it leaves the face weights and the
// reciprocal of the preconditioner's diagonal for the passes that follow.
template <class TS>
__device__ __forceinline__ bool pass_first_staged(const PressureRow<double, false>& op, const Work<TS>& g,
                                                  const NewtonArgs& na, Smem<PressureRow<double, false>>& sm, Sync& y,
                                                  const double* pc, double* pn, double Mbig, double* idg, bool raw) {
  using Op = PressureRow<double, false>;
  constexpr int C = Op::C, kStage = 4, kRow = 4 * C * 32;  // a slot: p, h, eta, b
  const DevParams& P = op.P;
  Shared& S = sm.S;
  const int lane = threadIdx.x & 31;
  double* const stage = reinterpret_cast<double*>(sm.ring[threadIdx.x >> 5]) + lane;
  acc_clear(S);
  NewtonSums sum;
  for_tasks<Op::W>(g, [&](int task) {
    Op::State st{};
    double bl[C];
    int ol[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      bl[c] = 0.0;
      ol[c] = 0;
    }
    auto copy = [&](int it, int c, int n) {
      double* d = stage + (it & (kStage - 1)) * kRow + c * 32;
      copy_async(d, pc + n);
      copy_async(d + C * 32, op.hh + n);
      copy_async(d + 2 * C * 32, op.eta + n);
      copy_async(d + 3 * C * 32, na.b + n);
    };
    const StagedRows<C, kStage> R(g.G, task);
    R.start(copy);
#pragma unroll 1
    for (int it = 0; it < R.count(); ++it) {
      int on[C];
      R.wait(it, on);
      double w[1][C], bn[C], out[1][C], wc[1][C];
      Op::Row n;
      Op::Emit em;
      const double* d = stage + (it & (kStage - 1)) * kRow;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        w[0][c] = d[c * 32];
        n.h[c] = d[(C + c) * 32];
        n.e[c] = d[(2 * C + c) * 32];
        bn[c] = d[(3 * C + c) * 32];
        em.vd[c] = 0.0;  // V_mod takes the diagonal's place
      }
      R.next(it, copy);
      op.step(st, w, n, em, out, wc);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        if (it >= 2 && R.own[c]) {
          const int o = ol[c];
          const double pv = wc[0][c];
          const bool fl = P.floor_on && !(pv >= P.p_floor);
          const double vs = fl ? Mbig : op.a, V = fl ? floored_V(op, Mbig, pv) : op.a * pv;
          const double gv = out[0][c] + V - bl[c], id = 1.0 / (vs + em.dg[c]);
          const double r0 = raw ? -gv * id : (double)(TS)(-gv * id);
          pn[o] = pv;
          if (!raw) {  // GMRES reads the right-hand side again at a restart, and the slopes
            na.g[o] = -gv;
            na.vdiag[o] = vs;
          }
          idg[o] = id;
          op.kx[o] = em.kx[c];
          op.ky[o] = em.ky[c];
          g.V0n[o] = (TS)(raw ? -gv : r0);
          sum.add(P, gv, r0, pv);
        }
        bl[c] = bn[c];
        ol[c] = on[c];
      }
    }
  });
  count(g, S, 1, Op::kCoef + 6 + (raw ? 0 : 2));
  return sum.template end<Op::W>(S, y);
}
// The rows come through slots two ahead, with the vectors of the pending update; at most
// kMaxPending of them fit.
constexpr int kMaxPending = 8;
template <class TS>
__device__ __forceinline__ bool pass_faces_staged(const PressureRow<double, false>& op, const Work<TS>& g,
                                                  const NewtonArgs& na, Smem<FaceRow<double>>& sm, Sync& y,
                                                  const double* pc, double* pn, double Mbig, const double* id,
                                                  double* idn, bool pending, bool dp_live) {
  using Op = FaceRow<double>;
  constexpr int C = Op::C, kStage = 3, kRow = (6 + kMaxPending) * C * 32;
  static_assert(kStage * kRow * 8 <= Ring<Op, double>::kBytes, "the stages live in the ring");
  const DevParams& P = op.P;
  Shared& S = sm.S;
  const int lane = threadIdx.x & 31, nv = pending ? S.nalpha : 0;
  double* const stage = reinterpret_cast<double*>(sm.ring[threadIdx.x >> 5]);
  acc_clear(S);
  NewtonSums sum;
  Op f{};
  const double zero[C] = {};
  for_tasks<Op::W>(g, [&](int task) {
    Op::State st{};
    double bl[C], il[C];
    int ol[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      bl[c] = il[c] = 0.0;
      ol[c] = 0;
    }
    // a slot: p, b, kx, ky, id, the part of the update that is formed already, then the vectors
    int sc = 0, sr = 0;  // slots of the copies and of the row in work
    auto copy = [&](int, int c, int n) {
      double* d = stage + sc * kRow + lane + c * 32;
      copy_async(d, pc + n);
      copy_async(d + C * 32, na.b + n);
      copy_async(d + 2 * C * 32, op.kx + n);
      copy_async(d + 3 * C * 32, op.ky + n);
      copy_async(d + 4 * C * 32, id + n);
      if (dp_live) copy_async(d + 5 * C * 32, na.dp + n);
      TS* t = reinterpret_cast<TS*>(stage + sc * kRow + 6 * C * 32) + lane + c * 32;
      const TS* v = g.V + n + g.G.N;
      if (nv > 0) copy_async(t, g.V0 + n);
      for (int i = 1; i < nv; ++i, v += g.G.N) copy_async(t + i * C * 32, v);
      if (c == C - 1) sc = sc == kStage - 1 ? 0 : sc + 1;
    };
    const StagedRows<C, kStage> R(g.G, task);
    R.start(copy);
#pragma unroll 1
    for (int it = 0; it < R.count(); ++it) {
      int on[C];
      R.wait(it, on);
      double w[C], bn[C], in[C], out[C], wc[C];
      Op::Row n;
      const double* d = stage + sr * kRow + lane;
      const TS* t = reinterpret_cast<const TS*>(stage + sr * kRow + 6 * C * 32) + lane;
      sr = sr == kStage - 1 ? 0 : sr + 1;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        bn[c] = d[(C + c) * 32];
        n.kx[c] = d[(2 * C + c) * 32];
        n.ky[c] = d[(3 * C + c) * 32];
        in[c] = d[(4 * C + c) * 32];
        double v = 0.0;
#pragma unroll
        for (int i = 0; i < kMaxPending; ++i)
          if (i < nv) v = fma(S.coef[i], (double)t[(i * C + c) * 32], v);
        w[c] = d[c * 32] + fma(in[c], v, dp_live ? d[(5 * C + c) * 32] : 0.0);
        wc[c] = st.x[c];
      }
      R.next(it, copy);
      f.complete(st, w, n, zero, out);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        if (it >= 2 && R.own[c]) {
          const int o = ol[c];
          const double pv = wc[c];
          const bool fl = P.floor_on && !(pv >= P.p_floor);
          const double gv = out[c] + (fl ? floored_V(op, Mbig, pv) : op.a * pv) - bl[c];
          const double ic = fl ? 1.0 / (Mbig + (1.0 / il[c] - op.a)) : il[c];
          pn[o] = pv;
          idn[o] = ic;
          g.V0n[o] = (TS)-gv;
          sum.add(P, gv, -gv * ic, pv);
        }
        bl[c] = bn[c];
        il[c] = in[c];
        ol[c] = on[c];
      }
    }
  });
  count(g, S, 1 + nv, 7 + (dp_live ? 1 : 0));
  return sum.template end<Op::W>(S, y);
}
template <class TS, bool kRK, bool kLong>
__device__ __forceinline__ int newton(const PressureRow<double, kRK>& op, Work<TS> g, const NewtonArgs& na,
                      Smem<PressureRow<double, kRK>>& smd, Sync& y) {
  using L = PressureRow<double, kRK>;
  auto J = krylov_op<TS>(op);
  using JOp = decltype(J);
  if constexpr (kRK) {
    J.jac = 1;
    J.vdiag = na.vdiag;
  }
  Smem<JOp>& sm = reinterpret_cast<Smem<JOp>&>(smd);
  Shared& S = sm.S;
  const DevParams& P = op.P;
  const long long N = g.G.N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // ---- Cor. 1 slope Mbig (implicit_operators.cpp:670-686)
  double Mbig = na.sc->Mbig;
  if (P.floor_on) {
    double bmin, vmax = -INFINITY;
    if (na.bkeys) {
      const unsigned long long kb = na.bkeys[0], kv = ~na.bkeys[1];
      bmin = kb == ~0ull ? INFINITY : dkey_value(kb);
      if (kv != 0ull) vmax = dkey_value(kv);
    } else {
      double m0 = INFINITY, m1 = INFINITY;
      for (long long c = ((long long)blockIdx.x - g.first) * 32 * L::W + threadIdx.x; c < N; c += (long long)g.nblk * 32 * L::W) {
        m0 = fmin(m0, na.b[c]);
        if (kRK) {
          const double v = Vbase(P, P.p_floor, __ldg(na.rho + c));
          if (isfinite(v)) m1 = fmin(m1, -v);
        }
      }
      m0 = warp_min(m0);
      m1 = warp_min(m1);
      acc_clear(S);
      if (lane == 0) {
        S.acc[warp][0] = m0;
        S.acc[warp][1] = m1;
      }
      if (!pass_end<L::W>(y, S, 2, 3u)) return GM_SYNC;
      bmin = S.red[0];
      if (kRK) vmax = -S.red[1];
      count(g, S, 0, kRK ? 2 : 1);
    }
    double Vpe = P.p_floor / (P.gamma - 1.0);
    if (kRK && vmax > Vpe) Vpe = vmax;
    const double q = Vpe - bmin;
    const double M_cor = ((0.0 < q) ? q : 0.0) / ((1.0 - P.theta) * P.p_floor);
    const double M_base = P.Mbig_fac / (P.gamma - 1.0);
    Mbig = (M_base < M_cor) ? M_cor : M_base;
    if (lead(g)) na.sc->Mbig = Mbig;
  }
  double res0 = -1.0;
  double *pc = na.p, *pn = na.pf;
  // 1 / precP's diagonal: a residual pass writes one plane while it scales the pending update by
  // the other (the slopes of floored cells change between Newton iterations)
  double *id = op.idg, *idn = kRK ? op.idg : na.idg2;
  bool pending = false, dp_live = false, scaled = false;
  bool cg = !kRK && g.kmax > 1, faces = false, put_slopes = false;
  Smem<FaceRow<double>>& sm_faces = reinterpret_cast<Smem<FaceRow<double>>&>(smd);
  int it, iters = 0, worst = GM_CONVERGED;
  int free = 0;  // iterations that do not count
  constexpr int kMore = 3;
  int more = 0;
  for (it = 0; it - free < P.Pnewton_max; ++it) {
    const double* scale = scaled ? id : nullptr;
    bool ok = false;
    if constexpr (kRK) {
      ok = it == 0 ? pass_newton<true>(op, g, na, smd, y, pc, pn, Mbig, scale, idn, false, false, cg)
                   : pass_newton<false>(op, g, na, smd, y, pc, pn, Mbig, scale, idn, pending, dp_live, cg);
    } else if (it == 0) {
      if constexpr (kLong) ok = pass_first_staged(op, g, na, smd, y, pc, pn, Mbig, idn, cg);
      else ok = pass_newton<true>(op, g, na, smd, y, pc, pn, Mbig, scale, idn, false, false, cg);
    } else if (faces && (!kLong || (scaled && (!pending || S.nalpha <= kMaxPending)))) {
      if constexpr (kLong) ok = pass_faces_staged(op, g, na, sm_faces, y, pc, pn, Mbig, id, idn, pending, dp_live);
      else ok = pass_newton_faces(op, g, na, sm_faces, y, pc, pn, Mbig, scale, id, idn, pending, dp_live);
    } else {
      ok = pass_newton<false>(op, g, na, smd, y, pc, pn, Mbig, scale, idn, pending, dp_live, cg);
    }
    if (!ok) return GM_SYNC;
    put_slopes = cg;
    {
      double* q = id;
      id = idn;
      idn = q;
    }
    J.idg = id;
    {
      double* t = pc;
      pc = pn;
      pn = t;
      TS* f = g.V0;
      g.V0 = g.V0n;
      g.V0n = f;
    }
    pending = false;
    const double res = sqrt(S.red[0]);
    if (it == 0) res0 = res;
    if (!isfinite(res)) {
      worst = GM_NONFINITE;
      break;
    }
    if (res < P.Pnewton_tol * res0 + P.Pnewton_tol) {
      // The FP32 solves can leave the residual just below the tolerance, and the tolerance can leave a pressure
      // below a floor smaller than itself, where an FP64 solve has gone far beyond: further iterations then,
      // at most kMore, before that counts as IMEX_POSITIVITY.
      if (!std::is_same<TS, float>::value || !P.floor_on || !(S.red[3] < P.theta * P.p_floor - 1e-14) || more >= kMore ||
          it + 1 - free >= P.Pnewton_max)
        break;
      ++more;
    }
    // ---- Jacobian solve J dp = -g (GMRES with precP) from dp = 0
    if (lead(g)) {
      g.st->gmres_solves += 1;
      g.st->newton_iters += 1;
    }
    faces = cg && S.red[2] == 0.0;
    if constexpr (!kRK) {
      // conjugate gradients take the slope of a cell from its pressure; without floored cells
      // every slope is the constant a and the passes read nothing
      J.p = cg && S.red[2] > 0.0 ? pc : nullptr;
      J.vdiag = cg ? nullptr : na.vdiag;
      J.p_floor = P.p_floor;
      J.Mbig = Mbig;
    }
    const double r0 = sqrt(S.red[1]), tol_eff = g.tol * r0 + g.tol_abs;
    if (!isfinite(r0)) {
      record_status(g, GM_NONFINITE);
      return GM_NONFINITE;
    }
    __syncthreads();
    dp_live = false;
    int code = GM_CONVERGED;
    if (r0 <= tol_eff) {
      if (threadIdx.x == 0) S.nalpha = 0;
      if (lead(g)) g.st->last_residual = r0;
      __syncthreads();
    } else {
      if (threadIdx.x == 0) S.gam[0] = r0;
      __syncthreads();
      scaled = cg;
      if constexpr (!kRK) {
        if (cg) code = cg_solve(J, g, sm, y, tol_eff, na.dp, dp_live, iters);
      }
      if (scaled && (code == GM_BREAK || code == GM_MAXIT)) {
        // not positive definite, or more steps than GMRES may take: the update so far is this iteration's, which
        // does not count; GMRES takes the next
        cg = faces = false;
        code = GM_CONVERGED;
        free = 1;
      }
      for (int outer = 0; !scaled; ++outer) {
        code = gmres_cycle(J, g, sm, y, tol_eff, iters);
        if (code != GM_MAXIT || outer + 1 >= g.max_restarts) break;
        apply_update<1, L::W>(g, S, na.dp, !dp_live);
        dp_live = true;
        if (!pass_end<L::W>(y, S, 1)) return GM_SYNC;
        if (!pass_residual<false>(J, g, S, y, na.dp, na.g)) return GM_SYNC;
        const double r = sqrt(S.red[0]);
        __syncthreads();
        if (threadIdx.x == 0) {
          S.gam[0] = r;
          S.nalpha = 0;
        }
        __syncthreads();
        if (!isfinite(r)) {
          code = GM_NONFINITE;
          break;
        }
        if (r <= tol_eff) {
          if (lead(g)) g.st->last_residual = r;
          code = GM_CONVERGED;
          break;
        }
      }
    }
    if (code != GM_CONVERGED) {
      record_status(g, code);
      if (code != GM_MAXIT) {
        if (lead(g)) g.st->gmres_iters += iters;
        return code;
      }
    }
    pending = true;
  }
  if (lead(g)) g.st->gmres_iters += iters;
  if (it - free == P.Pnewton_max && lead(g)) atomicMax(&g.st->status, (int)IMEX_NEWTON_MAXIT);
  // ---- the result in p; floored cells and smallest pressure (implicit_operators.cpp:722-737), and the
  // slopes of the last residual pass's iterate, which are the J mode's from here on (the reference's
  // p_freeze), unless that pass wrote them: conjugate gradients do without the plane, so it is written once
  // a solve instead of once a pass
  auto put_slope = [&](long long c, double pv) {
    if (put_slopes) na.vdiag[c] = P.floor_on && !(pv >= P.p_floor) ? Mbig : op.a;
  };
  if (pending || pc != na.p || P.Pnewton_max <= 0) {
    double nf = 0.0, mn = INFINITY;
    const int na_ = S.nalpha;
    for (long long c = ((long long)blockIdx.x - g.first) * 32 * L::W + threadIdx.x; c < N; c += (long long)g.nblk * 32 * L::W) {
      double pv = pc[c];
      put_slope(c, pv);
      if (pending) {
        double d = 0.0;
        for (int i = 0; i < na_; ++i) d = fma(S.coef[i], ldv(basis<L>(g, i) + c), d);
        pv += fma(scaled ? id[c] : 1.0, d, dp_live ? na.dp[c] : 0.0);
      }
      na.p[c] = pv;
      if (pv < P.p_floor) nf += 1.0;
      mn = fmin(mn, pv);
    }
    count(g, S, pending ? na_ : 0, 2);
    if ((pending || P.Pnewton_max <= 0) && P.floor_on) {
      nf = warp_sum(nf);
      mn = warp_min(mn);
      acc_clear(S);
      if (lane == 0) {
        S.acc[warp][2] = nf;
        S.acc[warp][3] = mn;
      }
      if (!pass_end<L::W>(y, S, 4, 8u)) return GM_SYNC;
    }
  } else if (put_slopes) {
    // without floored cells every slope is the constant a, and the iterate is not read
    const bool floored = P.floor_on && !(S.red[2] == 0.0 && isfinite(S.red[0]));
    for (long long c = ((long long)blockIdx.x - g.first) * 32 * L::W + threadIdx.x; c < N; c += (long long)g.nblk * 32 * L::W)
      put_slope(c, floored ? pc[c] : INFINITY);
  }
  if (put_slopes) count(g, S, 0, 1);
  if (P.floor_on && lead(g)) {
    const double nf = S.red[2], pmin = S.red[3];
    if ((int)nf > g.st->max_floored) g.st->max_floored = (int)nf;
    if (pmin < g.st->min_p) g.st->min_p = pmin;
    if (pmin < P.theta * P.p_floor - 1e-14) atomicMax(&g.st->status, (int)IMEX_POSITIVITY);
  }
  return worst;
}
template <bool kLong, class TS, bool kRK>
__device__ __forceinline__ void newton_body(const NewtonJob<TS, kRK>& j) {
  using Op = PressureRow<double, kRK>;
  extern __shared__ __align__(16) unsigned char dsm[];
  Smem<Op>& sm = *reinterpret_cast<Smem<Op>*>(dsm);
  Op op = j.op;
  if (!kRK) op.P.eos_type = IMEX_IDEAL_GAS;
  op.bind();
  Sync y = sync_begin(j.g, sm.S);
  const int code = newton<TS, kRK, kLong>(op, j.g, j.na, sm, y);
  record_status(j.g, code);
  solve_end(j.g, sm.S, y, code != GM_SYNC);
}
template <class TS, bool kRK, bool kLong>
__global__ void __launch_bounds__(32 * PressureRow<double, kRK>::W, 1)
    k_newton(const __grid_constant__ NewtonJob<TS, kRK> j) {
  newton_body<kLong>(j);
}
template <class TS, bool kRK>
__global__ void __launch_bounds__(32 * PressureRow<double, kRK>::W, 1)
    k_newton_jobs(const NewtonJob<TS, kRK>* jobs, const int* map) {
  __shared__ JobCopy<NewtonJob<TS, kRK>> s;
  newton_body<false>(copy_job(s, jobs + map[blockIdx.x]));
}

// ------------------------------------------------------------------ host side
// every device-wide wait gives up after barrier_timeout_s, counted at the maximum SM clock
long long wait_cycles(const imex_ctx* ctx) {
  const double khz = ctx->clock_khz > 0 ? (double)ctx->clock_khz : 2.0e6;
  return (long long)(ctx->barrier_timeout_s * khz * 1e3) + 1;
}

// The cut of a grid into tasks for at most `cap` blocks.  Strips are as wide as the lanes
// allow, evened out; a run has as many rows as give every warp one task, at least kMinRows (its
// halo rows are formed twice; two rows against four made the 64^2 solves 22 % faster, since a
// pass lasts as long as its rows one after another); tasks go evenly to as many blocks as leave
// each kMinTasks of them, since every block adds to the cost of a pass end.
constexpr int kMinRows = 2, kMinTasks = 4;
struct Cut {
  Geom G;
  int nblk, per;
};
template <class Op>
Cut make_cut(const imex_ctx* ctx, int cap) {
  Cut k{};
  Geom& G = k.G;
  G.nx = ctx->nx;
  G.ny = ctx->ny;
  G.xclamp = ctx->P.xclamp;
  G.yclamp = ctx->P.yclamp;
  G.N = (long long)ctx->N;
  const int widest = 32 * Op::C - 2 * Op::H;
  const int strips = (G.nx + widest - 1) / widest;
  G.wd = (G.nx + strips - 1) / strips;
  const long long warps = (long long)cap * Op::W;
  const long long runs = warps / strips > 1 ? warps / strips : 1;
  int L = (int)((G.ny + runs - 1) / runs);
  if (L < kMinRows) L = kMinRows;
  G.L = L;
  G.nseg = (G.ny + L - 1) / L;
  G.ntask = strips * G.nseg;
  k.per = (G.ntask + cap - 1) / cap;
  if (k.per < kMinTasks) k.per = kMinTasks;
  k.nblk = (G.ntask + k.per - 1) / k.per;
  return k;
}
// blocks of one launch that are resident together: one per SM (the launch bounds)
template <class Op, class K>
int capacity(imex_ctx* ctx, K kernel, size_t smem) {
  int per_sm = 0;
  cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)kernel, 32 * Op::W, smem);
  if (per_sm < 1) return 0;
  const int n = ctx->num_sms;
  return n < kMaxBlocks ? n : kMaxBlocks;
}

template <class TS>
TS* basis_of(imex_ctx* ctx) {
  if constexpr (std::is_same<TS, double>::value) return ctx->V;
  else return ctx->Vf;
}
template <class TS>
Work<TS> make_work(imex_ctx* ctx, const Cut& k, int M, int fam) {
  Work<TS> g{};
  g.V = basis_of<TS>(ctx);
  if constexpr (std::is_same<TS, double>::value) g.AV = ctx->AV;
  else g.AV = ctx->AVf;
  g.V0 = g.V;
  // the second first-vector: the basis arrays hold three planes per vector, of which a
  // one-component solve uses one; the mixed magnetic solves use the refinement residual's planes
  if (M == 1) g.V0n = g.V + (long long)(ctx->cfg.gmres_restart + 1) * (long long)ctx->N;
  else g.V0n = reinterpret_cast<TS*>(ctx->mres);
  g.s[0] = reinterpret_cast<TS*>(ctx->pg);
  g.s[1] = reinterpret_cast<TS*>(ctx->pdp);
  g.partial = ctx->partial;
  g.sync = ctx->sync;
  g.st = ctx->st;
  g.kmax = ctx->cfg.gmres_restart;
  // 0 = the system's dimension, as the reference's outmax = dim (implicit_operators.cpp:802)
  const long long dim = (long long)M * (long long)ctx->N;
  g.max_restarts = ctx->cfg.gmres_max_restarts > 0 ? ctx->cfg.gmres_max_restarts
                                                   : (int)(dim > 2000000000LL ? 2000000000LL : dim);
  g.fam = fam;
  g.nblk = k.nblk;
  g.per = k.per;
  g.first = 0;
  g.wait_cycles = wait_cycles(ctx);
  g.tol = ctx->P.GMREStol;
  g.tol_abs = ctx->P.GMREStol;
  if (std::is_same<TS, float>::value) g.tol = ctx->cfg.mixed_inner_tol;
  g.G = k.G;
  return g;
}
bool is_mixed(const imex_ctx* ctx, int kind) {
  return ctx->cfg.precision == IMEX_PRECISION_MIXED && (ctx->cfg.mixed_solves & kind) != 0;
}
double outer_tol(const imex_ctx* ctx) {
  return ctx->cfg.mixed_outer_tol > 0.0 ? ctx->cfg.mixed_outer_tol : ctx->P.GMREStol;
}

template <class Op>
Op make_op(imex_ctx* ctx, bool jac = false) {
  Op o{};
  o.P = ctx->P;
  o.sc = ctx->sc;
  if constexpr (std::is_base_of<PressureCoef, Op>::value) {
    o.hh = ctx->hh;
    o.eta = ctx->eta;
    o.vscale = ctx->vscale;
    o.vdiag = ctx->vdiag;
    o.idg = ctx->mx;
    o.kx = ctx->mx + ctx->N;
    o.ky = ctx->mx + 2 * ctx->N;
    o.jac = jac;
  } else if constexpr (std::is_base_of<EnergyCoef, Op>::value) {
    o.hh = ctx->hh;
    o.idg = ctx->mx;
    o.kx = ctx->mx + ctx->N;
    o.ky = ctx->mx + 2 * ctx->N;
  } else {
    o.Qe = ctx->Qe;
    if constexpr (std::is_base_of<MagBCoef, Op>::value) o.rho = ctx->cons;
    else o.irho = ctx->irho;
  }
  return o;
}

template <class Op, class K, class Job>
imex_status launch_one(imex_ctx* ctx, K kernel, const Job& job, int nblk, size_t smem) {
  void* params[] = {(void*)&job};
  return cuda_check(ctx, cudaLaunchCooperativeKernel((const void*)kernel, dim3(nblk), dim3(32 * Op::W), params, smem, ctx->stream),
                    "cooperative launch");
}

// Op: the FP64 solve's operator; MOp: the mixed form's
template <class Op, class MOp = Op>
imex_status solve(imex_ctx* ctx, bool jac, int fam, int kind, double* x, const double* b, const Scratch* scratch) {
  prof_begin(ctx);
  imex_status s;
  if (scratch || !is_mixed(ctx, kind)) {
    const size_t smem = sizeof(Smem<Op>);
    GmresJob<Op> j{};
    const int cap = capacity<Op>(ctx, k_gmres<Op>, smem);
    if (cap < 1) return set_error(ctx, IMEX_ERR_CUDA, "solver kernel does not fit on an SM");
    const Cut k = make_cut<Op>(ctx, cap);
    j.op = make_op<Op>(ctx, jac);
    j.g = make_work<double>(ctx, k, Op::M, fam);
    if (scratch) {
      j.g.V = j.g.V0 = scratch->V;
      j.g.AV = scratch->AV;
      j.g.partial = scratch->partial;
      j.g.sync = scratch->sync;
    }
    j.x = x;
    j.b = b;
    s = launch_one<Op>(ctx, k_gmres<Op>, j, k.nblk, smem);
  } else {
    const size_t smem = sizeof(Smem<MOp>);
    MixedJob<MOp> j{};
    const int cap = capacity<MOp>(ctx, k_mixed<MOp>, smem);
    if (cap < 1) return set_error(ctx, IMEX_ERR_CUDA, "solver kernel does not fit on an SM");
    const Cut k = make_cut<MOp>(ctx, cap);
    j.op = make_op<MOp>(ctx, jac);
    j.g = make_work<float>(ctx, k, MOp::M, fam);
    j.g.tol_abs = 0.0;
    j.x = x;
    j.xalt = ctx->mcor;
    j.b = b;
    j.max_sweeps = ctx->cfg.mixed_max_refine;
    j.tol = outer_tol(ctx);
    s = launch_one<MOp>(ctx, k_mixed<MOp>, j, k.nblk, smem);
  }
  prof_end(ctx, fam, 0.0, 1);
  return s;
}

template <class TS, bool kRK>
NewtonJob<TS, kRK> newton_job(imex_ctx* ctx, const Cut& k, double* p, const double* b, int keys) {
  NewtonJob<TS, kRK> j{};
  j.op = make_op<PressureRow<double, kRK>>(ctx);
  j.g = make_work<TS>(ctx, k, 1, F_NEWTON);
  // pg and pdp are the Newton's own: the conjugate gradients' planes come from the spare part of
  // the basis array (see make_work)
  j.g.s[0] = j.g.V0n + ctx->N;
  j.g.s[1] = j.g.s[0] + ctx->N;
  j.na.p = p;
  j.na.pf = ctx->pf;
  j.na.g = ctx->pg;
  j.na.dp = ctx->pdp;
  j.na.vdiag = ctx->vdiag;
  j.na.idg2 = ctx->mx + 3 * ctx->N;
  j.na.b = b;
  j.na.rho = ctx->cons;
  j.na.sc = ctx->sc;
  j.na.bkeys = keys ? ctx->sc->bkey[keys - 1] : nullptr;
  return j;
}
// rows per task from which the residual passes copy their rows ahead (pass_first_staged)
constexpr int kLongRows = 8;
template <class TS, bool kRK>
imex_status newton_one(imex_ctx* ctx, double* p, const double* b, int keys) {
  using Op = PressureRow<double, kRK>;
  const size_t smem = sizeof(Smem<Op>);
  const int cap = capacity<Op>(ctx, k_newton<TS, kRK, false>, smem);
  if (cap < 1) return set_error(ctx, IMEX_ERR_CUDA, "solver kernel does not fit on an SM");
  const Cut k = make_cut<Op>(ctx, cap);
  const NewtonJob<TS, kRK> j = newton_job<TS, kRK>(ctx, k, p, b, keys);
  prof_begin(ctx);
  imex_status s;
  // both instances have one block per SM, so the cut fits either
  if (!kRK && k.G.L >= kLongRows && capacity<Op>(ctx, k_newton<TS, kRK, !kRK>, smem) >= k.nblk)
    s = launch_one<Op>(ctx, k_newton<TS, kRK, !kRK>, j, k.nblk, smem);
  else
    s = launch_one<Op>(ctx, k_newton<TS, kRK, false>, j, k.nblk, smem);
  prof_end(ctx, F_NEWTON, 0.0, 1);
  return s;
}

// ---- ensembles: one cooperative launch (or a few chunks) for all members.  A chunk's blocks go to
// its members in proportion to their cells, at least one each and no more than their tasks fill.
//
// Chunks run one after another, each for as long as its slowest member.  A pass of a member lasts
// about as long as the rows of its tasks one after another, plus a pass end of some four rows
// (kEndRows).  Members are sorted by cells, and of the ways to cut their order into chunks of at most
// a block each (at every 24th of the members) the one is taken whose chunks' longest passes add up to
// the least: small members share a launch, a block each, and large ones have blocks to spare.  Ensemble
// steps, ms, tile kernels / chunks of half the blocks, dealt in turn / cut like this:
// 256 members of sides 64 to 256 35.1 / 38.0 / 24.4, 80 of 64 to 256 9.9 / 9.5 / 8.0, 256 of 16 to 64 4.41 /
// 5.10 / 3.61, 400 of 16 to 64 6.31 / 7.94 / 5.25, 80 of 8 to 60 1.22 / 1.84 / 1.33, 150 of 8 to 60 2.05 / 2.90 /
// 2.28.
constexpr int kEndRows = 4;
template <class Op, class Job, class K, class Make>
imex_status add_chunks(BatchSolvePlan* plan, const std::vector<imex_ctx*>& members, K kernel, size_t smem, Make make) {
  imex_ctx* c0 = members[0];
  const int cap = capacity<Op>(c0, kernel, smem);
  if (cap < 1) return set_error(c0, IMEX_ERR_CUDA, "batched solve kernel does not fit on an SM");
  const int nm = (int)members.size();
  std::vector<int> order(nm);
  for (int m = 0; m < nm; ++m) order[m] = m;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return members[a]->N > members[b]->N; });
  // the cut of every member of a chunk
  auto cuts = [&](const std::vector<int>& grp) {
    const int n = (int)grp.size();
    double cells = 0.0;
    for (int m : grp) cells += (double)members[m]->N;
    std::vector<Cut> k;
    for (int m : grp) k.push_back(make_cut<Op>(members[m], 1 + (int)((double)(cap - n) * (double)members[m]->N / cells)));
    return k;
  };
  auto slowest = [&](int from, int to) {
    long long rows = 0;
    for (const Cut& k : cuts(std::vector<int>(order.begin() + from, order.begin() + to)))
      rows = std::max(rows, kEndRows + (long long)((k.per + Op::W - 1) / Op::W) * (k.G.L + 2 * Op::H));
    return rows;
  };
  const int step = std::max(1, std::min(nm / 24, cap));
  std::vector<int> at;  // where a chunk may end
  for (int i = 0; i < nm; i += step) at.push_back(i);
  if (nm > cap) at.push_back(nm - cap);
  at.push_back(nm);
  std::sort(at.begin(), at.end());
  const int np = (int)at.size();
  std::vector<long long> least(np, -1);  // rows of the chunks up to there, and where the last one begins
  std::vector<int> begin(np, 0);
  least[0] = 0;
  for (int e = 1; e < np; ++e)
    for (int a = 0; a < e; ++a) {
      if (at[e] - at[a] > cap || least[a] < 0) continue;
      const long long rows = least[a] + (at[e] > at[a] ? slowest(at[a], at[e]) : 0);
      if (least[e] < 0 || rows < least[e]) {
        least[e] = rows;
        begin[e] = a;
      }
    }
  std::vector<std::vector<int>> groups;
  for (int e = np - 1; e > 0; e = begin[e])
    groups.insert(groups.begin(), std::vector<int>(order.begin() + at[begin[e]], order.begin() + at[e]));
  for (const std::vector<int>& grp : groups) {
    if (grp.empty()) continue;
    const int n = (int)grp.size();
    const std::vector<Cut> cut = cuts(grp);
    std::vector<Job> jobs;
    std::vector<int> map;
    int first = 0;
    for (int q = 0; q < n; ++q) {
      const Cut& k = cut[q];
      Job j = make(members[grp[q]], k);
      j.g.first = first;
      jobs.push_back(j);
      for (int u = 0; u < k.nblk; ++u) map.push_back(q);
      first += k.nblk;
    }
    Job* d_jobs = nullptr;
    int* d_map = nullptr;
    cudaError_t e = cudaMalloc(&d_jobs, jobs.size() * sizeof(Job));
    if (e == cudaSuccess) plan->dev.push_back(d_jobs);
    if (e == cudaSuccess) e = cudaMalloc(&d_map, map.size() * sizeof(int));
    if (e == cudaSuccess) plan->dev.push_back(d_map);
    if (e == cudaSuccess) e = cudaMemcpy(d_jobs, jobs.data(), jobs.size() * sizeof(Job), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d_map, map.data(), map.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_check(c0, e, "batched solve set-up");
    const int blocks = first;
    BatchChunk ch;
    ch.ctas = blocks;
    ch.members = n;
    ch.launch = [=](cudaStream_t st) {
      const Job* dj = d_jobs;
      const int* dm = d_map;
      void* params[] = {(void*)&dj, (void*)&dm};
      return cudaLaunchCooperativeKernel((const void*)kernel, dim3(blocks), dim3(32 * Op::W), params, smem, st);
    };
    plan->chunks.push_back(ch);
  }
  return IMEX_OK;
}
template <class Op, class MOp = Op, class Sys>
imex_status add_solves(BatchSolvePlan* plan, const std::vector<imex_ctx*>& members, int kind, int fam, Sys system) {
  if (!is_mixed(members[0], kind))
    return add_chunks<Op, GmresJob<Op>>(plan, members, k_gmres_jobs<Op>, sizeof(Smem<Op>), [&](imex_ctx* m, const Cut& k) {
      GmresJob<Op> j{};
      j.op = make_op<Op>(m);
      j.g = make_work<double>(m, k, Op::M, fam);
      system(m, &j.x, &j.b);
      return j;
    });
  return add_chunks<MOp, MixedJob<MOp>>(plan, members, k_mixed_jobs<MOp>, sizeof(Smem<MOp>), [&](imex_ctx* m, const Cut& k) {
    MixedJob<MOp> j{};
    j.op = make_op<MOp>(m);
    j.g = make_work<float>(m, k, MOp::M, fam);
    j.g.tol_abs = 0.0;
    system(m, &j.x, &j.b);
    j.xalt = m->mcor;
    j.max_sweeps = m->cfg.mixed_max_refine;
    j.tol = outer_tol(m);
    return j;
  });
}
template <class TS, bool kRK>
imex_status add_newtons(BatchSolvePlan* plan, const std::vector<imex_ctx*>& members) {
  using Op = PressureRow<double, kRK>;
  return add_chunks<Op, NewtonJob<TS, kRK>>(plan, members, k_newton_jobs<TS, kRK>, sizeof(Smem<Op>),
                                            [&](imex_ctx* m, const Cut& k) {
                                              // one plan serves both pressure solves of a stage: no keys
                                              return newton_job<TS, kRK>(m, k, m->pp, m->pb, 0);
                                            });
}
void energy_system(imex_ctx* m, double** x, const double** b) {
  *x = m->cons + 4 * m->N;
  *b = m->pb;
}
void pressure_system(imex_ctx* m, double** x, const double** b) {
  *x = m->pp;
  *b = m->pb;
}
void magnetic_system(imex_ctx* m, double** x, const double** b) {
  int op;
  mag_system(m, &op, x, b);
}

}  // namespace
}  // namespace march
}  // namespace imex
