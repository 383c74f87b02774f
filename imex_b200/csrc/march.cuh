// Row-marching passes of the implicit solves.
//
// A pass over the grid (a residual, or one Arnoldi step) is cut into tasks, one warp each: a
// strip of columns (the lanes, plus the stencil's halo columns) and a run of rows.  The warp
// marches up its strip: it forms the next row of the vector (a combination of Krylov vectors,
// or an iterate plus its pending update) for all its columns, halo included, and applies the
// operator to the row it has completed.  Rows below stay in registers, column neighbours come
// by shuffle and every face quantity is formed once, so a pass has no shared tile, no block
// barrier and no staged index arithmetic; the warps of an SM drift apart and one warp's loads
// overlap another's arithmetic.
#pragma once

#include <type_traits>

#include "cells.cuh"

namespace imex {
namespace march {

constexpr int kMaxWarps = 16;         // warps per block (an operator's W), one block per SM
constexpr int kCap = 30;              // largest supported restart length
constexpr int kSlots = kCap + 2;      // partial-sum slots per block

__device__ __forceinline__ double ldv(const double* p) { return *p; }
__device__ __forceinline__ double ldv(const float* p) { return (double)*p; }

// ------------------------------------------------------------------ geometry
struct Geom {
  int nx, ny;
  int wd, nseg, L;   // own columns per strip, runs per strip, rows per run
  int ntask;         // strips * nseg
  int xclamp, yclamp;
  long long N;
};
// A clamped halo column is column nx - 1; lanes past it may hold any cell, and take different
// ones (mirrored): asynchronous copies of one address by many lanes are served one after another,
// which made the last strip of an open 700 x 450 grid, ten columns wide, 50 % slower.
__device__ __forceinline__ int map_x(const Geom& G, int x) {
  if (x < 0) return G.xclamp ? 0 : x + G.nx;
  if (x >= G.nx) {
    const int w = x - G.nx, m = G.nx - 1 - w;
    return G.xclamp || w >= G.nx ? (m > 0 ? m : 0) : w;
  }
  return x;
}
__device__ __forceinline__ int map_y(const Geom& G, int y) {
  if (y < 0) return G.yclamp ? 0 : y + G.ny;
  if (y >= G.ny) {
    const int w = y - G.ny;
    return G.yclamp || w >= G.ny ? G.ny - 1 : w;
  }
  return y;
}

// Value of the column to the right / left.  C = 2: lane l holds columns l and l + 32, so the
// right neighbour of lane 31's first column is lane 0's second one (and the reverse); the
// outermost columns of the strip get no neighbour (they are halo).
template <class T>
__device__ __forceinline__ void right(const T (&v)[1], T (&r)[1]) {
  r[0] = __shfl_down_sync(0xffffffffu, v[0], 1);
}
template <class T>
__device__ __forceinline__ void left(const T (&v)[1], T (&r)[1]) {
  r[0] = __shfl_up_sync(0xffffffffu, v[0], 1);
}
template <class T>
__device__ __forceinline__ void right(const T (&v)[2], T (&r)[2]) {
  const int lane = threadIdx.x & 31;
  r[0] = __shfl_sync(0xffffffffu, lane == 0 ? v[1] : v[0], (lane + 1) & 31);
  r[1] = __shfl_down_sync(0xffffffffu, v[1], 1);
}
template <class T>
__device__ __forceinline__ void left(const T (&v)[2], T (&r)[2]) {
  const int lane = threadIdx.x & 31;
  r[0] = __shfl_up_sync(0xffffffffu, v[0], 1);
  r[1] = __shfl_sync(0xffffffffu, lane == 31 ? v[0] : v[1], (lane + 31) & 31);
}
template <class T>
__device__ __forceinline__ T right1(T v) {
  return __shfl_down_sync(0xffffffffu, v, 1);
}
template <class T>
__device__ __forceinline__ T left1(T v) {
  return __shfl_up_sync(0xffffffffu, v, 1);
}

// ------------------------------------------------------------------ operators
// A row operator has M vector components, H halo rows and columns, C columns per lane, and
//   Row   the coefficients of an arriving row (loaded kLag rows behind the vector's row),
//   Emit  the coefficients read where a row is completed,
//   State what it keeps of the rows below,
//   W     warps per block: what the registers of a row allow without spills (a block of 8 has 255
//         a thread, 12 have 168).  Measured: the ideal gas's pressure at 12 and 16 warps, with
//         spills, 11 and 35 % slower on 251 x 173; the B form at 12, 30 % slower on 768^2; the
//         Redlich-Kwong residual, compute bound, 3 % faster at 12 than at 8,
//   R     FP64 vectors of a row that the ring in shared memory holds (Ring; twice as many in FP32),
//   kDots   vectors whose dot products a lane sums in registers over its rows (the others' are added
//         across the warp at every row),
//   kAhead  vectors past the ring whose row is loaded ahead of its use, into registers,
//   step(st, w, in, em, out, wc): takes the arriving row w, completes the row H below it:
//         out = A w there, wc = w there.
// precond applies the solve's Jacobi preconditioner to a completed row (it uses the diagonal
// that step left in em).  All the arithmetic is in T.

// Pressure_Subsystem_AX (implicit_operators.cpp:505-616), global dissipation, and precP
// (implicit_operators.cpp:650-662).  Each face's two products (enthalpy and viscous) are
// formed once and differenced by the two cells that share it: the same operations on the same
// operands as the reference's per-cell form.  kRK: the viscosity's slope factor varies by
// cell (vscale); for the ideal gas it is the constant 1 / (gamma - 1).
struct PressureCoef {
  DevParams P;
  const DevScalars* sc;
  const double *hh, *eta, *vscale, *vdiag;
  double *idg, *kx, *ky;  // planes that the residual pass leaves for the Krylov passes (FaceRow)
  double h, hh2, idx2, idy2, cvx, cvy, a;
  int jac;
  __device__ __forceinline__ void bind() {
    h = sc->h;
    hh2 = h * h;
    idx2 = 1 / (P.dx * P.dx);
    idy2 = 1 / (P.dy * P.dy);
    double nu_x = 0.0, nu_y = 0.0;
    if (P.add_pvisc == IMEX_MaterialSpeedp) {
      nu_x = sc->vx_max * P.dx;
      nu_y = sc->vy_max * P.dy;
    } else if (P.add_pvisc == IMEX_AlfvenSpeedp) {
      nu_x = sc->cA_x * P.dx;
      nu_y = sc->cA_y * P.dy;
    }
    cvx = nu_x / (P.dx * P.dx);
    cvy = nu_y / (P.dy * P.dy);
    a = 1.0 / (P.gamma - 1.0);
  }
};
template <class T_, bool kRK>
struct PressureRow : PressureCoef {
  using T = T_;
  static constexpr int M = 1, H = 1, C = 2, kLag = 0, W = kRK ? 12 : 8, R = kRK ? 9 : 14, kDots = 8, kAhead = 0;
  static constexpr bool kIsRK = kRK;
  static constexpr int kCoef = 2 + (kRK ? 2 : 0);  // planes read per application (+ vdiag in J mode)
  template <class U>
  __device__ __forceinline__ PressureRow<U, kRK> as() const {
    PressureRow<U, kRK> o;
    static_cast<PressureCoef&>(o) = *this;
    return o;
  }
  struct Row {
    T h[C], e[C];
  };
  struct Emit {
    T vs[C], vd[C], id[C];
    T dg[C], kx[C], ky[C];  // from step: precP's diagonal less vd, the weights of the right and upper face
  };
  struct GeneralState {
    T x[C], h[C], e[C], gH[C], fH[C], fE[C];  // the row, and its lower face's mean and products
  };
  struct FaceState {
    T x[C], h[C], hS[C], sx[C], sy[C], f[C];  // the row, h below it, its halves of the face weights, the lower product
  };
  using State = typename std::conditional<kRK, GeneralState, FaceState>::type;
  __device__ __forceinline__ void load(const int (&o)[C], Row& r) const {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      r.h[c] = (T)__ldg(hh + o[c]);
      r.e[c] = (T)__ldg(eta + o[c]);
    }
  }
  __device__ __forceinline__ void load(const int (&o)[C], Emit& e) const {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      e.vd[c] = jac ? (T)vdiag[o[c]] : (T)a;
      e.vs[c] = kRK ? (T)__ldg(vscale + o[c]) : (T)a;
      if (kRK) e.id[c] = (T)idg[o[c]];
    }
  }
  __device__ __forceinline__ void step(State& s, const T (&w)[M][C], const Row& n, Emit& em, T (&out)[M][C],
                                       T (&wc)[M][C]) const {
    if constexpr (kRK) general(s, w, n, em, out, wc);
    else faces(s, w, n, em, out, wc);
  }
  // the ideal gas: the slope factor is the constant a, so the two products of a face are one with
  // the weight hh2 idx2 h + a h cvx e of the face means of h and e, which is the sum of a half from
  // either cell: five exchanges between columns instead of six and half the products
  __device__ __forceinline__ void faces(State& s, const T (&w)[M][C], const Row& n, Emit& em, T (&out)[M][C],
                                        T (&wc)[M][C]) const {
    const T hf = T(0.5), ax = hf * (T)(hh2 * idx2), bx = hf * (T)(a * h * cvx), ay = hf * (T)(hh2 * idy2),
            by = hf * (T)(a * h * cvy);
    T xE[C], hE[C], hW[C], sE[C], r[C], l[C];
    right(s.x, xE);
    right(s.h, hE);
    left(s.h, hW);
    right(s.sx, sE);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      em.kx[c] = s.sx[c] + sE[c];
      r[c] = em.kx[c] * (xE[c] - s.x[c]);
    }
    left(r, l);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const T sy = ay * n.h[c] + by * n.e[c];
      em.ky[c] = s.sy[c] + sy;
      const T u = em.ky[c] * (w[0][c] - s.x[c]);
      out[0][c] = em.vd[c] * s.x[c] - ((r[c] - l[c]) + (u - s.f[c]));
      const T h2 = s.h[c] + s.h[c];
      em.dg[c] = ax * (hE[c] + hW[c] + h2) + ay * (n.h[c] + s.hS[c] + h2);
      wc[0][c] = s.x[c];
      s.x[c] = w[0][c];
      s.hS[c] = s.h[c];
      s.h[c] = n.h[c];
      s.sx[c] = ax * n.h[c] + bx * n.e[c];
      s.sy[c] = sy;
      s.f[c] = u;
    }
  }
  __device__ __forceinline__ void general(State& s, const T (&w)[M][C], const Row& n, Emit& em, T (&out)[M][C],
                                          T (&wc)[M][C]) const {
    const T hf = T(0.5);
    T xE[C], hE[C], eE[C], gR[C], vR[C], rH[C], rE[C], gL[C], lH[C], lE[C];
    right(s.x, xE);
    right(s.h, hE);
    right(s.e, eE);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      gR[c] = hf * (hE[c] + s.h[c]);
      vR[c] = hf * (eE[c] + s.e[c]);
      rH[c] = gR[c] * (xE[c] - s.x[c]);
      rE[c] = vR[c] * (xE[c] - s.x[c]);
    }
    left(gR, gL);
    left(rH, lH);
    left(rE, lE);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const T gU = hf * (n.h[c] + s.h[c]), vU = hf * (n.e[c] + s.e[c]);
      const T uH = gU * (w[0][c] - s.x[c]);
      const T uE = vU * (w[0][c] - s.x[c]);
      const T r = em.vd[c] * s.x[c] - (T)hh2 * ((T)idx2 * (rH[c] - lH[c]) + (T)idy2 * (uH - s.fH[c]));
      const T lap = (T)cvx * (rE[c] - lE[c]) + (T)cvy * (uE - s.fE[c]);
      out[0][c] = r - em.vs[c] * (T)h * lap;
      em.dg[c] = (T)hh2 * ((T)idx2 * (gR[c] + gL[c]) + (T)idy2 * (gU + s.gH[c]));
      wc[0][c] = s.x[c];
      s.x[c] = w[0][c];
      s.h[c] = n.h[c];
      s.e[c] = n.e[c];
      s.gH[c] = gU;
      s.fH[c] = uH;
      s.fE[c] = uE;
    }
  }
  __device__ __forceinline__ void precond(const Emit& em, T (&v)[M][C]) const {
#pragma unroll
    for (int c = 0; c < C; ++c) v[0][c] *= em.id[c];
  }
};

// The symmetric one-component operators in the passes of their conjugate-gradient solves: the
// pressure operator of the ideal gas (its viscosity's slope factor is the constant
// 1 / (gamma - 1), so the enthalpy and viscous weights of a face add up to one) and the energy
// operator.  The residual pass (PressureRow, EnergyRow) leaves the weights of each cell's right
// and upper face and the reciprocal of the preconditioner's diagonal; a pass differences two
// face products per direction.
struct FaceCoef {
  const double *kx, *ky, *idg;
  double a;             // the operator's diagonal apart from the face weights, unless it varies:
  const double* vdiag;  // J mode: V_slope of every cell, or
  const double* p;      // the pressure, in a Newton iterate with floored cells (slope Mbig below p_floor)
  double p_floor, Mbig;
};
template <class T_>
struct FaceRow : FaceCoef {
  using T = T_;
  static constexpr int M = 1, H = 1, C = 2, kLag = 0, W = 8, R = 14, kDots = 8, kAhead = 0;
  static constexpr int kCoef = 3;
  __device__ __forceinline__ T slope(int o) const {
    if (p) return (T)(p[o] >= p_floor ? a : Mbig);
    return vdiag ? (T)vdiag[o] : (T)a;
  }
  // the passes of GMRES, which takes over where conjugate gradients break down
  struct Row {
    T kx[C], ky[C];
  };
  struct Emit {
    T vd[C], id[C];
  };
  struct State {
    T x[C], kx[C], ky[C], f[C];  // the row, its weights, the product of its lower face
  };
  __device__ __forceinline__ void load(const int (&o)[C], Row& r) const {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      r.kx[c] = (T)kx[o[c]];
      r.ky[c] = (T)ky[o[c]];
    }
  }
  __device__ __forceinline__ void load(const int (&o)[C], Emit& e) const {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      e.vd[c] = slope(o[c]);
      e.id[c] = (T)idg[o[c]];
    }
  }
  // the row s is completed by the row w above it
  __device__ __forceinline__ void complete(State& s, const T (&w)[C], const Row& n, const T (&vd)[C], T (&out)[C]) const {
    T xE[C], r[C], l[C];
    right(s.x, xE);
#pragma unroll
    for (int c = 0; c < C; ++c) r[c] = s.kx[c] * (xE[c] - s.x[c]);
    left(r, l);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const T u = s.ky[c] * (w[c] - s.x[c]);
      out[c] = vd[c] * s.x[c] - ((r[c] - l[c]) + (u - s.f[c]));
      s.x[c] = w[c];
      s.kx[c] = n.kx[c];
      s.ky[c] = n.ky[c];
      s.f[c] = u;
    }
  }
  __device__ __forceinline__ void step(State& s, const T (&w)[M][C], const Row& n, Emit& em, T (&out)[M][C],
                                       T (&wc)[M][C]) const {
#pragma unroll
    for (int c = 0; c < C; ++c) wc[0][c] = s.x[c];
    complete(s, w[0], n, em.vd, out[0]);
  }
  __device__ __forceinline__ void precond(const Emit& em, T (&v)[M][C]) const {
#pragma unroll
    for (int c = 0; c < C; ++c) v[0][c] *= em.id[c];
  }
};

// Energy_Subsystem_AX (implicit_operators.cpp:741-795) and precE (imex_subsystems.cpp:487-505).
struct EnergyCoef {
  DevParams P;
  const DevScalars* sc;
  const double* hh;
  double *idg, *kx, *ky;
  double gh2, idx2, idy2, dxdy;
  __device__ __forceinline__ void bind() {
    const double h = sc->h;
    gh2 = (P.gamma - 1) * h * h;
    idx2 = 1.0 / (P.dx * P.dx);
    idy2 = 1.0 / (P.dy * P.dy);
    dxdy = P.dx * P.dy;
  }
};
template <class T_>
struct EnergyRow : EnergyCoef {
  using T = T_;
  static constexpr int M = 1, H = 1, C = 2, kLag = 0, W = 8, R = 14, kDots = 8, kAhead = 0;
  static constexpr bool kIsRK = false;
  static constexpr int kCoef = 1;
  template <class U>
  __device__ __forceinline__ EnergyRow<U> as() const {
    EnergyRow<U> o;
    static_cast<EnergyCoef&>(o) = *this;
    return o;
  }
  struct Row {
    T h[C];
  };
  struct Emit {
    T vd[C], dg[C], kx[C], ky[C];  // as PressureRow's
  };
  struct State {
    T x[C], h[C], gH[C], fH[C];
  };
  __device__ __forceinline__ void load(const int (&o)[C], Row& r) const {
#pragma unroll
    for (int c = 0; c < C; ++c) r.h[c] = (T)__ldg(hh + o[c]);
  }
  __device__ __forceinline__ void load(const int (&)[C], Emit&) const {}
  __device__ __forceinline__ void step(State& s, const T (&w)[M][C], const Row& n, Emit& em, T (&out)[M][C],
                                       T (&wc)[M][C]) const {
    const T hf = T(0.5);
    T xE[C], hE[C], gR[C], rH[C], gL[C], lH[C];
    right(s.x, xE);
    right(s.h, hE);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      gR[c] = hf * (hE[c] + s.h[c]);
      rH[c] = gR[c] * (xE[c] - s.x[c]);
    }
    left(gR, gL);
    left(rH, lH);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const T gU = hf * (n.h[c] + s.h[c]);
      const T uH = gU * (w[0][c] - s.x[c]);
      out[0][c] = (s.x[c] - (T)gh2 * ((T)idx2 * (rH[c] - lH[c]) + (T)idy2 * (uH - s.fH[c]))) * (T)dxdy;
      em.vd[c] = (T)dxdy;
      em.dg[c] = (T)(gh2 * dxdy) * ((T)idx2 * (gR[c] + gL[c]) + (T)idy2 * (gU + s.gH[c]));
      em.kx[c] = (T)(gh2 * dxdy * idx2) * gR[c];
      em.ky[c] = (T)(gh2 * dxdy * idy2) * gU;
      wc[0][c] = s.x[c];
      s.x[c] = w[0][c];
      s.h[c] = n.h[c];
      s.gH[c] = gU;
      s.fH[c] = uH;
    }
  }
};

// Magnetic_Subsystem_AX (implicit_operators.cpp:141-353), global dissipation, fast arithmetic.
// The reference's four bracketed terms per component are the two sides of face fluxes: the
// terms of the lower (left) face of a cell are those of the upper (right) face of the cell
// below (to the left).  Each face flux and each corner average is formed once here, with one
// division per face instead of sixteen per cell.
struct MagBCoef {
  DevParams P;
  const DevScalars* sc;
  const double *Qe, *rho;
  double h, cx, cy;
  __device__ __forceinline__ void bind() {
    h = sc->h;
    cx = sc->B_max_x * P.dx / (P.dx * P.dx);
    cy = sc->B_max_y * P.dy / (P.dy * P.dy);
  }
};
// W_, R_, A_: warps per block, vectors in the ring, vectors past it loaded ahead.
template <class T_, int W_ = 8, int R_ = 8, int A_ = 5>
struct MagBRow : MagBCoef {
  using T = T_;
  static constexpr int M = 3, H = 1, C = 1, kLag = 0, W = W_, R = R_, kDots = 8, kAhead = A_;
  static constexpr int kCoef = 4;
  template <class U>
  __device__ __forceinline__ MagBRow<U, W_, R_, A_> as() const {
    MagBRow<U, W_, R_, A_> o;
    static_cast<MagBCoef&>(o) = *this;
    return o;
  }
  struct Row {
    T q[3], r;
  };
  struct Emit {};
  struct State {
    T x[3], q[3], r;         // the row: vector, Qe B, rho
    T sq[3], sx[3];          // q + q(E), x + x(E)
    T a[3];                  // (q.x)/2 - q6 x6, q6 x5, q6 x7
    T db[3], k[3];           // right face: differences of (q.x)/2 - q5 x5, q5 x6, q5 x7; mean Qe B / rho
    T lx[3], dy[3];          // x part of the Laplacian; x - x(S)
    T c1, c4, c5, c6;        // lower corner products
    T gx, gz;                // lower face fluxes
  };
  __device__ __forceinline__ void load(const int (&o)[C], Row& r) const {
#pragma unroll
    for (int m = 0; m < 3; ++m) r.q[m] = (T)__ldg(Qe + (5 + m) * P.N + o[0]);
    r.r = (T)__ldg(rho + o[0]);
  }
  __device__ __forceinline__ void load(const int (&)[C], Emit&) const {}
  __device__ __forceinline__ void step(State& s, const T (&w)[M][C], const Row& n, Emit&, T (&out)[M][C],
                                       T (&wc)[M][C]) const {
    const T hf = T(0.5), qf = T(0.25), one = T(1);
    const T idx = (T)P.rdx, idy = (T)P.rdy, hT = (T)h, cxT = (T)cx, cyT = (T)cy;
    // the arriving row: sums with its right neighbours, corner averages of the upper corner
    T sq[3], sx[3], dx[3], cq[3], cv[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const T qE = right1(n.q[m]), xE = right1(w[m][0]);
      sq[m] = n.q[m] + qE;
      sx[m] = w[m][0] + xE;
      dx[m] = xE - w[m][0];
      cq[m] = qf * (s.sq[m] + sq[m]);
      cv[m] = qf * (s.sx[m] + sx[m]);
    }
    const T W = hf * (cq[0] * cv[0] + cq[1] * cv[1] + cq[2] * cv[2]);
    const T c1 = cq[0] * cv[1], c2 = W - cq[0] * cv[0], c3 = cq[0] * cv[2];
    const T c4 = W - cq[1] * cv[1], c5 = cq[1] * cv[0], c6 = cq[1] * cv[2];
    const T p0 = n.q[0] * w[0][0], p1 = n.q[1] * w[1][0], p2 = n.q[2] * w[2][0];
    const T hs = hf * (p0 + p1 + p2);
    const T a0 = hs - p1, a1 = n.q[1] * w[0][0], a2 = n.q[1] * w[2][0];
    // the upper face of the completed row
    const T iv = one / (s.r + n.r);
    const T br = idx * (c1 - left1(c1)) - idy * (a0 - s.a[0]);
    const T f6 = (s.q[1] + n.q[1]) * iv;
    const T gx = (s.q[0] + n.q[0]) * iv * br + f6 * (idx * (c2 - left1(c2)) - idy * (a1 - s.a[1]));
    const T gz = (s.q[2] + n.q[2]) * iv * br - f6 * (idx * (c3 - left1(c3)) + idy * (a2 - s.a[2]));
    // its right face
    const T bf = idy * (c1 - s.c1) - idx * s.db[0];
    const T fy = s.k[1] * bf + s.k[0] * (idy * (c4 - s.c4) - idx * s.db[1]);
    const T fz = s.k[2] * (idy * (c5 - s.c5) - idx * s.db[0]) - s.k[0] * (idx * s.db[2] + idy * (c6 - s.c6));
    const T h2x = hT * hT * idx, h2y = hT * hT * idy;
    const T dfy = fy - left1(fy), dfz = fz - left1(fz);
    T dy[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      dy[m] = w[m][0] - s.x[m];
      const T lap = cxT * s.lx[m] + cyT * (dy[m] - s.dy[m]);
      const T f = m == 0 ? h2y * (gx - s.gx) : (m == 1 ? h2x * dfy : h2x * dfz + h2y * (gz - s.gz));
      out[m][0] = s.x[m] + f - hT * lap;
      wc[m][0] = s.x[m];
    }
    // the arriving row becomes the current one
    const T ivx = one / (n.r + right1(n.r));
    const T b0 = hs - p0, b1 = n.q[0] * w[1][0], b2 = n.q[0] * w[2][0];
    s.db[0] = right1(b0) - b0;
    s.db[1] = right1(b1) - b1;
    s.db[2] = right1(b2) - b2;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      s.x[m] = w[m][0];
      s.q[m] = n.q[m];
      s.sq[m] = sq[m];
      s.sx[m] = sx[m];
      s.k[m] = sq[m] * ivx;
      s.lx[m] = dx[m] - left1(dx[m]);
      s.dy[m] = dy[m];
    }
    s.r = n.r;
    s.a[0] = a0;
    s.a[1] = a1;
    s.a[2] = a2;
    s.c1 = c1;
    s.c4 = c4;
    s.c5 = c5;
    s.c6 = c6;
    s.gx = gx;
    s.gz = gz;
  }
  __device__ __forceinline__ void precond(const Emit&, T (&)[M][C]) const {}
};

// Magnetic_Subsystem_potential_AX (implicit_operators.cpp:355-503), global dissipation, fast
// arithmetic, periodic.  Row n arrives; curl A and the stress tensor T^B are formed on row
// n - 1 and the Lorentz term on row n - 2.
struct MagACoef {
  DevParams P;
  const DevScalars* sc;
  const double *Qe, *irho;
  double h, cx, cy;
  __device__ __forceinline__ void bind() {
    h = sc->h;
    cx = P.add_bvisc ? sc->gmax_bx * P.dx / (P.dx * P.dx) : 0.0;
    cy = P.add_bvisc ? sc->gmax_by * P.dy / (P.dy * P.dy) : 0.0;
  }
};
template <class T_>
struct MagARow : MagACoef {
  using T = T_;
  static constexpr int M = 3, H = 2, C = 1, kLag = 1, W = 12, R = 4, kDots = 8, kAhead = 0;
  static constexpr int kCoef = 4;
  template <class U>
  __device__ __forceinline__ MagARow<U> as() const {
    MagARow<U> o;
    static_cast<MagACoef&>(o) = *this;
    return o;
  }
  struct Row {
    T q[3];
  };
  struct Emit {
    T ir;
  };
  struct State {
    T a1[3], a2[3], a3[3];  // A on rows n - 1, n - 2, n - 3
    T by, d1;               // row n - 1: -dA2/dx, dA1/dx
    T l1[3], l2[3];         // x part of the Laplacian on rows n - 1, n - 2
    T q[3];                 // Qe B on row n - 2
    T tx[3], ty2[3], ty3[3];  // row n - 2: x difference of T; rows n - 2, n - 3: T in y
  };
  __device__ __forceinline__ void load(const int (&o)[C], Row& r) const {
#pragma unroll
    for (int m = 0; m < 3; ++m) r.q[m] = (T)__ldg(Qe + (5 + m) * P.N + o[0]);
  }
  __device__ __forceinline__ void load(const int (&o)[C], Emit& e) const { e.ir = (T)__ldg(irho + o[0]); }
  __device__ __forceinline__ void step(State& s, const T (&w)[M][C], const Row& n, Emit& em, T (&out)[M][C],
                                       T (&wc)[M][C]) const {
    const T hf = T(0.5), hT = (T)h;
    const T rx = hf * (T)P.rdx, ry = hf * (T)P.rdy;
    // row n - 1: B = curl A, T^B
    const T bx = ry * (w[2][0] - s.a2[2]);
    const T by = s.by;
    const T bz = s.d1 - ry * (w[0][0] - s.a2[0]);
    const T Bx = n.q[0], By = n.q[1], Bz = n.q[2];
    const T bh = hf * (Bx * bx + By * by + Bz * bz);
    const T txx = bh - Bx * bx, tyx = -Bx * by, tzx = -Bx * bz;
    const T ty[3] = {-By * bx, bh - By * by, -By * bz};
    const T tx[3] = {rx * (right1(txx) - left1(txx)), rx * (right1(tyx) - left1(tyx)), rx * (right1(tzx) - left1(tzx))};
    // row n - 2: F = h / rho div T, F x B, the Laplacian
    const T hr = hT * em.ir;
    const T Fx = hr * (s.tx[0] + ry * (ty[0] - s.ty3[0]));
    const T Fy = hr * (s.tx[1] + ry * (ty[1] - s.ty3[1]));
    const T Fz = hr * (s.tx[2] + ry * (ty[2] - s.ty3[2]));
    const T cr[3] = {s.q[1] * Fz - s.q[2] * Fy, s.q[2] * Fx - s.q[0] * Fz, s.q[0] * Fy - s.q[1] * Fx};
    T dW[3];  // A(E), A(W) of the arriving row
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const T lap = (T)cx * s.l2[m] + (T)cy * (s.a1[m] - 2 * s.a2[m] + s.a3[m]);
      out[m][0] = s.a2[m] - hT * cr[m] - hT * lap;
      wc[m][0] = s.a2[m];
      const T e = right1(w[m][0]), v = left1(w[m][0]);
      dW[m] = e - v;
      s.l2[m] = s.l1[m];
      s.l1[m] = e - 2 * w[m][0] + v;
      s.a3[m] = s.a2[m];
      s.a2[m] = s.a1[m];
      s.a1[m] = w[m][0];
      s.q[m] = n.q[m];
      s.ty3[m] = s.ty2[m];
      s.ty2[m] = ty[m];
      s.tx[m] = tx[m];
    }
    s.by = -rx * dW[2];
    s.d1 = rx * dW[1];
  }
  __device__ __forceinline__ void precond(const Emit&, T (&)[M][C]) const {}
};

// ------------------------------------------------------------------ the march
// One task.  fill.issue(it, off, eo, buf) starts the loads of the arriving row (plane offsets
// off; eo: of the row it completes), fill.finish(it, off, buf, w) forms the row from them; the
// next row's loads (and fill.ahead(eo), those of the row about to be completed) are issued before
// the current row's arithmetic.  emit(it, eo, own, wc, out,
// em, buf) receives each completed row in order.
template <class Op, class Fill, class EmitF>
__device__ __forceinline__ void run_task(const Op& op, const Geom& G, int task, Fill& fill, EmitF& emit) {
  constexpr int C = Op::C, M = Op::M, H = Op::H;
  using T = typename Op::T;
  const int strip = task / G.nseg, seg = task - strip * G.nseg, lane = threadIdx.x & 31;
  int xo[C];
  bool own[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int k = lane + 32 * c, x = strip * G.wd + k - H;
    own[c] = k >= H && k < H + G.wd && x < G.nx;
    xo[c] = map_x(G, x);
  }
  const int y0 = seg * G.L, y1 = y0 + G.L < G.ny ? y0 + G.L : G.ny;
  const int nit = y1 - y0 + 2 * H;
  typename Op::State st{};
  typename Op::Row in;
  typename Op::Emit em;
  typename Fill::Buf buf;
  int off[C], eo[C];
  auto issue = [&](int it) {
    const int y = y0 - H + it;
    const int r = map_y(G, y) * G.nx;
    int e = y - H;  // the row this one completes
    e = e < y0 ? y0 : e;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      off[c] = r + xo[c];
      eo[c] = e * G.nx + xo[c];
    }
    if (Op::kLag == 0) {
      op.load(off, in);
    } else {
      const int rl = map_y(G, y - Op::kLag < -H ? -H : y - Op::kLag) * G.nx;
      int ol[C];
#pragma unroll
      for (int c = 0; c < C; ++c) ol[c] = rl + xo[c];
      op.load(ol, in);
    }
    op.load(eo, em);
    fill.issue(it, off, eo, buf);
  };
  issue(0);
#pragma unroll 1
  for (int it = 0; it < nit; ++it) {
    T w[M][C], out[M][C], wc[M][C];
    fill.finish(it, off, buf, w);
    const typename Op::Row inc = in;
    typename Op::Emit emc = em;
    const typename Fill::Buf bufc = buf;
    int eoc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) eoc[c] = eo[c];
    fill.ahead(eoc);
    if (it + 1 < nit) issue(it + 1);
    op.step(st, w, inc, emc, out, wc);
    if (it >= 2 * H) emit(it, eoc, own, wc, out, emc, bufc);
  }
}

// ------------------------------------------------------------------ sums
// four lane values -> their four warp sums; lane 8 q holds the sum of x[q]
__device__ __forceinline__ double warp_sum4(double (&x)[4]) {
  const int lane = threadIdx.x & 31;
  const bool b4 = lane & 16, b3 = lane & 8;
  double y0 = b4 ? x[2] : x[0], y1 = b4 ? x[3] : x[1];
  y0 += __shfl_xor_sync(0xffffffffu, b4 ? x[0] : x[2], 16);
  y1 += __shfl_xor_sync(0xffffffffu, b4 ? x[1] : x[3], 16);
  double z = b3 ? y1 : y0;
  z += __shfl_xor_sync(0xffffffffu, b3 ? y0 : y1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
  return z;
}
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ double warp_min(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmin(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// ------------------------------------------------------------------ the device-wide pass end
// Every block publishes its partial sums and then adds one to an arrival counter (a release);
// one thread of each block polls the counter (an acquire) until all have arrived, and every
// block sums all partials itself in one fixed order, so all blocks hold identical values.
// Measured at 148 blocks with the sums of three slots: 4.7 thousand cycles a pass end; an
// array of per-block flags that every block reads takes 11 thousand (148 readers of the same
// lines hold up the writers), relaxed polls closed by a fence 5.3, cluster leaders with the sums
// in distributed shared memory 5.0 to 5.3.  The wait is bounded: after `limit` SM cycles the
// block gives the launch up, by a compare-and-swap that sets the counter's top bit only while the
// target is not reached.  The word that counts the arrivals thus also decides: either every block
// passes this end, or every block leaves here or at a later end, and none takes a launch that
// others gave up for a whole one.  The bit stays until the host starts the counters again, and
// launches before that end at their first wait.  The counter grows from launch to launch
// (SyncState::epoch is its value at the start), so no reset precedes a launch; the first block
// stores the next epoch when it leaves, which no block reads before the next launch.
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void arrive(unsigned long long* p) {
  asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(p) : "memory");
}
constexpr unsigned long long kGaveUp = 1ull << 63;
// gives the launch up unless the target has been reached in the meantime; the counter as decided (called:
// inlined it costs the B-form solve 16 bytes of spills, and its steps half a percent)
static __device__ __noinline__ unsigned long long give_up(unsigned long long* p, unsigned long long target) {
  unsigned long long v = ld_relaxed(p);
  while (v < target) {
    const unsigned long long was = atomicCAS(p, v, v | kGaveUp);
    if (was == v) return v | kGaveUp;
    v = was;
  }
  return ld_acquire(p);
}

struct Shared {
  double H[kCap + 2][kCap + 2];                // rotated Hessenberg columns
  double hcol[kCap + 2], coef[kCap + 2];       // the current raw column; an update's weights
  double comb[kCap + 3];                       // weights of the terms of the next vector
  double cs[kCap + 2], sn[kCap + 2], gam[kCap + 2], sigma[kCap + 2];
  double red[kSlots];
  double acc[kMaxWarps][kSlots];
  double cga[kCap + 2], cgb[kCap + 2];         // conjugate gradients: alpha_k, beta_k
  int nalpha;  // terms of an update that the caller's next pass applies
  int cycles;  // of this solve, counted by its first block
  double bytes;
};

struct Sync {
  SyncState* s;
  unsigned long long base, seq;  // arrivals before this launch; pass ends of this launch
  long long limit;
  int nblk, rank;
  double* partial;  // 2 x nblk x kSlots
};
__device__ __forceinline__ void acc_clear(Shared& S) {
  const int lane = threadIdx.x & 31;
  if (lane < kSlots) S.acc[threadIdx.x >> 5][lane] = 0.0;
  __syncwarp();
}
// S.red[0, kn) = the sums (minima for the slots of `mins`) of S.acc over all warps of all
// blocks; false when the wait ran out
template <int W>
__device__ __forceinline__ bool pass_end(Sync& y, Shared& S, int kn, unsigned mins = 0u) {
  constexpr int kNT = 32 * W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* part = y.partial + (long long)(y.seq & 1) * y.nblk * kSlots;
  const unsigned long long target = y.base + ++y.seq * (unsigned long long)y.nblk;
  __syncthreads();
  if (warp == 0) {
    if (lane < kn) {
      const bool mn = lane < 32 && ((mins >> lane) & 1u);
      double v = S.acc[0][lane];
#pragma unroll
      for (int q = 1; q < W; ++q) v = mn ? fmin(v, S.acc[q][lane]) : v + S.acc[q][lane];
      __stcg(part + (long long)y.rank * kSlots + lane, v);
    }
    __syncwarp();
    if (lane == 0) arrive(&y.s->arrivals);
  }
  int ok = 1;
  if (tid == 0) {
    unsigned long long v = ld_acquire(&y.s->arrivals);
    if (v < target) {
      const long long t0 = clock64();
      do {
        v = clock64() - t0 > y.limit ? give_up(&y.s->arrivals, target) : ld_acquire(&y.s->arrivals);
      } while (v < target);
    }
    ok = (v & kGaveUp) == 0;
  }
  ok = __syncthreads_and(ok);
  if (!ok) return false;
  // slot k of every block, summed by the threads with the same k in block order, then across
  // the lanes and warps: KS threads side by side read a block's slots
  const int KS = kn <= 4 ? 4 : (kn <= 8 ? 8 : (kn <= 16 ? 16 : 32));
  const int k = tid & (KS - 1), g0 = tid / KS, ng = kNT / KS;
  const bool mn = (mins >> k) & 1u;
  double v = mn ? INFINITY : 0.0;
  if (k < kn) {
    constexpr int U = 5;
    for (int b0 = g0; b0 < y.nblk; b0 += U * ng) {
      double t[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int b = b0 + u * ng;
        t[u] = b < y.nblk ? __ldcg(part + (long long)b * kSlots + k) : (mn ? INFINITY : 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) v = mn ? fmin(v, t[u]) : v + t[u];
    }
  }
  for (int o = 16; o >= KS; o >>= 1) {
    const double t = __shfl_xor_sync(0xffffffffu, v, o);
    v = mn ? fmin(v, t) : v + t;
  }
  if (lane < KS && lane < kn) S.acc[warp][lane] = v;
  __syncthreads();
  if (tid < kn) {
    const bool m2 = (mins >> tid) & 1u;
    double r = S.acc[0][tid];
#pragma unroll
    for (int q = 1; q < W; ++q) r = m2 ? fmin(r, S.acc[q][tid]) : r + S.acc[q][tid];
    S.red[tid] = r;
  }
  __syncthreads();
  return true;
}

}  // namespace march
}  // namespace imex
