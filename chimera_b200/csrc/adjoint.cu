// adjoint.cu -- hand-written discrete adjoint of one SSP-RK3 step (FP64).
//
// For a state U_n and the adjoint lambda_{n+1} = dL/dU_{n+1}, computes
// lambda_n = (dU_{n+1}/dU_n)^T lambda_{n+1} with the time step held at its
// forward value (the CFL dt is not differentiated: "frozen dt").
//
// Structure.  The step is re-run forward by the fused FP64 stage kernels with the
// tape (TapeOut): each stage leaves its primitives, a byte per cell that says
// which floors changed the cell, and at those cells the values that went into
// them.  The reverse sweep then transposes, stage 3 to 1, two kernels a stage:
//   k_rev_faces  one thread a face: the adjoint of its five fluxes from the cells
//                and corners around it --
//                  floors + RK blend      (src/mhd_change_states.f90:116-166, src/main.f90:202-267)
//                  flux divergence        (src/mhd_flux.f90:20-76)
//                  constrained transport  (src/mhd_flux.f90:79-136): lambda_Ez at the corners
//                -- the face states again from the primitives, with the forward's
//                decisions, and the solver's vector-Jacobian product (face_vjp.cuh):
//                  Riemann solver         (src/mhd_flux.f90:197-779)
//                  thermal check, face floors, MOOD  (src/mhd_derivatives.f90:130-293): a
//                                         reset face passes its adjoint to the cell it was reset to
//   k_rev_cells  one thread a cell: gathers its faces' adjoints through
//                  slope limiter          (src/mhd_derivatives.f90:50-127); where a one-sided
//                                         difference is exactly zero (uniform neighbourhood) the
//                                         limiter is not differentiable: (1/2, 1/2) if both are
//                                         zero, else 1 w.r.t. the zero one (slope_vjp)
//                  primitive recovery     (src/mhd_change_states.f90:61-113)
//                  face->cell B average   (src/mhd_field_ops.f90:120-156)
// as gathers (no atomics; deterministic).  At a kink (limiter branch, min / max,
// floor) the derivative is that of the branch the forward took; the rarely taken
// floors and the outflow correction are differentiated with forward-mode dual
// numbers (dual.cuh) through the same device functions.
//
// This unit is compiled without multiply-add contraction: the face states repeat
// the forward's bits and decisions.
//
// Boundary conditions: periodic or outflow (zero-gradient ghost cells), each
// side on its own -- a periodic side may face an outflow one, whose faces and
// ghosts then follow the rules of the side they lie beyond.  At an outflow side the forward
// takes the nearest cell for every ghost position (src/mhd_bc.f90:36-121), the
// outflow face->cell B (src/mhd_field_ops.f90:120-156), curl copy
// (src/mhd_flux.f90:79-136), update without the incoming face
// (src/mhd_flux.f90:20-76) and boundary flux correction (src/main.f90:118-148);
// the reverse gathers transpose each of them.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <new>

#include "../../include/chimera_gpu.h"
#include "abi_check.h"
#include "chimera_types.h"
#include "dual.cuh"
#include "face_vjp.cuh"
#include "grid_dep.cuh"
#include "kernel_table.h"
#include "mhd_device.cuh"

using namespace chimera;

namespace {

struct AdjGeom {
  int nx, ny;
  double dx, dy, inv_dx, inv_dy, inv_2dx, inv_2dy, hx, hy, gamma, vol;
  int riemann, limiter, slope, mood;
  double igm1, ivol;   // 1 / (gamma - 1), 1 / vol
  int px, py;     // the low side (x = 0 / y = 0) is periodic (else outflow)
  int pxh, pyh;   // the high side is periodic (differs from the low side in a mixed pair)
};

__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
// the cell a ghost position i (one or two cells beyond the grid) takes its
// value from, by the rule of the side it lies beyond (plo below 0, phi at n
// and above): periodic wrap, or the nearest cell (outflow)
__device__ __forceinline__ int src(int i, int n, int plo, int phi) {
  if (i >= 0 && i < n) return i;
  return (i < 0 ? plo : phi) ? wrap(i, n) : (i < 0 ? 0 : n - 1);
}

// One stage of the reverse sweep: what its two kernels read and write.
struct RevStage {
  AdjGeom g;
  int stage;
  double dt, c0, c1;               // RK blend weights of U^n and of the stage's update (0, 1 in stage 1)
  const double* U[6];              // the stage's input
  const double* lout[6];           // adjoint of the stage's output
  TapeOut tape;
  // per face (direction d: 0 x, 1 y; slot = the low cell) and field: the adjoints of
  // the left and the right state that go on through the slopes, and, where the
  // face's flag is set, what resets hand to the low cell's value directly
  double* fL[2][6];
  double* fR[2][6];
  double* fX[2][6];
  unsigned char* fflag[2];
  double* lin[6];                  // adjoint of the stage's input
  double* lU0[6];                  // adjoint of U^n through the blends: set in stage 3, added to in stage 2,
                                   // added to lin in stage 1
};

// neighbour indices for the face with low cell (i, j) in direction ydir
struct FaceIdx {
  int a, b, am, bp, axp, axm, ayp, aym;
  int to;       // the cell above the face, whose update takes the face's flux if b_in
  bool b_in;    // the flux enters that cell (not past an outflow high side, nor into an
                // outflow low side's first cell through a wrap)
  bool b_own;   // mixed pair, outflow low / periodic high side: the high cell is cell 0
                // through the wrap, and its slope's low neighbour is its own ghost
};
__device__ __forceinline__ FaceIdx face_idx(const AdjGeom& g, int i, int j, bool ydir) {
  FaceIdx f;
  const int nx = g.nx, ny = g.ny;
  f.a = j * nx + i;
  if (!ydir) {
    f.b = j * nx + src(i + 1, nx, g.px, g.pxh);
    f.am = j * nx + src(i - 1, nx, g.px, g.pxh);
    f.bp = j * nx + src(i + 2, nx, g.px, g.pxh);
    f.to = j * nx + wrap(i + 1, nx);
    f.b_in = i + 1 < nx || g.px;
    f.b_own = !g.px && g.pxh && i == nx - 1;
  } else {
    f.b = src(j + 1, ny, g.py, g.pyh) * nx + i;
    f.am = src(j - 1, ny, g.py, g.pyh) * nx + i;
    f.bp = src(j + 2, ny, g.py, g.pyh) * nx + i;
    f.to = wrap(j + 1, ny) * nx + i;
    f.b_in = j + 1 < ny || g.py;
    f.b_own = !g.py && g.pyh && j == ny - 1;
  }
  f.axp = j * nx + src(i + 1, nx, g.px, g.pxh);
  f.axm = j * nx + src(i - 1, nx, g.px, g.pxh);
  f.ayp = src(j + 1, ny, g.py, g.pyh) * nx + i;
  f.aym = src(j - 1, ny, g.py, g.pyh) * nx + i;
  return f;
}

// Outflow boundary flux correction (src/main.f90:118-148): a cell on an
// outflow low side gets dt*dx times the physical flux of its own stage
// primitives, in x (sx) and / or in y (sy).  Same operations as the fused
// stage kernel's, here on dual numbers.
template <typename R>
__device__ __forceinline__ void outflow_correction(bool sx, bool sy, R ax, R ay, R gamma, R cr, R cu, R cv, R cP,
                                                   R cBx, R cBy, R* U) {
  if (sx) {
    const R hb = R(0.5) * (cBx * cBx + cBy * cBy);
    const R en = ((cP - hb) / (gamma - R(1)) + R(0.5) * cr * (cu * cu + cv * cv)) + hb;
    U[0] = U[0] + ax * cr * cu;
    U[1] = U[1] + ax * ((cr * (cu * cu) + cP) - cBx * cBx);
    U[2] = U[2] + ax * (cr * cu * cv - cBx * cBy);
    U[3] = U[3] + ax * ((en + cP) * cu - cBx * (cBx * cu + cBy * cv));
  }
  if (sy) {
    const R hb = R(0.5) * (cBx * cBx + cBy * cBy);
    const R en = ((cP - hb) / (gamma - R(1)) + R(0.5) * cr * (cu * cu + cv * cv)) + hb;
    U[0] = U[0] + ay * cr * cv;
    U[2] = U[2] + ay * ((cr * (cv * cv) + cP) - cBy * cBy);
    U[1] = U[1] + ay * (cr * cv * cu - cBy * cBx);
    U[3] = U[3] + ay * ((en + cP) * cv - cBy * (cBy * cv + cBx * cu));
  }
}

// floors Jacobian-transpose product at inputs (M, Mx, My, E) with cell B
__device__ __forceinline__ void floors_vjp(const AdjGeom& g, const double* Uin4, double Bx, double By,
                                           const double* lam4, double* out4, double* lB) {
  using D = Dual<6>;
  D M = seed<6>(Uin4[0], 0), Mx = seed<6>(Uin4[1], 1), My = seed<6>(Uin4[2], 2), E = seed<6>(Uin4[3], 3);
  D bx = seed<6>(Bx, 4), by = seed<6>(By, 5);
  conserved_floors<D>(M, Mx, My, E, bx, by, D(g.gamma), D(g.vol));
  const D* o[4] = {&M, &Mx, &My, &E};
  for (int k = 0; k < 6; ++k) {
    double s = 0.0;
    for (int q = 0; q < 4; ++q) s += lam4[q] * o[q]->d[k];
    if (k < 4) out4[k] = s;
    else lB[k - 4] += s;
  }
}

// The adjoints at one cell whose floors changed it, or that carries the outflow
// correction: lup (of the updated, pre-floor values), lbl (of the blend, before its
// weights), lB (of the stage's cell B through the floors), lcor (of the stage's
// primitives through the correction).  Rare: kept out of line.
__device__ __noinline__ void cell_adjoint_slow(const RevStage& a, int c, double* lup, double* lbl, double* lB,
                                               double* lcor) {
  const unsigned hit = a.tape.hit[c];
  const double Bx = a.tape.P[4][c], By = a.tape.P[5][c];
  double l[4];
  lB[0] = lB[1] = 0.0;
  for (int q = 0; q < 4; ++q) l[q] = a.lout[q][c];
  if (hit & 2u) {
    const double ub[4] = {a.tape.Ublend[0][c], a.tape.Ublend[1][c], a.tape.Ublend[2][c], a.tape.Ublend[3][c]};
    floors_vjp(a.g, ub, Bx, By, l, lbl, lB);
  } else {
    for (int q = 0; q < 4; ++q) lbl[q] = l[q];
  }
  for (int q = 0; q < 4; ++q) l[q] = a.c1 * lbl[q];
  const int i = c % a.g.nx, j = c / a.g.nx;
  const bool sx = !a.g.px && i == 0, sy = !a.g.py && j == 0;
  for (int k = 0; k < 6; ++k) lcor[k] = 0.0;
  if (sx || sy) {   // added after the first floors: l is its adjoint too
    using D = Dual<6>;
    const double ax = a.dt * a.g.dy, ay = a.dt * a.g.dx;
    D pv[6];
    for (int k = 0; k < 6; ++k) pv[k] = seed<6>(a.tape.P[k][c], k);
    D U[4] = {D(0.0), D(0.0), D(0.0), D(0.0)};
    outflow_correction<D>(sx, sy, D(ax), D(ay), D(a.g.gamma), pv[0], pv[1], pv[2], pv[3], pv[4], pv[5], U);
    for (int k = 0; k < 6; ++k)
      for (int q = 0; q < 4; ++q) lcor[k] += l[q] * U[q].d[k];
  }
  if (hit & 1u) {
    const double up[4] = {a.tape.Upre[0][c], a.tape.Upre[1][c], a.tape.Upre[2][c], a.tape.Upre[3][c]};
    floors_vjp(a.g, up, Bx, By, l, lup, lB);
  } else {
    for (int q = 0; q < 4; ++q) lup[q] = l[q];
  }
}

// The adjoint of a cell's updated, pre-floor conserved values.
__device__ __forceinline__ void update_adjoint(const RevStage& a, int c, double* lup) {
  if (a.tape.hit[c]) {
    double lbl[4], lB[2], lcor[6], l[4];
    cell_adjoint_slow(a, c, l, lbl, lB, lcor);
#pragma unroll
    for (int q = 0; q < 4; ++q) lup[q] = l[q];
    return;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) lup[q] = a.c1 * a.lout[q][c];
}

// lambda_Ez at corner (i+1/2, j+1/2): b_x(i,j) gets -dt/dy Ez(i,j), b_x(i,j+1)
// gets +dt/dy Ez(i,j); b_y(i,j) gets +dt/dx Ez(i,j), b_y(i+1,j) gets -dt/dx.
// At an outflow low side b_x(i,0) takes row 1's difference, dt/dy (Ez(i,0) -
// Ez(i,1)), and b_y(0,j) column 1's, dt/dx (Ez(1,j) - Ez(0,j)); past an
// outflow high side there is no b_x(i,ny) / b_y(nx,j).
__device__ __forceinline__ double corner_adjoint(const RevStage& a, int i, int j) {
  const AdjGeom& g = a.g;
  const double* lx = a.lout[4];
  const double* ly = a.lout[5];
  const int c = j * g.nx + i;
  double sx = 0.0, sy = 0.0;
  if (j + 1 < g.ny || g.py) sx += lx[wrap(j + 1, g.ny) * g.nx + i];
  if (j > 0 || g.py) sx -= lx[c];
  if (!g.py && j == 0) sx += lx[i];
  if (!g.py && j == 1) sx -= lx[i];
  if (i > 0 || g.px) sy += ly[c];
  if (i + 1 < g.nx || g.px) sy -= ly[j * g.nx + wrap(i + 1, g.nx)];
  if (!g.px && i == 0) sy -= ly[j * g.nx];
  if (!g.px && i == 1) sy += ly[j * g.nx];
  return a.c1 * (a.dt * g.inv_dy * sx + a.dt * g.inv_dx * sy);
}

// One face: blockIdx.y gives the direction.  Bound by latency, of the FP64 chains
// of the slopes and the solver and of the loads before them, so by the warps in
// flight: five blocks of 128 an SM at 96 registers (HLLD, which spills twice as
// much there, four) ran a 512^2 HLLE launch in 61 us, four in 69, two at 214 in 118;
// with twelve forward tangents instead of the transposed solver it took 136.
template <int SOLVER>
__global__ void __launch_bounds__(128, SOLVER == RIEMANN_HLLD ? 4 : 5) k_rev_faces(const __grid_constant__ RevStage a) {
  const AdjGeom& g = a.g;
  const bool ydir = blockIdx.y != 0;
  const int d = ydir ? 1 : 0;
  const int nx = g.nx, ny = g.ny;
  const long long n = (long long)nx * ny;
  grid_wait();
  grid_release();
  const bool full_bounds = *a.tape.nan_seen != 0;   // a NaN somewhere: the bounds' comparisons decide
  for (long long cc = blockIdx.x * (long long)blockDim.x + threadIdx.x; cc < n; cc += (long long)gridDim.x * blockDim.x) {
    const int c = int(cc);
    const int i = c % nx, j = c / nx;
    // away from the sides every index is an offset (the corner one cell below takes
    // the general rule up to column and row 2, see corner_adjoint)
    const bool inner = i >= 3 && i < nx - 2 && j >= 3 && j < ny - 2;
    FaceIdx f;
    if (inner) {
      const int on = ydir ? nx : 1;
      f.a = c;
      f.b = f.to = c + on;
      f.am = c - on;
      f.bp = c + 2 * on;
      f.axp = c + 1; f.axm = c - 1; f.ayp = c + nx; f.aym = c - nx;
      f.b_in = true;
      f.b_own = false;
    } else {
      f = face_idx(g, i, j, ydir);
    }
    // the face states, normal components first (slots 1, 2 and 4, 5 trade places for
    // a y face), as phase 2 of the stage kernel makes them
    const double inv_h = ydir ? g.inv_dy : g.inv_dx, inv_2h = ydir ? g.inv_2dy : g.inv_2dx;
    const double hh = ydir ? g.hy : g.hx;
    auto field = [&](int q) { return (q == 1 || q == 4) ? q + d : ((q == 2 || q == 5) ? q - d : q); };
    auto slope = [&](double lo, double mid, double hi) {
      if (!g.slope) return (hi - lo) * inv_2h;
      if (g.limiter == LIMITER_VAN_LEER) return limit_slope<double, LIMITER_VAN_LEER>((mid - lo) * inv_h, (hi - mid) * inv_h);
      return limit_slope<double, LIMITER_MC>((mid - lo) * inv_h, (hi - mid) * inv_h);
    };
    double L[6], Rv[6];
    unsigned outside = 0;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const double* s = a.tape.P[field(q)];
      const double fm = s[f.am], f0 = s[f.a], fp = s[f.b], fpp = s[f.bp];
      const double fb0 = f.b_own ? fp : f0;   // the high cell's low neighbour in its slope
      L[q] = f0 + hh * slope(fm, f0, fp);
      Rv[q] = fp - hh * slope(fb0, fp, fpp);
      // between the two cells' values (and above the rho / P floor of the bounds):
      // inside the MOOD bounds
      const double vlo = (f0 < fp) ? f0 : fp, vhi = (f0 < fp) ? fp : f0;
      bool in = L[q] >= vlo && L[q] <= vhi && Rv[q] >= vlo && Rv[q] <= vhi;
      if (q == 0 || q == 3) in = in && L[q] >= 0.1e-8 && Rv[q] >= 0.1e-8;
      if (!in) outside |= 1u << q;
    }
    unsigned toL = 0, toR = 0;      // bit q: the state was reset to the low cell's value
    unsigned cutL = 0, cutR = 0;    // bit q: a face floor holds
    if (g.mood && (outside || full_bounds)) {
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const double* s = a.tape.P[field(q)];
        const double f0 = s[f.a];
        double lo = dmin(dmin(dmin(dmin(f0, s[f.axp]), s[f.axm]), s[f.ayp]), s[f.aym]);
        const double hi = dmax(dmax(dmax(dmax(f0, s[f.axp]), s[f.axm]), s[f.ayp]), s[f.aym]);
        if (q == 0 || q == 3) lo = dmax(0.1e-8, lo);
        if (L[q] < lo || L[q] > hi) { L[q] = f0; toL |= 1u << q; }
        if (Rv[q] < lo || Rv[q] > hi) { Rv[q] = f0; toR |= 1u << q; }
      }
    }
#pragma unroll
    for (int q = 0; q < 6; q += 3) {
      if (!(L[q] > 1.0e-8)) { L[q] = 1.0e-8; cutL |= 1u << q; }
      if (!(Rv[q] > 1.0e-8)) { Rv[q] = 1.0e-8; cutR |= 1u << q; }
    }
    const bool coldL = L[3] - 0.5 * (L[4] * L[4] + L[5] * L[5]) < K<double>::P_floor;
    const bool coldR = Rv[3] - 0.5 * (Rv[4] * Rv[4] + Rv[5] * Rv[5]) < K<double>::P_floor;
    if (coldL || coldR) {
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const double f0 = a.tape.P[field(q)][f.a];
        if (coldL) L[q] = f0;
        if (coldR) Rv[q] = f0;
      }
    }
    if (coldL) { toL = 0x3fu; cutL = 0; }
    if (coldR) { toR = 0x3fu; cutR = 0; }
    // adjoint of the face's fluxes: the flux leaves cell a and enters the cell above
    // (none past an outflow high side)
    double lF[5];
    {
      double lo[4], hi[4] = {0.0, 0.0, 0.0, 0.0};
      update_adjoint(a, f.a, lo);
      if (f.b_in) update_adjoint(a, f.to, hi);
      const double w = a.dt * (ydir ? g.dx : g.dy);
      const double mx = w * (hi[1] - lo[1]), my = w * (hi[2] - lo[2]);
      lF[0] = w * (hi[0] - lo[0]);
      lF[1] = ydir ? my : mx;
      lF[2] = ydir ? mx : my;
      lF[3] = w * (hi[3] - lo[3]);
    }
    // Ez(i,j) = 1/4 (-Fx(i,j) - Fx(i,j+1) + Fy(i,j) + Fy(i+1,j)); at an outflow
    // high side Fx(i,ny) / Fy(nx,j) is the face itself (zero gradient)
    {
      double s4;
      if (inner) {
        const double* lx = a.lout[4];
        const double* ly = a.lout[5];
        const int m = ydir ? c - 1 : c - nx;   // the face's other corner
        const double sx = (lx[c + nx] - lx[c]) + (lx[m + nx] - lx[m]), sy = (ly[c] - ly[c + 1]) + (ly[m] - ly[m + 1]);
        s4 = a.c1 * (a.dt * g.inv_dy * sx + a.dt * g.inv_dx * sy);
      } else {
      const double e0 = corner_adjoint(a, i, j);
      s4 = e0;
      if (!ydir) {
        if (j > 0 || g.pyh) s4 += corner_adjoint(a, i, wrap(j - 1, g.ny));
        if (j == g.ny - 1 && !g.pyh) s4 += e0;
      } else {
        if (i > 0 || g.pxh) s4 += corner_adjoint(a, wrap(i - 1, g.nx), j);
        if (i == g.nx - 1 && !g.pxh) s4 += e0;
      }
      }
      lF[4] = (ydir ? 0.25 : -0.25) * s4;
    }
    double gL[6], gR[6];
    face_vjp<SOLVER>(g.gamma, g.igm1, L, Rv, lF, gL, gR);
    // back through the decisions: on through the slope, to the low cell's value, or lost to a floor
    const unsigned direct = (toL & ~cutL) | (toR & ~cutR);
    a.fflag[d][c] = direct ? 1 : 0;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const unsigned b = 1u << q;
      a.fL[d][field(q)][c] = ((toL | cutL) & b) ? 0.0 : gL[q];
      a.fR[d][field(q)][c] = ((toR | cutR) & b) ? 0.0 : gR[q];
      if (direct) a.fX[d][field(q)][c] = ((toL & ~cutL & b) ? gL[q] : 0.0) + ((toR & ~cutR & b) ? gR[q] : 0.0);
    }
  }
}

// The slope's derivative w.r.t. its two one-sided differences dl, dr (times ls, the
// slope's adjoint), each back to the field: wl for (f0 - fm), wr for (fp - f0).
// Kink convention where a one-sided difference is exactly zero (a uniform
// neighbourhood): both zero -> the centred slope's (1/2, 1/2), the limit along
// dl = dr for MC and Van Leer; one zero -> the mean of the one-sided derivatives,
// 1 w.r.t. the zero argument (the limiters grow as 2|df| on the active side), 0
// w.r.t. the other.  Ties of the MC minimum: the mean.
__device__ __forceinline__ void slope_vjp(const AdjGeom& g, double dl, double dr, double& sl, double& sr) {
  const double prod = dl * dr, den = dl + dr;
  sl = sr = 0.0;
  if (dl == 0.0 || dr == 0.0) {
    sl = (dl != 0.0) ? 0.0 : ((dr == 0.0) ? 0.5 : 1.0);
    sr = (dl == 0.0) ? ((dr == 0.0) ? 0.5 : 0.0) : 1.0;
  } else if (!(prod <= 0.0 || fabs(den) < 1e-12)) {
    if (g.limiter == LIMITER_VAN_LEER) {
      const double ib = 1.0 / den, s = (2.0 * prod) * ib;
      sl = (2.0 * dr - s) * ib;
      sr = (2.0 * dl - s) * ib;
    } else {
      const double x = 2.0 * fabs(dl), y = 2.0 * fabs(dr), z = 0.5 * fabs(den);
      const double wx = min_weight(x, y), m = (x < y) ? x : y, wm = min_weight(m, z);
      sl = 2.0 * wx * wm + 0.5 * (1.0 - wm);
      sr = 2.0 * (1.0 - wx) * wm + 0.5 * (1.0 - wm);
    }
  }
}

// Where the magnetic floor X cut a recovered pressure, or ties with it: derivatives of
// the pressure w.r.t. the recovered value (from the quotient E / vol, rounded
// once as the forward rounds it) and w.r.t. X.  Rare: kept out of line.
__device__ __noinline__ double2 cut_pressure_weights(double E, double vol, double ke, double hB, double gm1,
                                                    double X) {
  const double P0 = ((E / vol - ke) - hB) * gm1 + hB;
  const bool warm = P0 > K<double>::P_floor;
  const double w = max_weight(warm ? P0 : K<double>::P_floor, X);
  return make_double2(warm ? w : 0.0, 1.0 - w);
}

__device__ __forceinline__ int wrap_far(int p, int n) {   // any p >= -n
  while (p < 0) p += n;
  while (p >= n) p -= n;
  return p;
}

constexpr int RC_TX = 32, RC_TY = 8, RC_NT = 352;   // cells of a CTA's tile, threads
constexpr int RC_EX = RC_TX + 1, RC_EY = RC_TY + 1;   // with the column and the row above, for the face B

// One cell: a CTA takes a 32 x 8 tile and the column and row beyond it, whose cell-B
// adjoints the tile's face B needs (297 cells on 352 threads).  Field by field, the
// limiter's derivative of every slope that touches the tile goes to shared memory
// once (35 x 9 in x, 33 x 11 in y: two a thread, whose indices are formed once) and
// each cell gathers its own and its neighbours'; fields in pairs (twice the loads in
// flight) and two buffers, so that three barriers are enough.  Bound by the latency of
// those loads (long-scoreboard stalls 11 an issue with one field a barrier): two CTAs
// an SM at 80 registers took 98 us at 512^2 field by field and 70 in pairs, one CTA at
// 168 registers 30 us more.
__global__ void __launch_bounds__(RC_NT, 2) k_rev_cells(const __grid_constant__ RevStage a) {
  constexpr int XW = RC_EX + 2, NX = XW * RC_EY, YW = RC_EX, NY = YW * (RC_EY + 2);
  constexpr int SLOTS = (NX + NY + RC_NT - 1) / RC_NT;
  __shared__ double sw[2][2][2][NX + NY];   // [buffer][field of the pair][wl, wr]: x slopes, then y slopes
  __shared__ double sB[2][RC_EX * RC_EY];
  const AdjGeom& g = a.g;
  const int nx = g.nx, ny = g.ny;
  const unsigned n = unsigned(nx) * unsigned(ny);
  const int tiles_x = (nx + RC_TX - 1) / RC_TX, tiles_y = (ny + RC_TY - 1) / RC_TY;
  const int tid = threadIdx.x;
  grid_wait();
  grid_release();
  for (int tile = blockIdx.x; tile < tiles_x * tiles_y; tile += gridDim.x) {
    const int i0 = (tile % tiles_x) * RC_TX, j0 = (tile / tiles_x) * RC_TY;
    // this thread's slopes: the cell, its neighbours in the slope (each side's ghost
    // rule) and the face below it, if it is that face's high cell
    // (faces of y at n + cell: the two directions' arrays of a field adjoin)
    int sk[SLOTS], slo[SLOTS], shi[SLOTS];
    unsigned sf[SLOTS];
    bool below[SLOTS];
#pragma unroll
    for (int t = 0; t < SLOTS; ++t) {
      const int e = tid + t * RC_NT;
      const bool yd = e >= NX;
      const int ee = yd ? e - NX : e;
      const int pi = wrap_far(i0 + (yd ? ee % YW : ee % XW - 1), nx), pj = wrap_far(j0 + (yd ? ee / YW - 1 : ee / XW), ny);
      sk[t] = pj * nx + pi;
      if (!yd) {
        slo[t] = pj * nx + src(pi - 1, nx, g.px, g.pxh);
        shi[t] = pj * nx + src(pi + 1, nx, g.px, g.pxh);
        below[t] = pi > 0 || g.pxh;
        sf[t] = unsigned(pj * nx + wrap(pi - 1, nx));
      } else {
        slo[t] = src(pj - 1, ny, g.py, g.pyh) * nx + pi;
        shi[t] = src(pj + 1, ny, g.py, g.pyh) * nx + pi;
        below[t] = pj > 0 || g.pyh;
        sf[t] = n + unsigned(wrap(pj - 1, ny) * nx + pi);
      }
    }
    const bool have = tid < RC_EX * RC_EY;
    const int li = tid % RC_EX, lj = have ? tid / RC_EX : 0;
    const int i = wrap_far(i0 + li, nx), j = wrap_far(j0 + lj, ny);
    const int c = j * nx + i;
    // the faces whose high cell this is: none at x = 0 / y = 0
    // unless the high side wraps to it; past an outflow high side the ghost's
    // value is this cell's (its slope, from two equal differences, depends on
    // no cell)
    const int fxm = (i > 0 || g.pxh) ? j * nx + wrap(i - 1, nx) : -1;
    const int fym = (j > 0 || g.pyh) ? wrap(j - 1, ny) * nx + i : -1;
    const bool ex = !g.pxh && i == nx - 1, ey = !g.pyh && j == ny - 1;
    const bool resetx = a.fflag[0][c] != 0, resety = a.fflag[1][c] != 0;
    double lP[6];
#pragma unroll
    for (int q0 = 0; q0 < 6; q0 += 2) {
#pragma unroll
      for (int t = 0; t < SLOTS; ++t) {
        const int e = tid + t * RC_NT;
        if (e >= NX + NY) break;
        const bool yd = e >= NX;
        const unsigned fk = yd ? n + unsigned(sk[t]) : unsigned(sk[t]);
        double fm[2], f0[2], fp[2], ls[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const double* P = a.tape.P[q0 + w];
          fm[w] = P[slo[t]];
          f0[w] = P[sk[t]];
          fp[w] = P[shi[t]];
          ls[w] = a.fL[0][q0 + w][fk] - (below[t] ? a.fR[0][q0 + w][sf[t]] : 0.0);
        }
        // the slope moves a face state by half a spacing, and its differences are over
        // a whole one (unlimited: two): factors 1/2 and 1/4 in all
        const double inv_h = yd ? g.inv_dy : g.inv_dx;
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          double sl = 0.5, sr = 0.5;
          if (g.slope)
            slope_vjp(g, (f0[w] - fm[w]) * inv_h, (fp[w] - f0[w]) * inv_h, sl, sr);
          sw[(q0 >> 1) & 1][w][0][e] = 0.5 * ls[w] * sl;
          sw[(q0 >> 1) & 1][w][1][e] = 0.5 * ls[w] * sr;
        }
      }
      __syncthreads();
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        if (!have) break;
        const double* const wl = sw[(q0 >> 1) & 1][w][0];
        const double* const wr = sw[(q0 >> 1) & 1][w][1];
        const int q = q0 + w;
        // this cell is the low cell of faces (c, x) and (c, y), the high cell of (fxm, x) and (fym, y)
        double v = a.fL[0][q][c] + a.fL[1][q][c];
        if (fxm >= 0) v += a.fR[0][q][fxm];
        if (fym >= 0) v += a.fR[1][q][fym];
        if (ex) v += a.fR[0][q][c];
        if (ey) v += a.fR[1][q][c];
        if (resetx) v += a.fX[0][q][c];
        if (resety) v += a.fX[1][q][c];
        // slopes: s(p) uses f(p-1), f(p), f(p+1).  The cell's own slope, with its own
        // ghost below / above where that side is outflow, then the slopes of the cells
        // whose low / high neighbour it is (across a periodic side, through the wrap)
#pragma unroll
        for (int dd = 0; dd < 2; ++dd) {
          const int at = dd ? NX + (lj + 1) * YW + li : lj * XW + li + 1, step = dd ? YW : 1;
          const bool per = dd ? g.py : g.px, perh = dd ? g.pyh : g.pxh;
          const int k = dd ? j : i, nk = dd ? ny : nx;
          v += ((k == 0 && !per) ? 0.0 : wl[at]) - ((k == nk - 1 && !perh) ? 0.0 : wr[at]);
          if (k + 1 < nk || per) v -= wl[at + step];
          if (k > 0 || perh) v += wr[at - step];
        }
        lP[q] = v;
      }
    }
    // primitives -> conserved (get_primitive transposed), and the cell B
    double lup[4], lbl[4], lin[4];
    if (have) {
      const unsigned hit = a.tape.hit[c];
      if (hit || (!g.px && i == 0) || (!g.py && j == 0)) {
        double u4[4], b4[4], lB[2], lcor[6];
        cell_adjoint_slow(a, c, u4, b4, lB, lcor);
#pragma unroll
        for (int q = 0; q < 4; ++q) { lup[q] = u4[q]; lbl[q] = b4[q]; }
        lP[4] += lB[0];
        lP[5] += lB[1];
#pragma unroll
        for (int q = 0; q < 6; ++q) lP[q] += lcor[q];
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          lbl[q] = a.lout[q][c];
          lup[q] = a.c1 * lbl[q];
        }
      }
      const double r = a.tape.P[0][c], u = a.tape.P[1][c], v = a.tape.P[2][c];
      const double Bx = a.tape.P[4][c], By = a.tape.P[5][c];
      const double gm1 = g.gamma - 1.0, hB = 0.5 * (Bx * Bx + By * By), vv = u * u + v * v, ke = 0.5 * r * vv;
      // The branches the recovery took, from what it left: its pressure is above X where
      // it was not cut by it, its density above the floor where the mass was.
      const double P = a.tape.P[3][c], X = hB + K<double>::e_floor_frac * (ke + hB);
      double2 w = make_double2(P > K<double>::P_floor ? 1.0 : 0.0, 0.0);
      if (!(P > X)) w = cut_pressure_weights(a.U[3][c], g.vol, ke, hB, gm1, X);
      const double a0 = w.x * lP[3], aX = w.y * lP[3];
      const double ake = K<double>::e_floor_frac * aX - a0 * gm1;
      const double ahB = (1.0 + K<double>::e_floor_frac) * aX + a0 * (1.0 - gm1);
      const double ir = 1.0 / r, im = ir * g.ivol;
      const double au = lP[1] + ake * r * u, av = lP[2] + ake * r * v;
      const double ar = lP[0] + ake * (0.5 * vv) - (au * u + av * v) * ir;
      lin[0] = (r > K<double>::rho_floor) ? ar * g.ivol : 0.0;
      lin[1] = au * im;
      lin[2] = av * im;
      lin[3] = a0 * gm1 * g.ivol;
      sB[0][tid] = lP[4] + ahB * Bx;
      sB[1][tid] = lP[5] + ahB * By;
    }
    __syncthreads();
    if (have && li < RC_TX && lj < RC_TY && i0 + li < nx && j0 + lj < ny) {
      // face B: the CT identity and the two cell averages it enters: b_x(i) enters Bx(i)
      // (alone at an outflow low side) and Bx(i+1) (none past the high side)
      const double o4 = a.lout[4][c], o5 = a.lout[5][c];
      double l[6];
#pragma unroll
      for (int q = 0; q < 4; ++q) l[q] = lup[q] + lin[q];
      l[4] = a.c1 * o4 + ((i > 0 || g.px) ? 0.5 : 1.0) * sB[0][tid] +
             ((i + 1 < nx || g.px) ? 0.5 * sB[0][tid + 1] : 0.0);
      l[5] = a.c1 * o5 + ((j > 0 || g.py) ? 0.5 : 1.0) * sB[1][tid] +
             ((j + 1 < ny || g.py) ? 0.5 * sB[1][tid + RC_EX] : 0.0);
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const double b = (q < 4) ? lbl[q < 4 ? q : 0] : (q == 4 ? o4 : o5);
        if (a.stage == 3) a.lU0[q][c] = a.c0 * b;
        else if (a.stage == 2) a.lU0[q][c] += a.c0 * b;
        else l[q] += a.lU0[q][c];
        a.lin[q][c] = l[q];
      }
    }
    __syncthreads();   // the shared arrays are reused by the next tile
  }
}

// Per-call descriptors of the stage kernels in device memory: one upload a call.
struct StepDesc {
  Member member;
  Control ctl;
  TapeOut tape[3];
  int nan_seen;
};

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct chimera_adjoint {
  AdjGeom g;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int n = 0;
  int sms = 148;
  KernelSet forward, taped;        // the fused stage kernels without and with the tape
  int grid_forward[3] = {}, grid_taped[3] = {};
  Member member;                   // without its buffers and tiling
  double* pool = nullptr;
  TapeOut tape[3];
  double* fL[2][6];
  double* fR[2][6];
  double* fX[2][6];
  unsigned char* fflag[2];
  double* U1[6];
  double* U2[6];
  double* lA[6];     // stage adjoint buffers
  double* lB[6];
  double* lU0[6];    // accumulated U^n adjoint from the blends
  StepDesc* desc = nullptr;   // device
};

static int adj_fail() {
  cudaGetLastError();
  return CHIMERA_ERR_CUDA;
}

// An adjoint is one grid: the single-grid instantiation where there is one.
static const void* function_of(const KernelEntry& k) { return k.one ? k.one : k.fn; }

static int resident_ctas(const chimera_adjoint* a, const KernelEntry& k) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, function_of(k), k.nt, k.smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  cudaGetLastError();
  return per_sm * a->sms;
}

static int tiles_of(const chimera_adjoint* a, const KernelEntry& k) {
  return ((a->g.nx + k.tx - 1) / k.tx) * ((a->g.ny + k.ty - 1) / k.ty);
}

// The stage kernels of this grid, as the solver's handles choose them: a small-grid
// tile where the device holds all of them at once, else a large one (without the
// caller's arrays' tensor maps it takes plain loads everywhere).
static void pick_kernels(chimera_adjoint* a, bool mixed) {
  auto allow = [&](KernelSet& ks) {
    for (int s = 0; s < 3; ++s)
      cudaFuncSetAttribute(function_of(ks.stage[a->g.riemann - 1][s]), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           int(ks.stage[a->g.riemann - 1][s].smem));
    cudaGetLastError();
  };
  auto fits = [&](const KernelSet& ks) {
    for (int s = 0; s < 3; ++s) {
      const KernelEntry& k = ks.stage[a->g.riemann - 1][s];
      if (tiles_of(a, k) > resident_ctas(a, k)) return false;
    }
    return true;
  };
  auto grids = [&](const KernelSet& ks, int* grid) {
    for (int s = 0; s < 3; ++s) {
      const KernelEntry& k = ks.stage[a->g.riemann - 1][s];
      grid[s] = std::max(1, std::min(tiles_of(a, k), resident_ctas(a, k)));
    }
  };
  if (mixed) {
    fp64_mixed_pair_kernels(&a->forward);
    tape_mixed_pair_kernels(&a->taped);
  } else {
    bool found = false;
    for (int v : {7, 8, 9}) {   // the small-grid variants
      fp64_kernels(v, &a->forward);
      allow(a->forward);
      if ((found = fits(a->forward))) break;
    }
    if (!found) fp64_kernels(a->g.riemann == CHIMERA_RIEMANN_HLLD ? 11 : 10, &a->forward);
    tape_kernels(true, &a->taped);
    allow(a->taped);
    if (!fits(a->taped)) tape_kernels(false, &a->taped);
  }
  allow(a->forward);
  allow(a->taped);
  grids(a->forward, a->grid_forward);
  grids(a->taped, a->grid_taped);
}

extern "C" int chimera_adjoint_create(const chimera_cfg* cfg, void* stream, chimera_adjoint** out) {
  if (!cfg || !out) return CHIMERA_ERR_BAD_ARG;
  *out = nullptr;
  if (cfg->nx < 4 || cfg->ny < 4 || !(cfg->dx > 0) || !(cfg->dy > 0) || !(cfg->gamma > 1.0)) return CHIMERA_ERR_BAD_ARG;
  if (cfg->riemann < 1 || cfg->riemann > 3 || cfg->limiter < 1 || cfg->limiter > 2) return CHIMERA_ERR_BAD_ARG;
  for (int b : {cfg->bc_xlo, cfg->bc_xhi, cfg->bc_ylo, cfg->bc_yhi})
    if (b < CHIMERA_BC_PERIODIC || b > CHIMERA_BC_INFLOW) return CHIMERA_ERR_BAD_ARG;
  // every non-periodic kind acts as outflow (src/mhd_bc.f90:36-121), each
  // side on its own (a periodic side may face an outflow one)
  if (cfg->precision != CHIMERA_FP64) return CHIMERA_ERR_UNSUPPORTED;
  if ((long long)cfg->nx * cfg->ny >= (1LL << 31)) return CHIMERA_ERR_TOO_LARGE;   // int cell indices
  chimera_adjoint* a = new (std::nothrow) chimera_adjoint();
  if (!a) return CHIMERA_ERR_NOMEM;
  AdjGeom& g = a->g;
  g.nx = cfg->nx; g.ny = cfg->ny;
  g.dx = cfg->dx; g.dy = cfg->dy;
  g.inv_dx = 1.0 / cfg->dx; g.inv_dy = 1.0 / cfg->dy;
  g.inv_2dx = 1.0 / (2.0 * cfg->dx); g.inv_2dy = 1.0 / (2.0 * cfg->dy);
  g.hx = 0.5 * cfg->dx; g.hy = 0.5 * cfg->dy;
  g.gamma = cfg->gamma;
  g.vol = cfg->dx * cfg->dy;
  g.igm1 = 1.0 / (cfg->gamma - 1.0);
  g.ivol = 1.0 / g.vol;
  g.riemann = cfg->riemann; g.limiter = cfg->limiter;
  g.slope = cfg->use_slope_limiting ? 1 : 0;
  g.mood = cfg->mood ? 1 : 0;
  g.px = cfg->bc_xlo == CHIMERA_BC_PERIODIC;
  g.py = cfg->bc_ylo == CHIMERA_BC_PERIODIC;
  g.pxh = cfg->bc_xhi == CHIMERA_BC_PERIODIC;
  g.pyh = cfg->bc_yhi == CHIMERA_BC_PERIODIC;
  a->n = cfg->nx * cfg->ny;
  if (stream) a->stream = (cudaStream_t)stream;
  else {
    if (cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking) != cudaSuccess) { delete a; return adj_fail(); }
    a->own_stream = true;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&a->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    a->sms = 148;
  }
  Member& m = a->member;
  memset(&m, 0, sizeof(m));
  m.nx = g.nx; m.ny = g.ny;
  m.periodic_x = g.px; m.periodic_y = g.py;
  m.periodic_xhi = g.pxh; m.periodic_yhi = g.pyh;
  m.square = (cfg->dx == cfg->dy) ? 1 : 0;
  m.dx = g.dx; m.dy = g.dy;
  m.inv_dx = g.inv_dx; m.inv_dy = g.inv_dy;
  m.inv_2dx = g.inv_2dx; m.inv_2dy = g.inv_2dy;
  m.hx = g.hx; m.hy = g.hy;
  m.gamma = g.gamma;
  m.vol = g.vol;
  m.len = (cfg->dx < cfg->dy) ? cfg->dx : cfg->dy;
  m.inv_vol = 1.0 / g.vol;
  m.rcp_vol = shared_reciprocal(g.vol);
  m.rcp_gm1 = shared_reciprocal(g.gamma - 1.0);
  pick_kernels(a, g.px != g.pxh || g.py != g.pyh);
  // doubles per cell: tapes 3 x (6 P + 4 Upre + 4 Ublend), faces 2 x 18, U1, U2, lA, lB, lU0 (30);
  // bytes: 3 floor marks and 2 face flags
  const size_t n = size_t(a->n), per_cell = 3 * 14 + 2 * 18 + 30;
  if (cudaMalloc(&a->pool, per_cell * n * sizeof(double) + 5 * n) != cudaSuccess ||
      cudaMalloc(&a->desc, sizeof(StepDesc)) != cudaSuccess) {
    cudaGetLastError();
    chimera_adjoint_destroy(a);
    return CHIMERA_ERR_NOMEM;
  }
  double* p = a->pool;
  auto take = [&]() { double* r = p; p += n; return r; };
  for (TapeOut& t : a->tape) {
    for (int q = 0; q < 6; ++q) t.P[q] = take();
    for (int q = 0; q < 4; ++q) t.Upre[q] = take();
    for (int q = 0; q < 4; ++q) t.Ublend[q] = take();
    t.nan_seen = &a->desc->nan_seen;
  }
  for (auto* f : {a->fL, a->fR, a->fX})
    for (int q = 0; q < 6; ++q)
      for (int d = 0; d < 2; ++d) f[d][q] = take();   // (a field's two directions adjoin)
  for (auto* f : {a->U1, a->U2, a->lA, a->lB, a->lU0})
    for (int q = 0; q < 6; ++q) f[q] = take();
  unsigned char* b = reinterpret_cast<unsigned char*>(p);
  for (TapeOut& t : a->tape) { t.hit = b; b += n; }
  for (int d = 0; d < 2; ++d) { a->fflag[d] = b; b += n; }
  *out = a;
  return CHIMERA_OK;
}

extern "C" void chimera_adjoint_destroy(chimera_adjoint* a) {
  if (!a) return;
  if (a->stream) cudaStreamSynchronize(a->stream);
  cudaFree(a->pool);
  cudaFree(a->desc);
  if (a->own_stream && a->stream) cudaStreamDestroy(a->stream);
  cudaGetLastError();
  delete a;
}

// A launch that overlaps the end of the kernel before it in the stream (grid_wait in
// the kernels).
static cudaError_t launch_after(const void* fn, dim3 grid, int threads, size_t smem, cudaStream_t stream, void** args,
                                bool overlap = true) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// The three stages from U_n on the stage kernels ks.  Taped: U1 and U2 stay in the
// handle's buffers and U_{n+1} is not written.  Else U_{n+1} goes to out, which
// serves as U1 on the way.  Control is the same for all three: dry launches leave
// it alone.
static int run_stages(chimera_adjoint* a, const KernelSet& ks, const int* grid, double dt, const double* const* U_n,
                      double* const* out, bool taped) {
  StepDesc d;
  memset(&d, 0, sizeof(d));
  d.member = a->member;
  const KernelEntry& k0 = ks.stage[a->g.riemann - 1][0];
  d.member.tiles_x = (a->g.nx + k0.tx - 1) / k0.tx;
  d.member.tiles_y = (a->g.ny + k0.ty - 1) / k0.ty;
  for (int q = 0; q < 6; ++q) {
    d.member.buf[0][q] = const_cast<double*>(U_n[q]);
    d.member.buf[1][q] = taped ? a->U1[q] : out[q];
    d.member.buf[2][q] = a->U2[q];
  }
  d.ctl.dt = dt;
  d.ctl.active = 1;
  d.ctl.output_count = 1;
  for (int s = 0; s < 3; ++s) d.tape[s] = a->tape[s];
  if (cudaMemcpyAsync(a->desc, &d, sizeof(d), cudaMemcpyHostToDevice, a->stream) != cudaSuccess) return adj_fail();
  StageArgs s;
  memset(&s, 0, sizeof(s));
  s.members = &a->desc->member;
  s.ctl = &a->desc->ctl;
  s.n_members = 1;
  s.total_tiles = d.member.tiles_x * d.member.tiles_y;
  s.limiter = a->g.limiter;
  s.slope_limiting = a->g.slope;
  s.mood = a->g.mood;
  s.dry = 1;
  s.one = d.member;
  for (int k = 0; k < 3; ++k) {
    const KernelEntry& e = ks.stage[a->g.riemann - 1][k];
    s.tape = taped ? &a->desc->tape[k] : nullptr;
    void* args[] = {&s};
    if (launch_after(function_of(e), dim3(grid[k]), e.nt, e.smem, a->stream, args, k > 0) != cudaSuccess) return adj_fail();
  }
  return CHIMERA_OK;
}

// One stage of the reverse sweep from input U and output adjoint lout to lin.
static int rev_stage(chimera_adjoint* a, int stage, double dt, const double* const* U, const double* const* lout,
                      double* const* lin) {
  RevStage r;
  r.g = a->g;
  r.stage = stage;
  r.dt = dt;
  r.c0 = (stage == 1) ? 0.0 : ((stage == 2) ? 0.75 : 1.0 / 3.0);
  r.c1 = (stage == 1) ? 1.0 : ((stage == 2) ? 0.25 : 2.0 / 3.0);
  r.tape = a->tape[stage - 1];
  for (int q = 0; q < 6; ++q) {
    r.U[q] = U[q];
    r.lout[q] = lout[q];
    r.lin[q] = lin[q];
    r.lU0[q] = a->lU0[q];
    for (int d = 0; d < 2; ++d) {
      r.fL[d][q] = a->fL[d][q];
      r.fR[d][q] = a->fR[d][q];
      r.fX[d][q] = a->fX[d][q];
    }
  }
  for (int d = 0; d < 2; ++d) r.fflag[d] = a->fflag[d];
  const dim3 faces(unsigned(std::min<long long>((a->n + 127) / 128, 1 << 20)), 2);
  const void* fn = (a->g.riemann == CHIMERA_RIEMANN_RUSANOV) ? (const void*)&k_rev_faces<RIEMANN_RUSANOV>
                   : (a->g.riemann == CHIMERA_RIEMANN_HLLE)  ? (const void*)&k_rev_faces<RIEMANN_HLLE>
                                                             : (const void*)&k_rev_faces<RIEMANN_HLLD>;
  void* args[] = {&r};
  if (launch_after(fn, faces, 128, 0, a->stream, args) != cudaSuccess) return adj_fail();
  const long long tiles = (long long)((a->g.nx + RC_TX - 1) / RC_TX) * ((a->g.ny + RC_TY - 1) / RC_TY);
  if (launch_after((const void*)&k_rev_cells, dim3(unsigned(std::min<long long>(tiles, 1 << 20))), RC_NT, 0, a->stream,
                   args) != cudaSuccess)
    return adj_fail();
  return CHIMERA_OK;
}

// Whether any of the six output arrays overlaps one of the six inputs.
static bool overlaps(const chimera_adjoint* a, const double* const* in, double* const* out) {
  const uintptr_t bytes = uintptr_t(a->n) * sizeof(double);
  for (int p = 0; p < 6; ++p)
    for (int q = 0; q < 6; ++q) {
      const uintptr_t x = reinterpret_cast<uintptr_t>(in[p]), y = reinterpret_cast<uintptr_t>(out[q]);
      if (x < y + bytes && y < x + bytes) return true;
    }
  return false;
}

static int copy6(chimera_adjoint* a, double* const* dst, double* const* src) {
  for (int q = 0; q < 6; ++q)
    if (cudaMemcpyAsync(dst[q], src[q], size_t(a->n) * sizeof(double), cudaMemcpyDeviceToDevice, a->stream) != cudaSuccess)
      return adj_fail();
  return CHIMERA_OK;
}

extern "C" int chimera_adjoint_step(chimera_adjoint* a, const double* const* U_n, double dt,
                                    const double* const* lambda_next, double* const* lambda_n) {
  if (!a || !U_n || !lambda_next || !lambda_n || !(dt > 0.0)) return CHIMERA_ERR_BAD_ARG;
  for (int q = 0; q < 6; ++q)
    if (!doubles_ok({U_n[q], lambda_next[q], lambda_n[q]})) return CHIMERA_ERR_BAD_ARG;
  int rc = run_stages(a, a->taped, a->grid_taped, dt, U_n, nullptr, true);
  if (rc) return rc;
  // lambda_n may be U_n's memory: the last stage reads U_n around the cells it writes
  const bool aside = overlaps(a, U_n, lambda_n);
  double* const* dst = aside ? a->lA : lambda_n;
  if ((rc = rev_stage(a, 3, dt, a->U2, lambda_next, a->lA))) return rc;   // lambda_U2 -> lA
  if ((rc = rev_stage(a, 2, dt, a->U1, a->lA, a->lB))) return rc;         // lambda_U1 -> lB
  if ((rc = rev_stage(a, 1, dt, U_n, a->lB, dst))) return rc;             // lambda_Un, with the blends' share
  if (aside && (rc = copy6(a, lambda_n, a->lA))) return rc;
  if (cudaGetLastError() != cudaSuccess) return CHIMERA_ERR_CUDA;
  if (cudaStreamSynchronize(a->stream) != cudaSuccess) return adj_fail();
  return CHIMERA_OK;
}

extern "C" int chimera_adjoint_forward_step(chimera_adjoint* a, const double* const* U_n, double dt,
                                            double* const* U_next) {
  if (!a || !U_n || !U_next || !(dt > 0.0)) return CHIMERA_ERR_BAD_ARG;
  for (int q = 0; q < 6; ++q)
    if (!doubles_ok({U_n[q], U_next[q]})) return CHIMERA_ERR_BAD_ARG;
  // U_next may be U_n's memory: the stages read U_n around the cells they write
  const bool aside = overlaps(a, U_n, U_next);
  int rc = run_stages(a, a->forward, a->grid_forward, dt, U_n, aside ? a->U1 : U_next, false);
  if (rc) return rc;
  if (aside && (rc = copy6(a, U_next, a->U1))) return rc;
  if (cudaGetLastError() != cudaSuccess) return CHIMERA_ERR_CUDA;
  if (cudaStreamSynchronize(a->stream) != cudaSuccess) return adj_fail();
  return CHIMERA_OK;
}
