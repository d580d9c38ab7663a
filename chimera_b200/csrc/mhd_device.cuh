// mhd_device.cuh -- per-cell and per-face arithmetic of CHIMERA's stage operator.
//
// Templated on the arithmetic type R.  With R = double and the translation
// unit compiled with --fmad=false, every expression below rounds exactly as
// the Fortran source it cites (same operands, same left-to-right order, no
// fused multiply-add), so the FP64 form is bit-compatible with the reference
// semantics.  With R = float the same expressions run in FP32 (the FP32-bulk
// form), with FMA contraction allowed.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace chimera {

// src/mhd_config.f90:27-43
enum { RIEMANN_RUSANOV = 1, RIEMANN_HLLE = 2, RIEMANN_HLLD = 3 };
enum { LIMITER_VAN_LEER = 1, LIMITER_MC = 2 };
enum { BC_PERIODIC = 1, BC_FIXED = 2, BC_OUTFLOW = 3, BC_INFLOW = 4 };

template <typename R> struct K {
  // src/mhd_config.f90:59-61
  static constexpr R P_floor = R(1.0e-12);
  static constexpr R rho_floor = R(1.0e-12);
  static constexpr R e_floor_frac = R(1.0e-10);
};

// max / min / abs as the Fortran intrinsics evaluate them on finite values.
// FP64 keeps the compare-and-select form (bit parity, signed zeros included);
// the FP32-bulk form uses the single-instruction min / max / abs, which give
// the same result on every finite input up to the sign of a zero result.
template <typename R> __device__ __forceinline__ R dmax(R a, R b) { return (a > b) ? a : b; }
template <typename R> __device__ __forceinline__ R dmin(R a, R b) { return (a < b) ? a : b; }
template <typename R> __device__ __forceinline__ R dabs(R a) { return a < R(0) ? -a : a; }
template <> __device__ __forceinline__ float dmax<float>(float a, float b) { return fmaxf(a, b); }
template <> __device__ __forceinline__ float dmin<float>(float a, float b) { return fminf(a, b); }
template <> __device__ __forceinline__ float dabs<float>(float a) { return fabsf(a); }

// hmax / hmin / habs: the hardware min / max / abs, used only where they
// equal the compare-and-select above on every valid state -- one operand a
// positive constant, a result that only feeds comparisons, or operands known
// to be nonzero -- since they can differ from it only in the sign of a zero
// result or with a NaN second operand.  In FP64 only the absolute value (a
// sign-bit clear) is cheaper than compare-and-select; FP64 min / max keep it
// (their IEEE forms measured 20% more instructions on sm_100), and so do the
// adjoint's dual numbers (hmax).
template <typename A, typename B> __device__ __forceinline__ auto hmax(A a, B b) { return dmax(a, b); }
template <typename A, typename B> __device__ __forceinline__ auto hmin(A a, B b) { return dmin(a, b); }
__device__ __forceinline__ double habs(double a) { return fabs(a); }
__device__ __forceinline__ float hmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float hmin(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float habs(float a) { return fabsf(a); }
__device__ __forceinline__ double dsqrt(double a) { return sqrt(a); }
__device__ __forceinline__ float dsqrt(float a) { return sqrtf(a); }
__device__ __forceinline__ double dcopysign(double a, double b) { return copysign(a, b); }
__device__ __forceinline__ float dcopysign(float a, float b) { return copysignf(a, b); }
__device__ __forceinline__ bool disfinite(double a) { return isfinite(a); }

// sqrt(0.5 (q + |q|)) for q > 0 or NaN: there 0.5 (q + |q|) = 0.5 (2 q) = q
// exactly (both products by powers of two): the reference's expression
// (src/mhd_flux.f90:277-278, 355-358) is sqrt(q).
template <typename R> __device__ __forceinline__ R sqrt_pos_part(R q) { return dsqrt(q); }
__device__ __forceinline__ bool disfinite(float a) { return isfinite(a); }

// a / b through a reciprocal y = RN(1/b) fixed for the launch (the cell volume,
// gamma - 1): q = RN(a y), r = fma(-q, b, a), RN(q + r y) -- one correction
// step (P. Markstein, IBM J. Res. Dev. 34(1), 1990) -- is the correctly rounded
// quotient RN(a / b) when no step underflows or overflows.  The host gives
// y = 0 for a b outside 2^-120 <= |b| < 2^121; a numerator outside
// 2^-900 <= |a| < 2^900 (zero, subnormal, huge, Inf, NaN) takes IEEE division.
// In that range q and r y stay normal and r = a - q b is exact.
// tests/numerics/div_sweep.c compares it with IEEE division on random
// quotients and on quotients within a few 2^-106 of a rounding midpoint.
// Other arithmetic types divide.
template <typename R> __device__ __forceinline__ R div_by(R a, R b, double) { return a / b; }
template <> __device__ __forceinline__ double div_by<double>(double a, double b, double y) {
  const unsigned e = (unsigned(__double2hiint(a)) >> 20) & 0x7ffu;   // biased exponent of a
  if (y != 0.0 && e - 123u < 1800u) {
    const double q = a * y;
    const double r = fma(-q, b, a);
    return fma(r, y, q);
  }
  return a / b;
}

// A running maximum: max(run, x) as fmax(run, x) gives it for a run that is
// not NaN (a NaN x leaves run), as one compare and select -- FP64 fmax takes
// several instructions on sm_100.
__device__ __forceinline__ double run_max(double run, double x) { return (x > run) ? x : run; }

// Primitive state of one cell: rho, vx, vy, P (TOTAL pressure), Bx, By.
template <typename R> struct Prim {
  R rho, vx, vy, P, Bx, By;
};

// src/mhd_change_states.f90:61-113 (get_primitive), one cell.
// rcp_vol: RN(1/vol) for div_by, or 0.
template <typename R>
__device__ __forceinline__ Prim<R> get_primitive(R M, R Mx, R My, R E, R Bx, R By, R gamma, R vol,
                                                 double rcp_vol = 0.0) {
  Prim<R> p;
  R r = hmax(div_by(M, vol, rcp_vol), K<R>::rho_floor);
  R u = Mx / (r * vol);
  R v = My / (r * vol);
  R halfB2 = R(0.5) * (Bx * Bx + By * By);
  R P = ((div_by(E, vol, rcp_vol) - R(0.5) * r * (u * u + v * v)) - halfB2) * (gamma - R(1)) + halfB2;
  P = hmax(P, K<R>::P_floor);
  P = hmax(P, halfB2 + K<R>::e_floor_frac * (R(0.5) * r * (u * u + v * v) + halfB2));
  p.rho = r; p.vx = u; p.vy = v; p.P = P; p.Bx = Bx; p.By = By;
  return p;
}

// src/mhd_change_states.f90:16-58 (get_conserved), one cell.
template <typename R>
__device__ __forceinline__ void get_conserved(R rho, R vx, R vy, R P, R Bx, R By, R gamma, R vol, R& M, R& Mx,
                                              R& My, R& E) {
  const R rho_cp = hmax(rho, K<R>::rho_floor);
  const R P_cp = hmax(P, K<R>::P_floor);
  M = rho_cp * vol;
  Mx = M * vx;
  My = M * vy;
  const R halfB2 = R(0.5) * (Bx * Bx + By * By);
  E = (((P_cp - halfB2) / (gamma - R(1)) + R(0.5) * rho_cp * (vx * vx + vy * vy)) + halfB2) * vol;
}

// FP32-bulk form: storage and bulk arithmetic are FP32, but the pressure
// recovery p = (gamma-1)(E/vol - rho v^2/2 - B^2/2) + B^2/2 -- a small
// difference of large terms at low plasma beta -- is done in FP64 from the
// FP32 inputs, then rounded to FP32.  Same floors as get_primitive.
__device__ __forceinline__ Prim<float> get_primitive_mixed(float M, float Mx, float My, float E,
                                                           float Bx, float By, double gamma,
                                                           double inv_vol, float inv_volf) {
  Prim<float> p;
  const float r = fmaxf(M * inv_volf, 1.0e-12f);
  const float ir = 1.0f / r;
  // u and v as the two lanes of paired FP32 multiplies (the same bits as scalar ones)
  const float2 uv = __fmul2_rn(__fmul2_rn(make_float2(Mx, My), make_float2(inv_volf, inv_volf)), make_float2(ir, ir));
  const float u = uv.x;
  const float v = uv.y;
  const double rd = r, ud = u, vd = v, bx = Bx, by = By;
  const double halfB2 = 0.5 * (bx * bx + by * by);
  const double ke = 0.5 * rd * (ud * ud + vd * vd);
  double P = ((double(E) * inv_vol - ke) - halfB2) * (gamma - 1.0) + halfB2;
  P = run_max(1.0e-12, P);                              // = fmax(P, 1e-12), NaN included
  P = run_max(P, halfB2 + 1.0e-10 * (ke + halfB2));      // P is not NaN here: = fmax
  p.rho = r; p.vx = u; p.vy = v; p.P = float(P); p.Bx = Bx; p.By = By;
  return p;
}

// src/mhd_derivatives.f90:86-96 (apply_slope_limiter), one slope.
template <typename R, int LIMITER>
__device__ __forceinline__ R limit_slope(R dfL, R dfR) {
  R prod = dfL * dfR;
  R den = dfL + dfR;
  if (prod <= R(0) || habs(den) < R(1e-12)) return R(0);
  if (LIMITER == LIMITER_VAN_LEER) return (R(2) * prod) / den;
  // Here dfL and dfR are nonzero with one sign and |den| >= 1e-12.  The reference's
  // value with fewer operations: min(2|a|, 2|b|) = 2 min(|a|, |b|) (a product by 2 is
  // exact), and sign(1, a) * m = copysign(m, a) for the non-negative m (a product by
  // +-1 is exact).
  return dcopysign(hmin(R(2) * hmin(habs(dfL), habs(dfR)), R(0.5) * habs(den)), dfL);
}

// One face's 5 fluxes in (normal, tangential) orientation.
template <typename R> struct Flux5 {
  R mass, momn, momt, energy, bt;
};

// src/mhd_flux.f90:197-288 (rusanov_flux), one interface.
template <typename R>
__device__ __forceinline__ Flux5<R> rusanov(R gamma, R rho_L, R rho_R, R vx_L, R vx_R, R vy_L, R vy_R,
                                            R P_L, R P_R, R Bx_L, R Bx_R, R By_L, R By_R,
                                            double rcp_gm1 = 0.0) {
  Flux5<R> F;
  R halfBL2 = R(0.5) * (Bx_L * Bx_L + By_L * By_L);
  R halfBR2 = R(0.5) * (Bx_R * Bx_R + By_R * By_R);
  R p_th_L = hmax(P_L - halfBL2, K<R>::P_floor);
  R p_th_R = hmax(P_R - halfBR2, K<R>::P_floor);
  R gm1 = gamma - R(1);
  R en_L = (div_by(p_th_L, gm1, rcp_gm1) + R(0.5) * rho_L * (vx_L * vx_L + vy_L * vy_L)) + halfBL2;
  R en_R = (div_by(p_th_R, gm1, rcp_gm1) + R(0.5) * rho_R * (vx_R * vx_R + vy_R * vy_R)) + halfBR2;
  R rho_avg = R(0.5) * (rho_L + rho_R);
  R inv_rho_avg = R(1) / rho_avg;
  R momx_avg = R(0.5) * (rho_L * vx_L + rho_R * vx_R);
  R momy_avg = R(0.5) * (rho_L * vy_L + rho_R * vy_R);
  R en_avg = R(0.5) * (en_L + en_R);
  R Bx_avg = R(0.5) * (Bx_L + Bx_R);
  R By_avg = R(0.5) * (By_L + By_R);
  R hB = R(0.5) * (Bx_avg * Bx_avg + By_avg * By_avg);
  R P_avg = gm1 * ((en_avg - R(0.5) * (momx_avg * momx_avg + momy_avg * momy_avg) * inv_rho_avg) - hB) + hB;
  F.mass = momx_avg;
  F.momn = (momx_avg * momx_avg * inv_rho_avg + P_avg) - Bx_avg * Bx_avg;
  F.momt = momx_avg * momy_avg * inv_rho_avg - Bx_avg * By_avg;
  F.energy = (en_avg + P_avg) * momx_avg * inv_rho_avg - Bx_avg * (Bx_avg * momx_avg + By_avg * momy_avg) * inv_rho_avg;
  F.bt = (By_avg * momx_avg - Bx_avg * momy_avg) * inv_rho_avg;
  R c_L2 = (gamma * p_th_L + R(2) * halfBL2) / rho_L;
  R c_R2 = (gamma * p_th_R + R(2) * halfBR2) / rho_R;
  // c_L2, c_R2 > 0 (the thermal pressure is floored; a NaN P floors to it), so C_L, C_R > 0
  R C_L = sqrt_pos_part(c_L2) + habs(vx_L);
  R C_R = sqrt_pos_part(c_R2) + habs(vx_R);
  R C = R(0.5) * hmax(C_L, C_R);
  F.mass = F.mass - C * (rho_R - rho_L);
  F.momn = F.momn - C * (rho_R * vx_R - rho_L * vx_L);
  F.momt = F.momt - C * (rho_R * vy_R - rho_L * vy_L);
  F.energy = F.energy - C * (en_R - en_L);
  F.bt = F.bt - C * (By_R - By_L);
  return F;
}

// src/mhd_flux.f90:291-405 (hlle_flux), one interface.
template <typename R>
__device__ __forceinline__ Flux5<R> hlle(R gamma, R rho_L, R rho_R, R vx_L, R vx_R, R vy_L, R vy_R,
                                         R P_L, R P_R, R Bx_L, R Bx_R, R By_L, R By_R,
                                         double rcp_gm1 = 0.0) {
  const R cf_max_hlle = R(1.0e2);
  R halfBL2 = R(0.5) * (Bx_L * Bx_L + By_L * By_L);
  R halfBR2 = R(0.5) * (Bx_R * Bx_R + By_R * By_R);
  R p_th_L = hmax(P_L - halfBL2, K<R>::P_floor);
  R p_th_R = hmax(P_R - halfBR2, K<R>::P_floor);
  R gm1 = gamma - R(1);
  R en_L = (div_by(p_th_L, gm1, rcp_gm1) + R(0.5) * rho_L * (vx_L * vx_L + vy_L * vy_L)) + halfBL2;
  R en_R = (div_by(p_th_R, gm1, rcp_gm1) + R(0.5) * rho_R * (vx_R * vx_R + vy_R * vy_R)) + halfBR2;
  R qL = (gamma * p_th_L + R(2) * halfBL2) / rho_L;
  R qR = (gamma * p_th_R + R(2) * halfBR2) / rho_R;
  R c_fL = hmin(sqrt_pos_part(qL), cf_max_hlle);   // qL, qR > 0 (or NaN)
  R c_fR = hmin(sqrt_pos_part(qR), cf_max_hlle);
  R S_L = dmin(vx_L - c_fL, vx_R - c_fR);
  R S_R = dmax(vx_L + c_fL, vx_R + c_fR);
  R FL_Mass = rho_L * vx_L;
  R FL_Momx = (rho_L * vx_L * vx_L + P_L) - Bx_L * Bx_L;
  R FL_Momy = rho_L * vx_L * vy_L - Bx_L * By_L;
  R FL_Energy = (en_L + P_L) * vx_L - Bx_L * (Bx_L * vx_L + By_L * vy_L);
  R FL_By = By_L * vx_L - Bx_L * vy_L;
  R FR_Mass = rho_R * vx_R;
  R FR_Momx = (rho_R * vx_R * vx_R + P_R) - Bx_R * Bx_R;
  R FR_Momy = rho_R * vx_R * vy_R - Bx_R * By_R;
  R FR_Energy = (en_R + P_R) * vx_R - Bx_R * (Bx_R * vx_R + By_R * vy_R);
  R FR_By = By_R * vx_R - Bx_R * vy_R;
  Flux5<R> F;
  if (S_L >= R(0)) {
    F.mass = FL_Mass; F.momn = FL_Momx; F.momt = FL_Momy; F.energy = FL_Energy; F.bt = FL_By;
  }
  if (S_R <= R(0)) {
    F.mass = FR_Mass; F.momn = FR_Momx; F.momt = FR_Momy; F.energy = FR_Energy; F.bt = FR_By;
  }
  if (!(S_L >= R(0)) && !(S_R <= R(0))) {
    R inv_Sdiff = R(1) / hmax(S_R - S_L, R(1.0e-12));
    R SLSR = S_L * S_R;
    F.mass = ((S_R * FL_Mass - S_L * FR_Mass) + SLSR * (rho_R - rho_L)) * inv_Sdiff;
    F.momn = ((S_R * FL_Momx - S_L * FR_Momx) + SLSR * (rho_R * vx_R - rho_L * vx_L)) * inv_Sdiff;
    F.momt = ((S_R * FL_Momy - S_L * FR_Momy) + SLSR * (rho_R * vy_R - rho_L * vy_L)) * inv_Sdiff;
    F.energy = ((S_R * FL_Energy - S_L * FR_Energy) + SLSR * (en_R - en_L)) * inv_Sdiff;
    F.bt = ((S_R * FL_By - S_L * FR_By) + SLSR * (By_R - By_L)) * inv_Sdiff;
  }
  return F;
}

// HLL average of the two physical fluxes (src/mhd_flux.f90:595-600, 762-767).
template <typename R>
__device__ __forceinline__ Flux5<R> hll_avg(R SL, R SR, const Flux5<R>& FL, const Flux5<R>& FR,
                                            R dM, R dMn, R dMt, R dE, R dB) {
  Flux5<R> F;
  R inv = R(1) / (SR - SL);
  R s = SL * SR;
  F.mass = ((SR * FL.mass - SL * FR.mass) + s * dM) * inv;
  F.momn = ((SR * FL.momn - SL * FR.momn) + s * dMn) * inv;
  F.momt = ((SR * FL.momt - SL * FR.momt) + s * dMt) * inv;
  F.energy = ((SR * FL.energy - SL * FR.energy) + s * dE) * inv;
  F.bt = ((SR * FL.bt - SL * FR.bt) + s * dB) * inv;
  return F;
}

// The catch-all guard of hlld_flux (src/mhd_flux.f90:747-768): a flux that is
// not finite or exceeds FAC_BND times a bound built from the two physical
// fluxes and states is replaced by the HLL average.
template <typename R>
__device__ __forceinline__ Flux5<R> hlld_guard(Flux5<R> F, R SL, R SR, const Flux5<R>& FL, const Flux5<R>& FR, R rhoL,
                                               R rhoR, R vxL, R vxR, R vyL, R vyR, R enL, R enR, R ByL, R ByR, R dM,
                                               R dMn, R dMt, R dE, R dB) {
  const R FAC_BND = R(8.0);
  R Smax = hmax(habs(SL), habs(SR));
  R bnd_mass = hmax(habs(FL.mass), habs(FR.mass)) + Smax * (rhoL + rhoR);
  R bnd_momx = hmax(habs(FL.momn), habs(FR.momn)) + Smax * (habs(rhoL * vxL) + habs(rhoR * vxR));
  R bnd_momy = hmax(habs(FL.momt), habs(FR.momt)) + Smax * (habs(rhoL * vyL) + habs(rhoR * vyR));
  R bnd_enr = hmax(habs(FL.energy), habs(FR.energy)) + Smax * (habs(enL) + habs(enR));
  R bnd_by = hmax(habs(FL.bt), habs(FR.bt)) + Smax * (habs(ByL) + habs(ByR));
  bool use_hll = false;
  if (!disfinite(F.mass) || habs(F.mass) > FAC_BND * bnd_mass) use_hll = true;
  if (!disfinite(F.momn) || habs(F.momn) > FAC_BND * bnd_momx) use_hll = true;
  if (!disfinite(F.momt) || habs(F.momt) > FAC_BND * bnd_momy) use_hll = true;
  if (!disfinite(F.energy) || habs(F.energy) > FAC_BND * bnd_enr) use_hll = true;
  if (!disfinite(F.bt) || habs(F.bt) > FAC_BND * bnd_by) use_hll = true;
  if (use_hll) F = hll_avg(SL, SR, FL, FR, dM, dMn, dMt, dE, dB);
  return F;
}

// src/mhd_flux.f90:408-779 (hlld_flux), one interface.
template <typename R>
__device__ __forceinline__ Flux5<R> hlld(R gamma, R rhoL, R rhoR, R vxL, R vxR, R vyL, R vyR,
                                         R pTL, R pTR, R BxL, R BxR, R ByL, R ByR, double rcp_gm1 = 0.0) {
  const R EPS_FAN = R(1.0e-6);
  const R cf_max_hlld = R(50.0);
  R halfBL2 = R(0.5) * (BxL * BxL + ByL * ByL);
  R halfBR2 = R(0.5) * (BxR * BxR + ByR * ByR);
  R p_thL = hmax(pTL - halfBL2, K<R>::P_floor);
  R p_thR = hmax(pTR - halfBR2, K<R>::P_floor);
  R gm1 = gamma - R(1);
  R enL = (div_by(p_thL, gm1, rcp_gm1) + R(0.5) * rhoL * (vxL * vxL + vyL * vyL)) + halfBL2;
  R enR = (div_by(p_thR, gm1, rcp_gm1) + R(0.5) * rhoR * (vxR * vxR + vyR * vyR)) + halfBR2;

  R vdotBL = vxL * BxL + vyL * ByL;
  Flux5<R> FL, FR;
  FL.mass = rhoL * vxL;
  FL.momn = (rhoL * (vxL * vxL) + pTL) - BxL * BxL;
  FL.momt = rhoL * vxL * vyL - BxL * ByL;
  FL.energy = (enL + pTL) * vxL - BxL * vdotBL;
  FL.bt = ByL * vxL - BxL * vyL;
  R vdotBR = vxR * BxR + vyR * ByR;
  FR.mass = rhoR * vxR;
  FR.momn = (rhoR * (vxR * vxR) + pTR) - BxR * BxR;
  FR.momt = rhoR * vxR * vyR - BxR * ByR;
  FR.energy = (enR + pTR) * vxR - BxR * vdotBR;
  FR.bt = ByR * vxR - BxR * vyR;

  R caL = (BxL * BxL) / rhoL;
  R caR = (BxR * BxR) / rhoR;
  R csL2 = gamma * p_thL / rhoL;
  R csR2 = gamma * p_thR / rhoR;
  R b2L = (BxL * BxL + ByL * ByL) / rhoL;
  R b2R = (BxR * BxR + ByR * ByR) / rhoR;
  R tmpL = csL2 + b2L;
  R tmpR = csR2 + b2R;
  R cfL = hmin(dsqrt(R(0.5) * (tmpL + dsqrt(dmax(tmpL * tmpL - R(4) * csL2 * caL, R(0))))), cf_max_hlld);
  R cfR = hmin(dsqrt(R(0.5) * (tmpR + dsqrt(dmax(tmpR * tmpR - R(4) * csR2 * caR, R(0))))), cf_max_hlld);
  R SL = dmin(vxL - cfL, vxR - cfR);
  R SR = dmax(vxL + cfL, vxR + cfR);

  if (cfL >= cf_max_hlld || cfR >= cf_max_hlld) return (cfL <= cfR) ? FL : FR;   // :548-559
  if (SL >= R(0)) return FL;                                                      // :562-567
  if (SR <= R(0)) return FR;                                                      // :568-573

  R dM = rhoR - rhoL;
  R dMn = rhoR * vxR - rhoL * vxL;
  R dMt = rhoR * vyR - rhoL * vyL;
  R dE = enR - enL;
  R dB = ByR - ByL;

  R denMD = rhoR * (SR - vxR) - rhoL * (SL - vxL);
  if (habs(denMD) < R(1.0e-15)) denMD = dcopysign(R(1.0e-15), denMD);
  R SM = ((rhoR * vxR * (SR - vxR) - rhoL * vxL * (SL - vxL)) - (pTR - pTL)) / denMD;
  R pT_star = pTL + rhoL * (SL - vxL) * (SM - vxL);
  if (SM <= SL + EPS_FAN * (SR - SL) || SM >= SR - EPS_FAN * (SR - SL))          // :594-602
    return hll_avg(SL, SR, FL, FR, dM, dMn, dMt, dE, dB);
  pT_star = hmax(pT_star, K<R>::P_floor);

  R rho_Ls = rhoL * (SL - vxL) / (SL - SM);
  R denL = rhoL * (SL - vxL) * (SL - SM) - BxL * BxL;
  R vy_Ls, By_Ls;
  if (habs(denL) > R(1.0e-3) * hmax(hmax(habs(rhoL * (SL - vxL) * (SL - SM)), BxL * BxL), R(1.0e-30))) {
    vy_Ls = vyL - BxL * ByL * (SM - vxL) / denL;
    By_Ls = ByL * (rhoL * ((SL - vxL) * (SL - vxL)) - BxL * BxL) / denL;
  } else {
    vy_Ls = vyL; By_Ls = ByL;
  }
  R vdotBLs = SM * BxL + vy_Ls * By_Ls;
  R en_Ls = (((enL * (SL - vxL) - pTL * vxL) + pT_star * SM) + BxL * (vdotBL - vdotBLs)) / (SL - SM);

  R rho_Rs = rhoR * (SR - vxR) / (SR - SM);
  R denR = rhoR * (SR - vxR) * (SR - SM) - BxR * BxR;
  R vy_Rs, By_Rs;
  if (habs(denR) > R(1.0e-3) * hmax(hmax(habs(rhoR * (SR - vxR) * (SR - SM)), BxR * BxR), R(1.0e-30))) {
    vy_Rs = vyR - BxR * ByR * (SM - vxR) / denR;
    By_Rs = ByR * (rhoR * ((SR - vxR) * (SR - vxR)) - BxR * BxR) / denR;
  } else {
    vy_Rs = vyR; By_Rs = ByR;
  }
  R vdotBRs = SM * BxR + vy_Rs * By_Rs;
  R en_Rs = (((enR * (SR - vxR) - pTR * vxR) + pT_star * SM) + BxR * (vdotBR - vdotBRs)) / (SR - SM);

  R SqrtRhoLs = dsqrt(hmax(rho_Ls, K<R>::rho_floor));
  R SqrtRhoRs = dsqrt(hmax(rho_Rs, K<R>::rho_floor));
  R Bx_avg = R(0.5) * (BxL + BxR);
  R SLs = SM - dabs(Bx_avg) / SqrtRhoLs;
  R SRs = SM + dabs(Bx_avg) / SqrtRhoRs;
  R vy_ss, By_ss, en_Lss, en_Rss;
  if (habs(Bx_avg) > R(1.0e-10)) {
    R signBx = dcopysign(R(1), Bx_avg);
    R denom_ss = SqrtRhoLs + SqrtRhoRs;
    vy_ss = ((SqrtRhoLs * vy_Ls + SqrtRhoRs * vy_Rs) + signBx * (By_Rs - By_Ls)) / denom_ss;
    By_ss = ((SqrtRhoLs * By_Rs + SqrtRhoRs * By_Ls) + signBx * SqrtRhoLs * SqrtRhoRs * (vy_Rs - vy_Ls)) / denom_ss;
    R vdotBss = SM * Bx_avg + vy_ss * By_ss;
    en_Lss = en_Ls - SqrtRhoLs * signBx * (vdotBLs - vdotBss);
    en_Rss = en_Rs + SqrtRhoRs * signBx * (vdotBRs - vdotBss);
  } else {
    vy_ss = R(0.5) * (vy_Ls + vy_Rs);
    By_ss = R(0.5) * (By_Ls + By_Rs);
    en_Lss = en_Ls;
    en_Rss = en_Rs;
    SLs = SM;
    SRs = SM;
  }

  Flux5<R> F;
  if (SM >= R(0)) {
    F.mass = FL.mass + SL * (rho_Ls - rhoL);
    F.momn = FL.momn + SL * (rho_Ls * SM - rhoL * vxL);
    F.momt = FL.momt + SL * (rho_Ls * vy_Ls - rhoL * vyL);
    F.energy = FL.energy + SL * (en_Ls - enL);
    F.bt = FL.bt + SL * (By_Ls - ByL);
    if (!(SLs >= R(0))) {
      F.momt = F.momt + SLs * rho_Ls * (vy_ss - vy_Ls);
      F.energy = F.energy + SLs * (en_Lss - en_Ls);
      F.bt = F.bt + SLs * (By_ss - By_Ls);
    }
  } else {
    F.mass = FR.mass + SR * (rho_Rs - rhoR);
    F.momn = FR.momn + SR * (rho_Rs * SM - rhoR * vxR);
    F.momt = FR.momt + SR * (rho_Rs * vy_Rs - rhoR * vyR);
    F.energy = FR.energy + SR * (en_Rs - enR);
    F.bt = FR.bt + SR * (By_Rs - ByR);
    if (!(SRs <= R(0))) {
      F.momt = F.momt + SRs * rho_Rs * (vy_ss - vy_Rs);
      F.energy = F.energy + SRs * (en_Rss - en_Rs);
      F.bt = F.bt + SRs * (By_ss - By_Rs);
    }
  }

  return hlld_guard(F, SL, SR, FL, FR, rhoL, rhoR, vxL, vxR, vyL, vyR, enL, enR, ByL, ByR, dM, dMn, dMt, dE, dB);
}

// rcp_gm1: RN(1/(gamma - 1)) for div_by, or 0.
template <typename R, int SOLVER>
__device__ __forceinline__ Flux5<R> riemann(R gamma, R rL, R rR, R uL, R uR, R vL, R vR, R PL, R PR,
                                            R BnL, R BnR, R BtL, R BtR, double rcp_gm1 = 0.0) {
  if (SOLVER == RIEMANN_RUSANOV)
    return rusanov<R>(gamma, rL, rR, uL, uR, vL, vR, PL, PR, BnL, BnR, BtL, BtR, rcp_gm1);
  if (SOLVER == RIEMANN_HLLE)
    return hlle<R>(gamma, rL, rR, uL, uR, vL, vR, PL, PR, BnL, BnR, BtL, BtR, rcp_gm1);
  return hlld<R>(gamma, rL, rR, uL, uR, vL, vR, PL, PR, BnL, BnR, BtL, BtR, rcp_gm1);
}

// src/mhd_change_states.f90:116-166 (apply_conserved_floors), one cell.
// Returns a bit mask: 1 = mass floor hit, 2 = velocity cap hit.
template <typename R>
__device__ __forceinline__ int conserved_floors(R& M, R& Mx, R& My, R& E, R Bx, R By, R gamma, R vol) {
  int hit = 0;
  R halfB2 = R(0.5) * (Bx * Bx + By * By);
  if (M < K<R>::rho_floor * vol) {
    Mx = R(0);
    My = R(0);
    M = K<R>::rho_floor * vol;
    E = hmax(E, (K<R>::P_floor / (gamma - R(1)) + halfB2) * vol);
    hit |= 1;
  }
  // The velocity cap |Mom| / M > 50 can only apply where |Mom|^2 >= (40 M)^2:
  // if the computed Mx^2 + My^2 < 1600 M^2, then |Mom| / M < 40 (1 + a few
  // ulp), so the reference's test (square root, division, compare) would
  // leave the cell alone -- skipping it there changes no bit.  NaN inputs fail
  // the comparison and take the reference's path.
  if (!(Mx * Mx + My * My < R(1600) * (M * M))) {
    R mag = dsqrt(Mx * Mx + My * My);
    R v_mag = mag / M;
    if (v_mag > R(50)) {
      R scale = R(50) * M / mag;
      Mx = Mx * scale;
      My = My * scale;
      hit |= 2;
    }
  }
  return hit;
}

}  // namespace chimera
