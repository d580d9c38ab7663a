// face_vjp.cuh -- vector-Jacobian products of the Riemann solvers (FP64).
//
// face_vjp<SOLVER> takes the two states of a face and the adjoint of its five
// fluxes and returns the adjoint of the states: the solver's expressions
// (mhd_device.cuh) evaluated once and transposed by hand, in place of twelve
// forward tangents.  Values are divided as the forward divides them; the adjoints
// are multiplied by reciprocals formed once.  The branches are the forward's; where an argument sits at a
// kink the conventions are dual.cuh's: the mean of the two one-sided derivatives
// at an exact tie of a minimum / maximum, zero for |x| at 0 and for the square
// root at 0, and no derivative through a constant that a floor, a cap or a guard
// put in place.
//
// State slots: 0 rho, 1 normal velocity, 2 tangential velocity, 3 total pressure,
// 4 normal B, 5 tangential B.  Flux slots: mass, normal momentum, tangential
// momentum, energy, tangential B.
#pragma once
#include "mhd_device.cuh"

namespace chimera {

// One state with what every solver computes from it.
struct FaceSide {
  double r, u, v, P, Bn, Bt;
  double hB, p, en;   // magnetic pressure, floored thermal pressure, total energy
  double ir;          // 1 / rho
  bool warm;          // the thermal pressure is above its floor

  __device__ __forceinline__ FaceSide() {}
  // a where first, else b, field by field (no pointer to either: they stay in registers)
  static __device__ __forceinline__ FaceSide pick(bool first, const FaceSide& a, const FaceSide& b) {
    FaceSide s;
    s.r = first ? a.r : b.r; s.u = first ? a.u : b.u; s.v = first ? a.v : b.v; s.P = first ? a.P : b.P;
    s.Bn = first ? a.Bn : b.Bn; s.Bt = first ? a.Bt : b.Bt; s.hB = first ? a.hB : b.hB; s.p = first ? a.p : b.p;
    s.en = first ? a.en : b.en; s.ir = first ? a.ir : b.ir; s.warm = first ? a.warm : b.warm;
    return s;
  }
  __device__ __forceinline__ FaceSide(const double* S, double gm1)
      : r(S[0]), u(S[1]), v(S[2]), P(S[3]), Bn(S[4]), Bt(S[5]) {
    hB = 0.5 * (Bn * Bn + Bt * Bt);
    warm = P - hB > K<double>::P_floor;
    p = warm ? P - hB : K<double>::P_floor;
    en = (p / gm1 + 0.5 * r * (u * u + v * v)) + hB;
    ir = 1.0 / r;
  }
  // conserved variables in flux-slot order (tangential B in the last)
  __device__ __forceinline__ void conserved(double* U) const {
    U[0] = r; U[1] = r * u; U[2] = r * v; U[3] = en; U[4] = Bt;
  }
  __device__ __forceinline__ void flux(double* F) const {
    const double vB = u * Bn + v * Bt;
    F[0] = r * u;
    F[1] = (r * (u * u) + P) - Bn * Bn;
    F[2] = r * u * v - Bn * Bt;
    F[3] = (en + P) * u - Bn * vB;
    F[4] = Bt * u - Bn * v;
  }
};

// Adjoints of one side, gathered from everything that depends on it.
struct SideAdj {
  double r = 0.0, u = 0.0, v = 0.0, P = 0.0, Bn = 0.0, Bt = 0.0;   // the slots themselves
  double p = 0.0, en = 0.0, hB = 0.0;                              // thermal pressure, energy, magnetic pressure

  __device__ __forceinline__ void add(bool on, const SideAdj& o) {
    if (!on) return;
    r += o.r; u += o.u; v += o.v; P += o.P; Bn += o.Bn; Bt += o.Bt; p += o.p; en += o.en; hB += o.hB;
  }
  // the physical flux, with adjoint a
  __device__ __forceinline__ void through_flux(const FaceSide& s, const double* a) {
    const double vB = s.u * s.Bn + s.v * s.Bt;
    r += a[0] * s.u + a[1] * (s.u * s.u) + a[2] * (s.u * s.v);
    u += a[0] * s.r + 2.0 * a[1] * s.r * s.u + a[2] * s.r * s.v + a[3] * ((s.en + s.P) - s.Bn * s.Bn) + a[4] * s.Bt;
    v += a[2] * s.r * s.u - a[3] * s.Bn * s.Bt - a[4] * s.Bn;
    P += a[1] + a[3] * s.u;
    en += a[3] * s.u;
    Bn -= 2.0 * a[1] * s.Bn + a[2] * s.Bt + a[3] * (vB + s.Bn * s.u) + a[4] * s.v;
    Bt += a[4] * s.u - a[2] * s.Bn - a[3] * s.Bn * s.v;
  }
  // the conserved variables, with adjoint a
  __device__ __forceinline__ void through_conserved(const FaceSide& s, const double* a) {
    r += a[0] + a[1] * s.u + a[2] * s.v;
    u += a[1] * s.r;
    v += a[2] * s.r;
    en += a[3];
    Bt += a[4];
  }
  // c = sqrt((gamma p + 2 hB) / r), with adjoint a (0 where a cap holds)
  __device__ __forceinline__ void through_fast(const FaceSide& s, double gamma, double c, double a) {
    const double aq = (c > 0.0) ? a * (0.5 / c) * s.ir : 0.0;
    p += aq * gamma;
    hB += 2.0 * aq;
    r -= aq * (c * c);
  }
  // energy, thermal and magnetic pressure down to the slots; the state adjoint
  __device__ __forceinline__ void finish(const FaceSide& s, double igm1, double* g) {
    hB += en;
    p += en * igm1;
    r += en * (0.5 * (s.u * s.u + s.v * s.v));
    u += en * s.r * s.u;
    v += en * s.r * s.v;
    if (s.warm) { P += p; hB -= p; }
    g[0] = r; g[1] = u; g[2] = v; g[3] = P; g[4] = Bn + s.Bn * hB; g[5] = Bt + s.Bt * hB;
  }
};

// weight of the first argument of a minimum / maximum it takes part in
__device__ __forceinline__ double min_weight(double a, double b) { return (a < b) ? 1.0 : ((b < a) ? 0.0 : 0.5); }
__device__ __forceinline__ double max_weight(double a, double b) { return (a > b) ? 1.0 : ((b > a) ? 0.0 : 0.5); }

// The HLL average (S_R F_L - S_L F_R + S_L S_R (U_R - U_L)) / d of flux adjoint l,
// d = S_R - S_L: adjoints of the two speeds; the flux and conserved adjoints go to
// the sides.  dd: derivative of d in S_R - S_L.
__device__ __forceinline__ void hll_vjp(const FaceSide& sL, const FaceSide& sR, double SL, double SR, double d,
                                        double dd, const double* l, SideAdj& aL, SideAdj& aR, double& aSL,
                                        double& aSR) {
  double UL[5], UR[5], FL[5], FR[5];
  sL.conserved(UL); sR.conserved(UR); sL.flux(FL); sR.flux(FR);
  const double inv = 1.0 / d, s = SL * SR;
  double fl[5], fr[5], ul[5], ur[5];
  double sumL = 0.0, sumR = 0.0, sumF = 0.0;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const double n = l[k] * inv, dU = UR[k] - UL[k];
    fl[k] = SR * n;
    fr[k] = -(SL * n);
    ur[k] = s * n;
    ul[k] = -ur[k];
    sumR += n * (FL[k] + SL * dU);
    sumL += n * (SR * dU - FR[k]);
    sumF += n * (((SR * FL[k] - SL * FR[k]) + s * dU) * inv);
  }
  aSR += sumR - dd * sumF;
  aSL += sumL + dd * sumF;
  aL.through_flux(sL, fl); aL.through_conserved(sL, ul);
  aR.through_flux(sR, fr); aR.through_conserved(sR, ur);
}

// src/mhd_flux.f90:197-288
__device__ __forceinline__ void rusanov_vjp(double gamma, double igm1, const double* L, const double* Rv, const double* l,
                                            double* gL, double* gR) {
  const double gm1 = gamma - 1.0;
  const FaceSide sL(L, gm1), sR(Rv, gm1);
  double UL[5], UR[5];
  sL.conserved(UL); sR.conserved(UR);
  const double rho = 0.5 * (sL.r + sR.r), inv = 1.0 / rho;
  const double mx = 0.5 * (UL[1] + UR[1]), my = 0.5 * (UL[2] + UR[2]), en = 0.5 * (sL.en + sR.en);
  const double Bx = 0.5 * (sL.Bn + sR.Bn), By = 0.5 * (sL.Bt + sR.Bt);
  const double hB = 0.5 * (Bx * Bx + By * By);
  const double P = gm1 * ((en - 0.5 * (mx * mx + my * my) * inv) - hB) + hB;
  const double w = Bx * mx + By * my;
  const double cL = sqrt((gamma * sL.p + 2.0 * sL.hB) / sL.r), cR = sqrt((gamma * sR.p + 2.0 * sR.hB) / sR.r);
  const double CL = cL + fabs(sL.u), CR = cR + fabs(sR.u);
  const double C = 0.5 * ((CL > CR) ? CL : CR);
  const double aP = l[1] + l[3] * mx * inv;
  const double a_en = l[3] * mx * inv + gm1 * aP;
  const double a_inv = l[1] * (mx * mx) + l[2] * (mx * my) + l[3] * ((en + P) * mx - Bx * w) +
                       l[4] * (By * mx - Bx * my) - aP * gm1 * (0.5 * (mx * mx + my * my));
  const double a_mx = l[0] + inv * (2.0 * l[1] * mx + l[2] * my + l[3] * ((en + P) - Bx * Bx) + l[4] * By - aP * gm1 * mx);
  const double a_my = inv * (l[2] * mx - l[3] * Bx * By - l[4] * Bx - aP * gm1 * my);
  const double a_hB = aP * (1.0 - gm1);
  const double a_Bx = Bx * a_hB - 2.0 * l[1] * Bx - l[2] * By - inv * (l[3] * (w + Bx * mx) + l[4] * my);
  const double a_By = By * a_hB - l[2] * Bx + inv * (l[4] * mx - l[3] * Bx * my);
  const double a_rho = -(a_inv * inv * inv);
  double aC = 0.0;
#pragma unroll
  for (int k = 0; k < 5; ++k) aC -= l[k] * (UR[k] - UL[k]);
  const double half[5] = {0.5 * a_rho, 0.5 * a_mx, 0.5 * a_my, 0.5 * a_en, 0.5 * a_By};
  double ul[5], ur[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    ul[k] = half[k] + C * l[k];
    ur[k] = half[k] - C * l[k];
  }
  SideAdj aL, aR;
  aL.through_conserved(sL, ul); aR.through_conserved(sR, ur);
  aL.Bn += 0.5 * a_Bx; aR.Bn += 0.5 * a_Bx;
  const double wt = max_weight(CL, CR);
  const double aCL = 0.5 * wt * aC, aCR = 0.5 * (1.0 - wt) * aC;
  aL.u += (sL.u > 0.0) ? aCL : ((sL.u < 0.0) ? -aCL : 0.0);
  aR.u += (sR.u > 0.0) ? aCR : ((sR.u < 0.0) ? -aCR : 0.0);
  aL.through_fast(sL, gamma, cL, aCL); aR.through_fast(sR, gamma, cR, aCR);
  aL.finish(sL, igm1, gL); aR.finish(sR, igm1, gR);
}

// src/mhd_flux.f90:291-405
__device__ __forceinline__ void hlle_vjp(double gamma, double igm1, const double* L, const double* Rv, const double* l, double* gL,
                                         double* gR) {
  const double gm1 = gamma - 1.0;
  const FaceSide sL(L, gm1), sR(Rv, gm1);
  const double qL = sqrt((gamma * sL.p + 2.0 * sL.hB) / sL.r), qR = sqrt((gamma * sR.p + 2.0 * sR.hB) / sR.r);
  const double cL = (qL < 100.0) ? qL : 100.0, cR = (qR < 100.0) ? qR : 100.0;
  const double SL = dmin(sL.u - cL, sR.u - cR), SR = dmax(sL.u + cL, sR.u + cR);
  SideAdj aL, aR;
  if (SR <= 0.0) {
    aR.through_flux(sR, l);
  } else if (SL >= 0.0) {
    aL.through_flux(sL, l);
  } else {
    const double gap = SR - SL;
    double aSL = 0.0, aSR = 0.0;
    hll_vjp(sL, sR, SL, SR, (gap > 1.0e-12) ? gap : 1.0e-12, max_weight(gap, 1.0e-12), l, aL, aR, aSL, aSR);
    const double wl = min_weight(sL.u - cL, sR.u - cR), wr = max_weight(sL.u + cL, sR.u + cR);
    const double lowL = wl * aSL, highL = wr * aSR, lowR = (1.0 - wl) * aSL, highR = (1.0 - wr) * aSR;
    aL.u += lowL + highL;
    aR.u += lowR + highR;
    const double acL = highL - lowL, acR = highR - lowR;
    aL.through_fast(sL, gamma, cL, (qL < 100.0) ? acL : (qL > 100.0 ? 0.0 : 0.5 * acL));
    aR.through_fast(sR, gamma, cR, (qR < 100.0) ? acR : (qR > 100.0 ? 0.0 : 0.5 * acR));
  }
  aL.finish(sL, igm1, gL); aR.finish(sR, igm1, gR);
}

// One side's fast speed and star state of the HLLD solver.
struct HlldSide {
  double ca, cs, tmp, root, c0;   // Alfven and sound speed squared, their fast combination, its roots
  double S, X, w;                 // outer speed, S - u, rho (S - u)
  double g, ig, d, id, vB, rs, vs, Bs, vBs, es, sq;   // star state
  bool ok;                        // the star state's denominator is usable

  __device__ __forceinline__ void fast(const FaceSide& s, double gamma) {
    ca = (s.Bn * s.Bn) / s.r;
    cs = gamma * s.p / s.r;
    tmp = cs + (s.Bn * s.Bn + s.Bt * s.Bt) / s.r;
    root = sqrt(dmax(tmp * tmp - 4.0 * cs * ca, 0.0));
    c0 = sqrt(0.5 * (tmp + root));
  }
  __device__ __forceinline__ void star(const FaceSide& s, double SM, double PT) {
    vB = s.u * s.Bn + s.v * s.Bt;
    g = S - SM;
    ig = 1.0 / g;
    rs = w / g;
    d = w * g - s.Bn * s.Bn;
    ok = fabs(d) > 1.0e-3 * dmax(dmax(fabs(w * g), s.Bn * s.Bn), 1.0e-30);
    id = 1.0 / d;
    vs = ok ? s.v - s.Bn * s.Bt * (SM - s.u) / d : s.v;
    Bs = ok ? s.Bt * (s.r * (X * X) - s.Bn * s.Bn) / d : s.Bt;
    vBs = SM * s.Bn + vs * Bs;
    es = (((s.en * X - s.P * s.u) + PT * SM) + s.Bn * (vB - vBs)) / g;
    sq = sqrt(dmax(rs, K<double>::rho_floor));
  }
  __device__ __forceinline__ void through_fast(const FaceSide& s, double gamma, double a, SideAdj& A) const {
    const double aA = (c0 > 0.0) ? a * (0.5 / c0) : 0.0;
    const double ad = (root > 0.0) ? 0.5 * aA * (0.5 / root) : 0.0;
    const double at = 0.5 * aA + ad * (2.0 * tmp);
    const double acs = at - ad * (4.0 * ca), aca = -(ad * (4.0 * cs));
    A.p += acs * gamma * s.ir;
    A.r -= (acs * cs + aca * ca + at * (tmp - cs)) * s.ir;
    A.Bn += (aca + at) * (2.0 * s.Bn) * s.ir;
    A.Bt += at * (2.0 * s.Bt) * s.ir;
  }
  // adjoints of the star state (density, v, energy, B, v . B, root of the density)
  // down to the side, the outer speed (aS), X (aX), w (aw), the contact speed and the
  // star pressure
  __device__ __forceinline__ void through_star(const FaceSide& s, double SM, double PT, double ars, double avs,
                                               double aes, double aBs, double avBs, double asq, SideAdj& A,
                                               double& aX, double& aw, double& aS, double& aSM, double& aPT) const {
    if (rs > K<double>::rho_floor) ars += asq * (0.5 / sq);
    double ag = 0.0;
    {
      const double t = aes * ig;
      ag -= t * es;
      A.en += t * X;
      aX += t * s.en;
      A.P -= t * s.u;
      A.u -= t * s.P;
      aPT += t * SM;
      aSM += t * PT;
      A.Bn += t * (vB - vBs) + t * s.Bn * s.u;   // Bn (u Bn + v Bt): the factor and the product
      A.u += t * s.Bn * s.Bn;
      A.v += t * s.Bn * s.Bt;
      A.Bt += t * s.Bn * s.v;
      avBs -= t * s.Bn;
    }
    aSM += avBs * s.Bn;
    A.Bn += avBs * SM;
    avs += avBs * Bs;
    aBs += avBs * vs;
    if (ok) {
      const double q = s.r * (X * X) - s.Bn * s.Bn;
      const double tB = aBs * id;
      A.Bt += tB * q;
      const double aq = tB * s.Bt;
      A.r += aq * (X * X);
      aX += aq * (2.0 * s.r * X);
      A.Bn -= aq * (2.0 * s.Bn);
      double ad = -(tB * Bs);
      const double tv = -(avs * id), du = SM - s.u;
      A.v += avs;
      A.Bn += tv * s.Bt * du;
      A.Bt += tv * s.Bn * du;
      aSM += tv * s.Bn * s.Bt;
      A.u -= tv * s.Bn * s.Bt;
      ad -= tv * (s.Bn * s.Bt * du) * id;
      aw += ad * g;
      ag += ad * w;
      A.Bn -= ad * (2.0 * s.Bn);
    } else {
      A.v += avs;
      A.Bt += aBs;
    }
    const double tr = ars * ig;
    aw += tr;
    ag -= tr * rs;
    aS += ag;
    aSM -= ag;
  }
};

// The star state of the side that `left` names.
struct HlldStar {
  double S, rs, vs, es, Bs, vBs, sq;
  static __device__ __forceinline__ HlldStar pick(bool left, const HlldSide& a, const HlldSide& b) {
    HlldStar h;
    h.S = left ? a.S : b.S; h.rs = left ? a.rs : b.rs; h.vs = left ? a.vs : b.vs; h.es = left ? a.es : b.es;
    h.Bs = left ? a.Bs : b.Bs; h.vBs = left ? a.vBs : b.vBs; h.sq = left ? a.sq : b.sq;
    return h;
  }
};

// src/mhd_flux.f90:408-779
__device__ __forceinline__ void hlld_vjp(double gamma, double igm1, const double* L, const double* Rv, const double* l, double* gL,
                                         double* gR) {
  const double gm1 = gamma - 1.0, cap = 50.0;
  const FaceSide sL(L, gm1), sR(Rv, gm1);
  HlldSide hL, hR;
  hL.fast(sL, gamma); hR.fast(sR, gamma);
  const double cL = (hL.c0 < cap) ? hL.c0 : cap, cR = (hR.c0 < cap) ? hR.c0 : cap;
  const double SL = dmin(sL.u - cL, sR.u - cR), SR = dmax(sL.u + cL, sR.u + cR);
  SideAdj aL, aR;
  const bool capped = cL >= cap || cR >= cap;
  if (capped ? (cL <= cR) : (SL >= 0.0)) {
    aL.through_flux(sL, l);
  } else if (capped || SR <= 0.0) {
    aR.through_flux(sR, l);
  } else {
    hL.S = SL; hL.X = SL - sL.u; hL.w = sL.r * hL.X;
    hR.S = SR; hR.X = SR - sR.u; hR.w = sR.r * hR.X;
    double den = hR.w - hL.w;
    const bool guarded = fabs(den) < 1.0e-15;
    if (guarded) den = copysign(1.0e-15, den);
    const double SM = ((sR.r * sR.u * hR.X - sL.r * sL.u * hL.X) - (sR.P - sL.P)) / den;
    const double PT0 = sL.P + hL.w * (SM - sL.u);
    double aSL = 0.0, aSR = 0.0;
    bool average = SM <= SL + 1.0e-6 * (SR - SL) || SM >= SR - 1.0e-6 * (SR - SL);
    if (!average) {
      const double PT = (PT0 > K<double>::P_floor) ? PT0 : K<double>::P_floor;
      hL.star(sL, SM, PT); hR.star(sR, SM, PT);
      const double Bn = 0.5 * (sL.Bn + sR.Bn);
      const bool left = SM >= 0.0, alfven = fabs(Bn) > 1.0e-10;
      const FaceSide s = FaceSide::pick(left, sL, sR);     // the upwind side
      const HlldStar h = HlldStar::pick(left, hL, hR);
      const double sg = copysign(1.0, Bn), sigma = left ? -1.0 : 1.0;
      const double Z = alfven ? SM + sigma * (fabs(Bn) / h.sq) : SM;   // its Alfven speed
      const bool inner = left ? !(Z >= 0.0) : !(Z <= 0.0);            // the face lies behind it
      const double dss = hL.sq + hR.sq, ids = 1.0 / dss;
      const double vss = alfven ? ((hL.sq * hL.vs + hR.sq * hR.vs) + sg * (hR.Bs - hL.Bs)) / dss : 0.5 * (hL.vs + hR.vs);
      const double Bss = alfven ? ((hL.sq * hR.Bs + hR.sq * hL.Bs) + sg * hL.sq * hR.sq * (hR.vs - hL.vs)) / dss
                                : 0.5 * (hL.Bs + hR.Bs);
      const double vBss = SM * Bn + vss * Bss;
      const double ess = alfven ? h.es + sigma * (h.sq * sg * (h.vBs - vBss)) : h.es;
      // the flux (its catch-all guard compares it with a bound)
      double U[5], F[5], FL[5], FR[5];
      s.conserved(U); s.flux(F); sL.flux(FL); sR.flux(FR);
      const double Us[5] = {h.rs, h.rs * SM, h.rs * h.vs, h.es, h.Bs};
      double G[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) G[k] = F[k] + h.S * (Us[k] - U[k]);
      if (inner) {
        G[2] += Z * h.rs * (vss - h.vs);
        G[3] += Z * (ess - h.es);
        G[4] += Z * (Bss - h.Bs);
      }
      const double top = dmax(fabs(SL), fabs(SR));
      double UL[5], UR[5];
      sL.conserved(UL); sR.conserved(UR);
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const double bound = dmax(fabs(FL[k]), fabs(FR[k])) + top * (fabs(UL[k]) + fabs(UR[k]));
        if (!isfinite(G[k]) || fabs(G[k]) > 8.0 * bound) average = true;
      }
      if (!average) {
        SideAdj A;
        double ul[5], m[5], aS = 0.0, aSM = 0.0, aPT = 0.0;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          aS += l[k] * (Us[k] - U[k]);
          m[k] = h.S * l[k];
          ul[k] = -m[k];
        }
        A.through_flux(s, l);
        A.through_conserved(s, ul);
        aL.add(left, A);
        aR.add(!left, A);
        double ars = m[0] + m[1] * SM + m[2] * h.vs, avs = m[2] * h.rs, aes = m[3], aBs = m[4], avBs = 0.0, asq = 0.0;
        aSM += m[1] * h.rs;
        double ovs = 0.0, oBs = 0.0, osq = 0.0;   // the other side's star state
        if (inner) {   // (alfven: without it the Alfven speed is SM, which is not behind the face)
          const double dv = vss - h.vs, dB = Bss - h.Bs;
          const double aZ = l[2] * h.rs * dv + l[3] * (ess - h.es) + l[4] * dB;
          ars += l[2] * Z * dv;
          double avss = l[2] * Z * h.rs, aBss = l[4] * Z;
          avs -= avss;
          aBs -= aBss;
          const double ae = l[3] * Z * sigma * sg;   // of sq (vBs - vBss)
          asq += ae * (h.vBs - vBss);
          avBs += ae * h.sq;
          const double avBss = -(ae * h.sq);
          aSM += avBss * Bn;
          double aBn = avBss * SM;
          avss += avBss * Bss;
          aBss += avBss * vss;
          const double tv = avss * ids, tB = aBss * ids;
          const double dvs = hR.vs - hL.vs, ad = -(tv * vss + tB * Bss);
          const double asqL = tv * hL.vs + tB * (hR.Bs + sg * hR.sq * dvs) + ad;
          const double asqR = tv * hR.vs + tB * (hL.Bs + sg * hL.sq * dvs) + ad;
          const double both = tB * sg * hL.sq * hR.sq;
          const double avL = tv * hL.sq - both, avR = tv * hR.sq + both;
          const double aBL = tB * hR.sq - tv * sg, aBR = tB * hL.sq + tv * sg;
          asq += left ? asqL : asqR; avs += left ? avL : avR; aBs += left ? aBL : aBR;
          osq += left ? asqR : asqL; ovs += left ? avR : avL; oBs += left ? aBR : aBL;
          aSM += aZ;
          const double tz = aZ * sigma / h.sq;
          aBn += tz * sg;
          asq -= tz * fabs(Bn) / h.sq;
          aL.Bn += 0.5 * aBn;
          aR.Bn += 0.5 * aBn;
        }
        double aXL = 0.0, awL = 0.0, aXR = 0.0, awR = 0.0;
        if (left || inner)
          hL.through_star(sL, SM, PT, left ? ars : 0.0, left ? avs : ovs, left ? aes : 0.0, left ? aBs : oBs,
                          left ? avBs : 0.0, left ? asq : osq, aL, aXL, awL, aSL, aSM, aPT);
        if (!left || inner)
          hR.through_star(sR, SM, PT, left ? 0.0 : ars, left ? ovs : avs, left ? 0.0 : aes, left ? oBs : aBs,
                          left ? 0.0 : avBs, left ? osq : asq, aR, aXR, awR, aSR, aSM, aPT);
        if (left) aSL += aS; else aSR += aS;
        if (PT0 > K<double>::P_floor) {
          aL.P += aPT;
          awL += aPT * (SM - sL.u);
          aSM += aPT * hL.w;
          aL.u -= aPT * hL.w;
        }
        const double t = aSM / den;
        aR.r += t * sR.u * hR.X; aR.u += t * sR.r * hR.X; aXR += t * sR.r * sR.u;
        aL.r -= t * sL.u * hL.X; aL.u -= t * sL.r * hL.X; aXL -= t * sL.r * sL.u;
        aR.P -= t; aL.P += t;
        if (!guarded) { awR -= t * SM; awL += t * SM; }
        aL.r += awL * hL.X; aXL += awL * sL.r; aSL += aXL; aL.u -= aXL;
        aR.r += awR * hR.X; aXR += awR * sR.r; aSR += aXR; aR.u -= aXR;
      }
    }
    if (average) hll_vjp(sL, sR, SL, SR, SR - SL, 1.0, l, aL, aR, aSL, aSR);
    const double wl = min_weight(sL.u - cL, sR.u - cR), wr = max_weight(sL.u + cL, sR.u + cR);
    const double lowL = wl * aSL, highL = wr * aSR, lowR = (1.0 - wl) * aSL, highR = (1.0 - wr) * aSR;
    aL.u += lowL + highL;
    aR.u += lowR + highR;
    hL.through_fast(sL, gamma, highL - lowL, aL);
    hR.through_fast(sR, gamma, highR - lowR, aR);
  }
  aL.finish(sL, igm1, gL); aR.finish(sR, igm1, gR);
}

template <int SOLVER>
__device__ __forceinline__ void face_vjp(double gamma, double igm1, const double* L, const double* Rv, const double* l, double* gL,
                                         double* gR) {
  if constexpr (SOLVER == RIEMANN_RUSANOV) rusanov_vjp(gamma, igm1, L, Rv, l, gL, gR);
  else if constexpr (SOLVER == RIEMANN_HLLE) hlle_vjp(gamma, igm1, L, Rv, l, gL, gR);
  else hlld_vjp(gamma, igm1, L, Rv, l, gL, gR);
}

}  // namespace chimera
