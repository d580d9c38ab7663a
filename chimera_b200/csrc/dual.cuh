// dual.cuh -- forward-mode dual numbers for the adjoint's local Jacobians.
//
// Dual<N> carries a value and N tangents.  Evaluating conserved_floors
// (mhd_device.cuh) or the outflow correction (adjoint.cu) -- what a few cells only
// go through, the rest being transposed by hand (face_vjp.cuh) -- with Dual
// arguments returns the outputs and their exact derivatives with respect to the
// seeded inputs, through the same operations and the same branch decisions as the
// FP64 forward: comparisons look at values only, so at a kink the derivative is that
// of the branch the forward took (a one-sided derivative), except at an exact tie of
// a maximum, where it is the mean of the two one-sided derivatives.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "mhd_device.cuh"

namespace chimera {

template <int N> struct Dual {
  double v;
  double d[N];
  __host__ __device__ constexpr Dual() : v(0.0), d{} {}
  __host__ __device__ constexpr Dual(double x) : v(x), d{} {}
  __host__ __device__ constexpr Dual(int x) : v(double(x)), d{} {}
};

template <int N> __device__ __forceinline__ Dual<N> seed(double v, int k) {
  Dual<N> r(v);
  r.d[k] = 1.0;
  return r;
}

#define DUAL_BIN(OP, VEXPR, DEXPR)                                                   \
  template <int N> __device__ __forceinline__ Dual<N> operator OP(const Dual<N>& a, const Dual<N>& b) { \
    Dual<N> r;                                                                       \
    r.v = VEXPR;                                                                     \
    _Pragma("unroll") for (int k = 0; k < N; ++k) r.d[k] = DEXPR;                    \
    return r;                                                                        \
  }
DUAL_BIN(+, a.v + b.v, a.d[k] + b.d[k])
DUAL_BIN(-, a.v - b.v, a.d[k] - b.d[k])
DUAL_BIN(*, a.v * b.v, a.d[k] * b.v + a.v * b.d[k])
#undef DUAL_BIN

template <int N> __device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a.v / b.v;
  const double ib = 1.0 / b.v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = (a.d[k] - r.v * b.d[k]) * ib;
  return r;
}

// a plain constant in front (the floors)
template <int N> __device__ __forceinline__ Dual<N> operator*(double a, const Dual<N>& b) {
  Dual<N> r;
  r.v = b.v * a;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = b.d[k] * a;
  return r;
}
template <int N> __device__ __forceinline__ Dual<N> operator/(double a, const Dual<N>& b) { return Dual<N>(a) / b; }

template <int N> __device__ __forceinline__ bool operator<(const Dual<N>& a, const Dual<N>& b) { return a.v < b.v; }
template <int N> __device__ __forceinline__ bool operator>(const Dual<N>& a, const Dual<N>& b) { return a.v > b.v; }

template <int N> __device__ __forceinline__ Dual<N> dsqrt(const Dual<N>& a) {
  Dual<N> r;
  r.v = sqrt(a.v);
  const double h = (r.v > 0.0) ? 0.5 / r.v : 0.0;   // one-sided: zero derivative at sqrt(0)
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = a.d[k] * h;
  return r;
}

// max of two duals: at an exact tie the derivative is the mean of the two one-sided
// ones, which is what a central difference sees; off a tie it is that of the larger
template <int N> __device__ __forceinline__ Dual<N> dmax(const Dual<N>& a, const Dual<N>& b) {
  if (a.v > b.v) return a;
  if (b.v > a.v) return b;
  Dual<N> r(a.v);
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = 0.5 * (a.d[k] + b.d[k]);
  return r;
}

template <int N> struct K<Dual<N>> {
  static constexpr double P_floor = 1.0e-12;
  static constexpr double rho_floor = 1.0e-12;
};

}  // namespace chimera
