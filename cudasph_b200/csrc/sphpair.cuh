// sphpair.cuh -- what the list-driven FP64 pair loops share (hydro.cu,
// adjoint.cu): distances by one reciprocal square root, the M4 kernel slopes
// without divisions, sums over the lanes of a particle.
#pragma once

#include "sph_math.cuh"

namespace sph {

// the distance r and 1 / r of a pair from its squared distance; the self
// pair (d2 = 0) gets r = 1 / r = 0 (its terms multiply a zero vector or
// take the u = 0 branch)
__device__ __forceinline__ void dist_and_inverse(double d2, double &r, double &ir) {
  ir = d2 > 0 ? rsqrt(d2) : 0.0;
  r = d2 * ir;
}

// u d(ig)/du (k_digdh) and (1/u) d(ig)/du (k_dig) share 4 pi x^2 w(x) at
// x = 4u (u < 1) or x = 4 (2 - u) (1 <= u < 2); w(x) vanishes for x >= 2
__device__ __forceinline__ double ig_slope_core(double u, double &sign) {
  constexpr double ipi = KC<double>::ipi, pi4 = 4.0 * KC<double>::pi;
  double x;
  if (u < 1) {
    x = 4.0 * u;
    sign = 4.0;
  } else {
    x = 4.0 * (2.0 - u);
    sign = -4.0;
  }
  double wx;
  if (x < 1) wx = ipi * (1.0 - 1.5 * x * x + 0.75 * x * x * x);
  else if (x < 2) wx = ipi * 0.25 * (2.0 - x) * (2.0 - x) * (2.0 - x);
  else wx = 0.0;
  return pi4 * x * x * wx;
}

__device__ __forceinline__ double ig_digdh(double u) {
  if (!(u > 0) || !(u < 2)) return 0.0;
  double sign;
  const double d = ig_slope_core(u, sign);
  return sign * u * d;
}

__device__ __forceinline__ double ig_dig(double u, double iu) {
  if (!(u > 0) || !(u < 2)) return 0.0;
  double sign;
  const double d = ig_slope_core(u, sign);
  return sign * iu * d;
}

// (1/u) dW/du for hydro at u = r / h
__device__ __forceinline__ double kernel_dw(double u, double iu) {
  constexpr double ipi = KC<double>::ipi;
  if (u < 1) return ipi * (-3.0 + 2.25 * u);
  if (u < 2) {
    const double t = 2.0 - u;
    return -ipi * 0.75 * t * t * iu;
  }
  return 0.0;
}

// sum over the S lanes of a particle (every lane gets it)
template <int S>
__device__ __forceinline__ double sub_sum(double v) {
#pragma unroll
  for (int o = S / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int S>
__device__ __forceinline__ double sub_max(double v) {
#pragma unroll
  for (int o = S / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace sph
