// divby.cuh -- correctly rounded quotients by a divisor whose reciprocal is at
// hand (neighbours.cu); plain C++ as well, so that it can be tested on the CPU.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define SPH_DIVBY_FN __host__ __device__ __forceinline__
#else
#define SPH_DIVBY_FN inline
#endif

namespace sph {

// a / b rounded to nearest, y = 1 / b rounded to nearest: Markstein's method
// (Computation of elementary functions on the IBM RISC System/6000, 1990).
// The first correction brings q within an ulp, the second then rounds
// correctly, as long as nothing is denormal: b, y and the quotient are normal
// numbers, and a is 0 or at least 1e-290 in magnitude (the remainders are 2^-53
// of it).
SPH_DIVBY_FN double div_by(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-b, q, a), y, q);
  return fma(fma(-b, q, a), y, q);
}

}  // namespace sph
