// Divisions by one divisor many times over: its reciprocal once, then five operations each, with the bits of
// a / b.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define SIH26_BOTH __host__ __device__ __forceinline__
#else
#define SIH26_BOTH inline
#endif

namespace sih26 {

// What quotient() takes beside b. NaN, which makes it divide, where b is too small or too large for its
// remainders to be exact.
SIH26_BOTH double quotient_reciprocal(double b) {
  const double rb = 1.0 / b;
  return b > 1e-40 && b < 1e40 ? rb : NAN;
}

// a / b for a positive b and rb = quotient_reciprocal(b). Two corrections of a * rb by the exact remainder give
// the correctly rounded quotient from a correctly rounded reciprocal (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990, theorem 8.2). A remainder is a multiple of the
// last places of q and b multiplied, 2^-104 |q b| or more, which a double holds while |q b| > 1e-290: with the
// bounds here and on b. Quotients beyond them are divided.
SIH26_BOTH double quotient(double a, double b, double rb) {
  double q = a * rb;
  q = std::fma(std::fma(-q, b, a), rb, q);
  q = std::fma(std::fma(-q, b, a), rb, q);
  const double mag = std::fabs(q);
  if (!(mag > 1e-250 && mag < 1e250)) q = a == 0.0 ? a : a / b;
  return q;
}

}  // namespace sih26
