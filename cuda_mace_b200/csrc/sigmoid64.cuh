// Logistic function in float64 for kernels whose elementwise phase is as long as their products; also compiled for the host,
// where its error is checked against the long double exponential.
#pragma once
#include <cstring>

#include "edge_math.cuh"

namespace cmace {

// 1 / d to 20 bits: the start of the reciprocal below
CMACE_HD double reciprocal_seed(double d) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  return y;
#else   // no better than the instruction: the quotient cut to 20 bits
  const double y = 1.0 / d;
  unsigned long long w;
  std::memcpy(&w, &y, 8);
  w &= ~((1ull << 33) - 1);
  double cut;
  std::memcpy(&cut, &w, 8);
  return cut;
#endif
}

// 1 / (1 + e^-z).  The elementwise phase has as many FP64 operations as the products if the library's exp and divide are
// used (the kernel took 1.26 ms at 8 000 atoms, 0.78 of them the products' own time), so: e^x by Tang's table-driven
// method (ACM TOMS 15, 1989): x = (32 m + j) ln2 / 32 + r with |r| <= ln2 / 64, e^x = 2^m 2^(j/32) (1 + p(r)); the
// remainder of the exponential series after r^6 is below 4e-18.  The reciprocal starts from the hardware's 20-bit
// approximation and one step of third order, 1/d = y (1 + e + e^2), e = 1 - d y: e^3 < 2^-57.
// |z| beyond 700 saturates the exponent (the result is 0 or 1 to 300 digits).  etab[j] = 2^(j/32).  Worst error found over
// |z| < 700: 3.5e-16 of the result.
CMACE_HD double table_sigmoid(double z, const double *etab) {
  const double x = fmin(fmax(-z, -700.0), 700.0);
  const double kd = fma(x, 46.16624130844683, 6755399441055744.0);   // 32 / ln 2; 1.5 * 2^52 rounds to an integer
#ifdef __CUDA_ARCH__
  const int k = __double2loint(kd);
#else
  long long bits;
  std::memcpy(&bits, &kd, 8);
  const int k = (int)bits;
#endif
  const double n = kd - 6755399441055744.0;
  double r = fma(n, -0.021660849391992087, x);                           // ln2 / 32 in two parts, the first 35 bits long
  r = fma(n, -5.062034433330175e-13, r);
  double p = fma(r, 1.0 / 720.0, 1.0 / 120.0);
  p = fma(p, r, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p, r * r, r);
  const double t = etab[k & 31];
  const double e0 = fma(t, p, t);
#ifdef __CUDA_ARCH__
  const double e = __hiloint2double(__double2hiint(e0) + ((k >> 5) << 20), __double2loint(e0));
#else
  std::memcpy(&bits, &e0, 8);
  bits += (long long)(k >> 5) * (1ll << 52);
  double e;
  std::memcpy(&e, &bits, 8);
#endif
  const double d = 1.0 + e, y = reciprocal_seed(d);
  const double c = fma(-d, y, 1.0);
  return fma(y, fma(c, c, c), y);
}

}  // namespace cmace
