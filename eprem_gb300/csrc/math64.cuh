// math64.cuh -- natural logarithm and exponential in double for the FP64 pipe,
// table-driven after Tang (exp: ACM TOMS 15 (1989) 144-157; log: ACM TOMS 16
// (1990) 378-400), with tables long enough that short polynomials do: 11 FP64
// operations each where CUDA's own take about 38 and 21 of the FP64 pipe's slots
// (measured on a GB300 against independent multiply-adds).  The tables are made
// on the host (math64_tables, run creation) and read through L1.
//   ln x:  x = 2^m z, c the inverse of the centre of z's 1/256 of [1, 2), r =
//          z c - 1, |r| < 2^-9: ln x = m ln 2 - ln c + r - r^2/2 + r^3/3 - r^4/4 +
//          r^5/5; m ln 2 - ln c is exact in its leading part (both on a grid of
//          2^-41) and adds its trailing part to the polynomial.
//   exp x: x = (256 m + j) ln 2 / 256 + r, |r| < 2^-9.5: 2^m 2^(j/256) (1 + r +
//          r^2/2 + r^3/6 + r^4/24 + r^5/120).
// Truncation is below 2^-56 in both (exp without its last term was off by up to
// 0.84 units in the last place).  Against 80-bit results over the normal range (6e7
// arguments) exp is within 0.503 units in the last place, ln within 0.54 where
// |ln x| > 1 and 7e-17 absolutely below, less than f's own rounding in exp(ln f +
// d).  Arguments outside the normal range go to log and exp.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

namespace eprem {

constexpr int kMath64Steps = 256;
// exp: {2^(j/256), what its rounding left}; log: {c, leading -ln c} pairs, then
// the trailing parts
constexpr int kMath64Size = 5 * kMath64Steps;
constexpr double kMath64Grid = 2199023255552.0;  // 2^41

inline std::vector<double> math64_tables() {
  std::vector<double> t(kMath64Size);
  for (int j = 0; j < kMath64Steps; j++) {
    const long double e = exp2l((long double)j / kMath64Steps);
    t[2 * j] = (double)e;
    t[2 * j + 1] = (double)(e - (long double)t[2 * j]);
    const double c = (double)(1.0L / (1.0L + (j + 0.5L) / kMath64Steps));
    const long double l = -logl((long double)c);
    const double hi = (double)(rintl(l * (long double)kMath64Grid) / (long double)kMath64Grid);
    t[2 * kMath64Steps + 2 * j] = c;
    t[2 * kMath64Steps + 2 * j + 1] = hi;
    t[4 * kMath64Steps + j] = (double)(l - (long double)hi);
  }
  return t;
}

// ln 2 on the grid and what is left of it.
constexpr double kLn2Hi = 1524246769572.0 / kMath64Grid;
constexpr double kLn2Lo = -1.7239444525614835e-13;

__device__ __forceinline__ double ln64(double x, const double *__restrict__ tab) {
  const int hi = __double2hiint(x);
  if ((unsigned)(hi - 0x00100000) >= 0x7fe00000u) return log(x);  // not a normal positive number
  const int m = (hi >> 20) - 1023, j = (hi >> 12) & 255;
  const double z = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(x));
  const double2 ch = __ldg(reinterpret_cast<const double2 *>(tab + 2 * kMath64Steps) + j);
  const double lo = __ldg(tab + 4 * kMath64Steps + j);
  // m as a double: 2^52 + 2^31 + m, exactly, less the constant
  const double md = __hiloint2double(0x43300000, m ^ (int)0x80000000) - 4503601774854144.0;
  const double r = fma(z, ch.x, -1.0);
  const double t = fma(md, kLn2Hi, ch.y);
  const double p = fma(r, fma(r, fma(r, 0.2, -0.25), 1.0 / 3.0), -0.5);
  return t + (r + fma(r * r, p, fma(md, kLn2Lo, lo)));
}

__device__ __forceinline__ double exp64(double x, const double *__restrict__ tab) {
  if (!(fabs(x) < 708.0)) return exp(x);
  const double t = fma(x, 369.329930467574632, 6755399441055744.0);
  const int n = __double2loint(t);
  const double k = t - 6755399441055744.0;
  constexpr double kStep = 0.6931471805599453 / 256.0, kStepLo = 2.3190468138462996e-17 / 256.0;
  const double r = fma(k, -kStepLo, fma(k, -kStep, x));
  const double2 T = __ldg(reinterpret_cast<const double2 *>(tab) + (n & 255));
  const double p = fma(r * r, fma(r, fma(r, fma(r, 1.0 / 120.0, 1.0 / 24.0), 1.0 / 6.0), 0.5), r);
  const double y = T.x + fma(T.x, p, T.y);
  return __hiloint2double(__double2hiint(y) + ((n >> 8) << 20), __double2loint(y));
}

}  // namespace eprem
