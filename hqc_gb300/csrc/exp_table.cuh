// exp(x) for -708 < x <= 0 (0 below) from a 64-entry table of 2^(j/64), after
// P. T. P. Tang, "Table-driven implementation of the exponential function in
// IEEE floating-point arithmetic", ACM Trans. Math. Softw. 15 (1989) 144-157:
// x = (64 m + j) ln2 / 64 + r, |r| <= ln2 / 128, exp(x) = 2^m 2^(j/64) e^r with
// the Taylor polynomial of e^r - 1 to r^5 (the next term is 4e-17).  Ten FP64
// instructions, for the kernels that the FP64 pipe bounds (2 multiply-adds a
// cycle and SM).  ln2 is split so that k ln2_hi is exact for |k| < 2^20.
#pragma once
#include <cmath>

namespace hqcgb {

constexpr int kExpTable = 64;

// The table's entries (host), to be copied into a kernel's shared memory.
inline void exp_table(double *t) {
  for (int j = 0; j < kExpTable; ++j) t[j] = std::exp2(j / 64.0);
}

constexpr double kExpMagic = 6755399441055744.0;  // 1.5 * 2^52: the sum's low word is the rounded integer
constexpr double kExpInv = kExpTable / 0.693147180559945309417;
constexpr double kExpHi = 0x1.62e42feep-1 / kExpTable, kExpLo = 0x1.a39ef35793c76p-33 / kExpTable;

// 2^(k/64) e^r
__device__ inline double exp_reduced(int k, double r, const double *__restrict__ tab) {
  double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
  q = fma(q, r, 1.0 / 6.0);
  q = fma(q, r, 0.5);
  const double p = fma(q, r * r, r);
  const double T = tab[k & (kExpTable - 1)];
  const double s = __hiloint2double(__double2hiint(T) + ((k >> 6) << 20), __double2loint(T));
  return fma(s, p, s);
}

__device__ inline double exp_neg(double x, const double *__restrict__ tab) {
  const double t = fma(x, kExpInv, kExpMagic);
  const double kd = t - kExpMagic;
  double r = fma(kd, -kExpHi, x);
  r = fma(kd, -kExpLo, r);
  const double v = exp_reduced(__double2loint(t), r, tab);
  return x > -708.0 ? v : (x != x ? x : 0.0);
}

// exp(-al y), c = al kExpInv: the product enters the reduction unrounded (rounded, an
// exponent of 41 costs up to 20 eps).
__device__ inline double exp_neg_product(double al, double c, double y, const double *__restrict__ tab) {
  const double t = fma(y, -c, kExpMagic);
  const double kd = t - kExpMagic;
  double r = fma(-al, y, -(kd * kExpHi));
  r = fma(kd, -kExpLo, r);
  const double v = exp_reduced(__double2loint(t), r, tab);
  return kd > -708.0 * kExpInv ? v : (kd != kd ? kd : 0.0);
}

}  // namespace hqcgb
