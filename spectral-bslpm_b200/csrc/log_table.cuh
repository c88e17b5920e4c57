// The natural logarithm of the Poisson sums, by table.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "geometry.cuh"

namespace sbslpm {

// log(a) of a positive normal a by table (P. T. P. Tang, "Table-driven
// implementation of the logarithm function in IEEE floating-point
// arithmetic", ACM TOMS 16, 1990): a = 2^k m with m in [0.6875, 1.375), the
// interval of m gives c close to 1/m, r = m c - 1 is exact in one fused
// multiply-add up to its rounding, and log a = k log 2 - log c + log(1 + r)
// with |r| <= 2^-7 and the series of log(1 + r) to r^8.  The reduction -- the
// high word less that of the interval's start, whose exponent bits are k and
// whose next bits the interval's number -- is arranged as that of log in Arm's
// Optimized Routines; the table's entries, their two parts and the series are
// this file's.  log c and log 2 are held in two parts, the high ones short
// enough that k log 2 - log c is exact; c = 1 on both sides of 1.
//
// Error: 2^-53 relative from the final rounding and, outside the two intervals
// of c = 1, 2^-54 from that of r (below 1 |r| <= 2^-9 and |log a| >= 2^-8,
// above 2^-8 and 2^-7); all other roundings are of terms of order r^2.  Against
// long double over [2^-51, 2], powers of two and near 1 (2.8 million values):
// rms 4.7e-17 as CUDA's log, at most 1.3e-16 (log: 1.1e-16), far below that of
// its argument 1 - x.y (1e-16 absolute); 6.4e11 against 3.3e11 per second.
constexpr int kLogBits = 7, kLogN = 1 << kLogBits, kLogFirst = 0x3fe60000;  // the high word of 0.6875
constexpr double kLn2Hi = 0x1.62e42fefap-1, kLn2Lo = 0x1.cf79abc9e3b3ap-40;

// Words of a double, and a double of given words.
SB_HD int high_word(double a) {
#ifdef __CUDA_ARCH__
  return __double2hiint(a);
#else
  unsigned long long u;
  std::memcpy(&u, &a, sizeof u);
  return (int)(u >> 32);
#endif
}

SB_HD double with_high_word(double a, int hi) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(hi, __double2loint(a));
#else
  unsigned long long u;
  std::memcpy(&u, &a, sizeof u);
  u = ((unsigned long long)(unsigned)hi << 32) | (u & 0xffffffffu);
  std::memcpy(&a, &u, sizeof a);
  return a;
#endif
}

SB_HD double table_log(double a, const double2* cv, const double* lo) {
  const int hi = high_word(a), t = hi - kLogFirst, k = t >> 20, i = (t >> (20 - kLogBits)) & (kLogN - 1);
  const double m = with_high_word(a, hi - k * (1 << 20));
  const double2 c = cv[i];
  const double r = fma(m, c.x, -1.0);
  const double kd = (double)k;
  double p = fma(r, -1.0 / 8, 1.0 / 7);
  p = fma(r, p, -1.0 / 6);
  p = fma(r, p, 1.0 / 5);
  p = fma(r, p, -1.0 / 4);
  p = fma(r, p, 1.0 / 3);
  p = fma(r, p, -1.0 / 2);
  const double tail = fma(r * r, p, fma(kd, kLn2Lo, lo[i]));
  const double big = fma(kd, kLn2Hi, c.y), sum = big + r;  // |big| > |r| or big = 0: the remainder is exact
  return sum + ((r - (sum - big)) + tail);
}

// [kLogN] (c, high part of -log c), then [kLogN] its low part.
inline std::vector<double> log_table() {
  std::vector<double> t(3 * kLogN);
  auto edge = [](int i) { return with_high_word(0.0, kLogFirst + (i << (20 - kLogBits))); };
  for (int i = 0; i < kLogN; i++) {
    const double a = edge(i), b = edge(i + 1);
    const double c = a == 1.0 || b == 1.0 ? 1.0 : 2.0 / (a + b);
    const long double v = -std::log((long double)c);
    const double hi = (double)(std::nearbyint(v * 0x1p40L) * 0x1p-40L);  // k log 2's high part ends at 2^-40 as well
    t[2 * i] = c;
    t[2 * i + 1] = hi;
    t[2 * kLogN + i] = (double)(v - hi);
  }
  return t;
}

}  // namespace sbslpm
