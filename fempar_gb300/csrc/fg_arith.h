// fg_arith.h -- small arithmetic that kernels rely on to the last bit, compiled for the device and for
// the host (where the tests check it against exact arithmetic).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define FG_HD __host__ __device__ __forceinline__
#else
#define FG_HD inline
#endif

namespace fg {

// s / d from the correctly rounded reciprocal r of d: the quotient with one correction step
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J.
// Res. Dev. 34, 1990), in three operations where many values are divided by the same d.  It has the
// rounding of a division where quotient_exact holds.
FG_HD double quotient(double s, double d, double r) {
  const double q = s * r;
  return ::fma(::fma(-q, d, s), r, q);
}
FG_HD float quotient(float s, float d, float r) {
  const float q = s * r;
  return ::fmaf(::fmaf(-q, d, s), r, q);
}

// q = quotient(s, d, 1 / d) is s / d to the last bit: d, its reciprocal and q are normal numbers, and the
// remainder s - q d is a normal number's multiple of their last places (exact).  Also where q is 0
// (s is 0, or s / d at most the smallest subnormal).  False for infinities and NaN.
FG_HD bool quotient_exact(double q, double d) {
  uint64_t bq, bd;
  memcpy(&bq, &q, 8);
  memcpy(&bd, &d, 8);
  const int eq = (int)((bq >> 52) & 0x7FF) - 1023, ed = (int)((bd >> 52) & 0x7FF) - 1023;
  return (bq << 1) == 0 ? ed <= 1020 : (unsigned)(eq + 1020) <= 2042u && (unsigned)(ed + 1020) <= 2040u &&
                                           (unsigned)(eq + ed + 960) <= 1980u;
}
FG_HD bool quotient_exact(float q, float d) {
  uint32_t bq, bd;
  memcpy(&bq, &q, 4);
  memcpy(&bd, &d, 4);
  const int eq = (int)((bq >> 23) & 0xFF) - 127, ed = (int)((bd >> 23) & 0xFF) - 127;
  return (bq << 1) == 0 ? ed <= 125 : (unsigned)(eq + 124) <= 250u && (unsigned)(ed + 125) <= 250u &&
                                          (unsigned)(eq + ed + 100) <= 225u;
}

// s + e = a + b exactly (Knuth's TwoSum)
FG_HD void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Sum of FP32 pairs hi + lo (|lo| at most a few last places of hi) in three FP32 words: the first two by
// exact sums, their errors in the third, so what is lost is ~2^-70 of the sum of magnitudes, less than
// FP64 additions lose, on the FP32 pipe.
struct Sum3 {
  float h = 0.f, m = 0.f, l = 0.f;
  FG_HD void add(float h2, float m2, float l2) {
    float e, t, e2, e3;
    two_sum(h, h2, h, e);
    two_sum(m, m2, t, e2);
    two_sum(t, e, m, e3);
    l += l2 + (e2 + e3);
  }
  FG_HD double value() const { return ((double)m + (double)l) + (double)h; }
};

}  // namespace fg
