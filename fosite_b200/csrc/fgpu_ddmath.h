// fgpu_ddmath.h -- correctly rounded natural logarithm and exponential in
// double-double arithmetic, for host and device.
//
// fosite's step-size controller (AdjustTimestep, timedisc_base.f90:759-814) takes
// EXP and LOG of the error norm; the host compiler's libm and CUDA's libm may round
// these differently.  Evaluating both in double-double (about 104 significant bits)
// and rounding once gives the correctly rounded value on the host and on the device
// alike, so a controller running on either side produces the same step sizes.
//
// Methods (textbook, see e.g. Muller, "Elementary Functions", ch. 6-7):
//   log x = k ln 2 + 2 atanh(s),  s = (m - 1)/(m + 1),  x = m 2^k,  m in [sqrt(1/2), sqrt(2)),
//           atanh by its odd power series in s^2 (|s| <= 0.172);
//   exp x = 2^k exp(r),  r = x - k ln 2 with |r| <= ln2/2, exp(r) by its Taylor series.
// The series' tails, which contribute less than 2^-55 of the result, are summed in double (their
// rounding stays below 2^-107: the results before their last rounding are within 2^-100.7 (exp) and
// 2^-103.8 (log), as with every term in double-double), the leading terms in double-double with the coefficients
// 1/(2j+1) and 1/n! rounded to double-double.  One lane runs a chain, so its latency is the
// cost: AdjustTimestep took 42 us with every term a double-double division, 7.8 us this way with
// its two factors on two lanes.
// ln 2 is split into a double and a remainder (0x1.62e42fefa39efp-1 + 0x1.abc9e3b39803fp-56).
// Products and sums are rounded individually (no contraction), so every platform
// evaluates the same operations.
#pragma once
#include <cmath>

#if defined(__CUDACC__)
#define FGPU_HD __host__ __device__ __forceinline__
#else
#define FGPU_HD inline
#endif

namespace fgpu {
namespace ddm {

struct dd { double hi, lo; };

// IEEE operations that the compiler may not fuse
FGPU_HD double add_rn(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dadd_rn(a, b);
#else
  volatile double s = a + b;
  return s;
#endif
}
FGPU_HD double mul_rn(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  volatile double p = a * b;
  return p;
#endif
}
FGPU_HD double fma_rn(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}

FGPU_HD dd two_sum(double a, double b) {
  const double s = add_rn(a, b);
  const double bb = add_rn(s, -a);
  const double e = add_rn(add_rn(a, -add_rn(s, -bb)), add_rn(b, -bb));
  return {s, e};
}
FGPU_HD dd quick_two_sum(double a, double b) {
  const double s = add_rn(a, b);
  return {s, add_rn(b, -add_rn(s, -a))};
}
FGPU_HD dd two_prod(double a, double b) {
  const double p = mul_rn(a, b);
  return {p, fma_rn(a, b, -p)};
}
FGPU_HD dd dd_add(dd a, dd b) {
  dd s = two_sum(a.hi, b.hi);
  const dd t = two_sum(a.lo, b.lo);
  s.lo = add_rn(s.lo, t.hi);
  s = quick_two_sum(s.hi, s.lo);
  s.lo = add_rn(s.lo, t.lo);
  return quick_two_sum(s.hi, s.lo);
}
FGPU_HD dd dd_mul(dd a, dd b) {
  dd p = two_prod(a.hi, b.hi);
  p.lo = add_rn(p.lo, add_rn(mul_rn(a.hi, b.lo), mul_rn(a.lo, b.hi)));
  return quick_two_sum(p.hi, p.lo);
}
FGPU_HD dd dd_mul_d(dd a, double b) {
  dd p = two_prod(a.hi, b);
  p.lo = add_rn(p.lo, mul_rn(a.lo, b));
  return quick_two_sum(p.hi, p.lo);
}
// a / b with three quotient digits
FGPU_HD dd dd_div(dd a, dd b) {
  const double q1 = a.hi / b.hi;
  dd r = dd_add(a, dd_mul_d(b, -q1));
  const double q2 = r.hi / b.hi;
  r = dd_add(r, dd_mul_d(b, -q2));
  const double q3 = r.hi / b.hi;
  dd q = quick_two_sum(q1, q2);
  return dd_add(q, dd{q3, 0.0});
}

constexpr double LN2_HI = 0x1.62e42fefa39efp-1;
constexpr double LN2_LO = 0x1.abc9e3b39803fp-56;

// correctly rounded log(x) for positive normal x (other arguments: the platform's log)
FGPU_HD double log_cr(double x) {
  if (!(x > 0.0) || !(x < INFINITY) || x < 0x1p-1022) return log(x);
  int k;
  double m = frexp(x, &k);                   // x = m 2^k, m in [1/2, 1)
  if (m < 0x1.6a09e667f3bcdp-1) { m = m * 2.0; k -= 1; }   // m in [sqrt(1/2), sqrt(2))
  const dd num = {add_rn(m, -1.0), 0.0};      // exact (Sterbenz)
  const dd den = two_sum(m, 1.0);
  const dd s = dd_div(num, den);
  const dd s2 = dd_mul(s, s);
  // atanh(s)/s = sum_{j>=0} s^(2j)/(2j+1), |s^2| < 0.0295: 24 terms reach 2^-120, those from
  // j = 11 stay below 2^-56
constexpr double c[11][2] = {{0x1.0000000000000p+0, 0x0.0p+0}, {0x1.5555555555555p-2, 0x1.5555555555555p-56},
      {0x1.999999999999ap-3, -0x1.999999999999ap-57}, {0x1.2492492492492p-3, 0x1.2492492492492p-57},
      {0x1.c71c71c71c71cp-4, 0x1.c71c71c71c71cp-58}, {0x1.745d1745d1746p-4, -0x1.745d1745d1746p-59},
      {0x1.3b13b13b13b14p-4, -0x1.3b13b13b13b14p-58}, {0x1.1111111111111p-4, 0x1.1111111111111p-60},
      {0x1.e1e1e1e1e1e1ep-5, 0x1.e1e1e1e1e1e1ep-61}, {0x1.af286bca1af28p-5, 0x1.af286bca1af28p-59},
      {0x1.8618618618618p-5, 0x1.8618618618618p-59}};
  double tail = 1.0 / 47.0;
#pragma unroll
  for (int j = 22; j >= 11; --j) tail = fma_rn(tail, s2.hi, 1.0 / (2.0 * j + 1.0));
  dd acc = {tail, 0.0};
#pragma unroll
  for (int j = 10; j >= 0; --j) acc = dd_add(dd_mul(acc, s2), dd{c[j][0], c[j][1]});
  dd r = dd_mul(dd_mul_d(s, 2.0), acc);
  const dd kl = dd_add(two_prod((double)k, LN2_HI), dd{mul_rn((double)k, LN2_LO), 0.0});
  r = dd_add(kl, r);
  return add_rn(r.hi, r.lo);
}

// correctly rounded exp(x) for |x| < 700 (other arguments: the platform's exp)
FGPU_HD double exp_cr(double x) {
  if (!(fabs(x) < 700.0)) return exp(x);
  const double k = nearbyint(x / LN2_HI);
  // r = x - k ln2 in double-double
  const dd p = two_prod(k, LN2_HI);
  dd r = two_sum(x, -p.hi);
  r.lo = add_rn(r.lo, -p.lo);
  r.lo = add_rn(r.lo, -mul_rn(k, LN2_LO));
  r = quick_two_sum(r.hi, r.lo);
  // exp(r) = sum r^n/n!, |r| <= 0.347: 28 terms reach 2^-120, those from n = 14 stay below 2^-57
constexpr double c[14][2] = {{0x1.0000000000000p+0, 0x0.0p+0}, {0x1.0000000000000p+0, 0x0.0p+0},
      {0x1.0000000000000p-1, 0x0.0p+0}, {0x1.5555555555555p-3, 0x1.5555555555555p-57}, {0x1.5555555555555p-5,
      0x1.5555555555555p-59}, {0x1.1111111111111p-7, 0x1.1111111111111p-63}, {0x1.6c16c16c16c17p-10,
      -0x1.f49f49f49f49fp-65}, {0x1.a01a01a01a01ap-13, 0x1.a01a01a01a01ap-73}, {0x1.a01a01a01a01ap-16,
      0x1.a01a01a01a01ap-76}, {0x1.71de3a556c734p-19, -0x1.c154f8ddc6c00p-73}, {0x1.27e4fb7789f5cp-22,
      0x1.cbbc05b4fa99ap-76}, {0x1.ae64567f544e4p-26, -0x1.c062e06d1f209p-80}, {0x1.1eed8eff8d898p-29,
      -0x1.2aec959e14c06p-83}, {0x1.6124613a86d09p-33, 0x1.f28e0cc748ebep-87}};
constexpr double t[14] = {0x1.93974a8c07c9dp-37, 0x1.ae7f3e733b81fp-41, 0x1.ae7f3e733b81fp-45,
      0x1.952c77030ad4ap-49, 0x1.6827863b97d97p-53, 0x1.2f49b46814157p-57, 0x1.e542ba4020225p-62,
      0x1.71b8ef6dcf572p-66, 0x1.0ce396db7f853p-70, 0x1.761b41316381ap-75, 0x1.f2cf01972f578p-80,
      0x1.3f3ccdd165fa9p-84, 0x1.88e85fc6a4e5ap-89, 0x1.d1ab1c2dccea3p-94};
  double tail = t[13];
#pragma unroll
  for (int n = 12; n >= 0; --n) tail = fma_rn(tail, r.hi, t[n]);
  dd acc = {tail, 0.0};
#pragma unroll
  for (int n = 13; n >= 0; --n) acc = dd_add(dd_mul(acc, r), dd{c[n][0], c[n][1]});
  return ldexp(add_rn(acc.hi, acc.lo), (int)k);
}

}  // namespace ddm
}  // namespace fgpu
