// div_dev.h -- correctly rounded FP64 quotients by divisors whose reciprocal
// is known: the bits of the division in a handful of multiply-adds.
#ifndef PIC_DIV_DEV_H
#define PIC_DIV_DEV_H

namespace pic {

// a / d with y = 1/d rounded to nearest (NaN where d is out of the range in
// which this holds), the same bits as the division: a correction of a y makes
// it the quotient to within its last place, and by Markstein's theorem (IBM
// J. Res. Dev. 34, 1990) one more with the exact remainder rounds correctly.
// Five dependent operations and no branch; zeros keep their sign.  exact is
// cleared where the caller has to divide.
__device__ __forceinline__ double div_const(double a, double d, double y, bool &exact) {
  double q = a * y;
  const double zero = q;
  q = fma(fma(-q, d, a), y, q);
  q = fma(fma(-q, d, a), y, q);
  const double m = fabs(a);
  exact = exact && y == y && ((m > 1e-250 && m < 1e250) || m == 0.0);
  return m == 0.0 ? zero : q;
}

__device__ __forceinline__ double recip_const(double d) {
  const double m = fabs(d);
  return m > 1e-40 && m < 1e40 ? 1.0 / d : __longlong_as_double(0x7ff8000000000000ll);
}

// 1/d rounded to nearest, from y0 = 1/d0 of a divisor d0 that d equals to
// about 1e-9 (NaN stays NaN): one Newton step brings it to within its last
// place, and the next rounds correctly (Markstein's theorem for reciprocals).
// The theorem leaves out a significand of all ones, where y can stay a place
// low and the quotient of a power of two with it: NaN there, so the caller divides.
__device__ __forceinline__ double recip_near(double d, double y0) {
  const long long ones = (1ll << 52) - 1;
  double y = fma(fma(-d, y0, 1.0), y0, y0);
  y = fma(fma(-d, y, 1.0), y, y);
  return (__double_as_longlong(d) & ones) == ones ? __longlong_as_double(0x7ff8000000000000ll) : y;
}

}  // namespace pic

#endif
