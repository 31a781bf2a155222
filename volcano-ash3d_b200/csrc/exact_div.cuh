// exact_div.cuh -- correctly rounded double division without a branchy
// library call in the common case.
//
// The transport path needs quotients that are bit-identical to IEEE division
// (the limiter's theta = dqu/dq, src/AdvectionHorz_DCU.f90:204, and the back
// substitution of the tridiagonal solve).  Method: Goldschmidt's iteration
// (R. E. Goldschmidt, "Applications of division by convergence", MIT thesis
// 1964) for the quotient, then Markstein's correction step (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. R&D 1990; Muller et al., Handbook of Floating-Point
// Arithmetic, ch. 5):
//   y  ~ 1/b from the hardware reciprocal approximation (PTX
//        rcp.approx.ftz.f64), e = 1 - b*y (exact with an FMA);
//   q  = a*y*(1 + e)*(1 + e^2): relative error e^4, the two products and
//        y' = y*(1 + e) formed side by side, so the dependent chain after
//        the estimate is five operations instead of the seven of two
//        sequential Newton-Raphson steps on y;
//   r  = a - b*q (exact with an FMA);  q = q + r*y'.
// The result is then certified exactly: r = a - b*q is computed again with an
// FMA, and q is accepted only if |r| < |b| * ulp(q)/2, i.e. the true quotient
// lies strictly inside the rounding interval of q, and q is not a power of two
// (whose rounding interval is asymmetric).  Everything else -- operands
// outside the fast ranges below, a zero divisor, non-finite values, a residual
// on or beyond the half-ulp bound -- falls back to the IEEE division operator.
// A zero dividend over an in-range divisor returns a*b, the zero whose sign
// IEEE division gives (the signs' exclusive or).  Every path therefore
// returns RN(a/b) exactly.
//
// The fast ranges keep every intermediate normal and the residual exact.
// With q within an ulp or two of a/b, r = a - b*q is a multiple of
// ulp(b)*ulp(q) = 2^(e_b+e_q-104) smaller than |b|*ulp(q) < 2^(e_b+e_q-51), so
// it is a double whenever 2^(e_b+e_q-104) >= 2^-1074, i.e. e_a (which is
// e_b+e_q or one more) >= -969; ulp(q)/2 = 2^(e_q-53) must be normal
// (e_q >= -969), and nothing may overflow.  Both ranges below give e_a and
// e_q in [-951, 951]:
//   div_rn:     |b| in [2^-200, 2^201), |a| in [2^-700, 2^701) or a = 0
//               (the limiter's theta = dqu/dq divides only when |dq| >= the
//               cycle threshold, 1e-10 in the reference);
//   div_rn_rcp: |b| in [2^-50, 2^51), |a| in [2^-900, 2^901) or a = 0
//               (the back substitution's pivots D' are >= 1 on the
//               diagonally dominant Crank-Nicolson matrices, and its
//               dividends run down the diffused tails of a cloud).
#pragma once

namespace a3g {

// The IEEE division operator for the rare operands the fast path does not
// certify, kept out of line so that its code is not repeated at every call
// site (the sweeps inline many divisions).  A translation unit that measured
// faster with it inlined defines A3G_DIV_FALLBACK_INLINE first.
#if defined(A3G_HOST_TEST)
// A host build of this header (the CPU test of the certification) supplies
// its own reciprocal estimates, including deliberately poor ones, and counts
// the quotients that were not certified.
double host_rcp_estimate(double b);
long &host_fallback_count();
static inline double ieee_div(double a, double b) {
  ++host_fallback_count();
  return a / b;
}
#elif defined(A3G_DIV_FALLBACK_INLINE)
static __device__ __forceinline__ double ieee_div(double a, double b) { return a / b; }
#else
static __device__ __noinline__ double ieee_div(double a, double b) { return a / b; }
#endif

__device__ __forceinline__ double rcp_approx(double b) {
#ifdef A3G_HOST_TEST
  return host_rcp_estimate(b);
#else
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
#endif
}

// True when the binary exponent of x lies in [LO, HI] (or x is zero and
// ALLOW_ZERO).
template <int LO, int HI, bool ALLOW_ZERO>
__device__ __forceinline__ bool exp_in(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  return (e - (unsigned)(1023 + LO)) <= (unsigned)(HI - LO) || (ALLOW_ZERO && x == 0.0);
}

// Certifies q against a/b (see above); returns true if q == RN(a/b).
__device__ __forceinline__ bool certified(double a, double b, double q) {
  const double r = fma(-b, q, a);
  const long long qb = __double_as_longlong(q);
  const long long ex = qb & 0x7ff0000000000000LL;
  const double half_ulp = __longlong_as_double(ex - (53LL << 52));  // 2^(e_q - 53)
  const bool pow2 = (qb & 0x000fffffffffffffLL) == 0;
  return fabs(r) < fabs(b) * half_ulp && !pow2;
}

// RN(a/b).
__device__ __forceinline__ double div_rn(double a, double b) {
  if (!(exp_in<-200, 200, false>(b) && exp_in<-700, 700, true>(a))) return ieee_div(a, b);
  if (a == 0.0) return a * b;  // +-0 with the quotient's sign (b finite, nonzero)
  double y = rcp_approx(b);
  const double e = fma(-b, y, 1.0);
  double q = a * y;
  const double e2 = e * e;
  q = fma(q, e, q);
  y = fma(y, e, y);
  q = fma(q, e2, q);
  const double r = fma(-b, q, a);
  q = fma(r, y, q);
  if (certified(a, b, q)) return q;
  return ieee_div(a, b);
}

// RN(a/b) given y = RN(1/b) (precomputed once for a divisor shared by many
// quotients, e.g. a tridiagonal pivot).
__device__ __forceinline__ double div_rn_rcp(double a, double b, double y) {
  if (!(exp_in<-50, 50, false>(b) && exp_in<-900, 900, true>(a))) return ieee_div(a, b);
  if (a == 0.0) return a * b;  // +-0 with the quotient's sign (b finite, nonzero)
  double q = a * y;
  const double r = fma(-b, q, a);
  q = fma(r, y, q);
  if (certified(a, b, q)) return q;
  return ieee_div(a, b);
}

// RN(a/b) without a certificate, for |a| < 2|b|: returns true with the
// quotient in *q, or false (*q unspecified) when the caller has to divide
// with the operator.  Markstein's method with two residual steps:
//   y0 ~ 1/b with |1 - b*y0| < 2^-19; two Newton-Raphson steps give y within
//   (1/2 + 2^-23) ulp of 1/b;
//   q0 = a*y;  q1 = q0 + (a - b*q0)*y  is within (1/2 + 2^-50) ulp of a/b;
//   r = a - b*q1 is exact, and q = RN(q1 + r*y).
// Scaled to 1 <= b < 2, the last sum misses a/b by |a/b - q1|*|b*y - 1| <=
// (1/2 + 2^-50)(1/2 + 2^-23) b 2^-53 ulp(q), while a/b keeps at least 2^-53/b
// ulp(q) from every midpoint m of two doubles (a - b*m is a nonzero multiple
// of 2^-53 ulp(q)): q = RN(a/b) whenever b < 2(1 - 2^-22).  Divisors whose
// leading 20 mantissa bits are all ones are refused; the estimate's error is
// at most 2^-19.93 over all leading 20-bit mantissas (measured on B200:
// a3g_selftest_quotients, which a test holds below 2^-19).  |a| >= 2^-700 and 2^-200 <= |b| < 2^201 keep every
// intermediate normal and the residual exact (see above); a zero dividend is
// refused.
__device__ __forceinline__ bool quot_rn(double a, double b, double *q) {
  const unsigned ha = (unsigned)__double2hiint(a) & 0x7fffffffu, hb = (unsigned)__double2hiint(b) & 0x7fffffffu;
  constexpr unsigned ALO = (1023u - 700u) << 20, BLO = (1023u - 200u) << 20, BHI = (1023u + 201u) << 20;
  double y = rcp_approx(b);
  double e = fma(-b, y, 1.0);
  y = fma(y, e, y);
  e = fma(-b, y, 1.0);
  y = fma(y, e, y);
  double v = a * y;
  double r = fma(-b, v, a);
  v = fma(r, y, v);
  r = fma(-b, v, a);
  *q = fma(r, y, v);
  return ha >= ALO && (hb - BLO) < (BHI - BLO) && (hb & 0xfffffu) != 0xfffffu;
}

// RN(a/b) from 1/b = zh + zl + zll (zh = RN(1/b), zl = RN(1/b - zh), zll =
// RN(1/b - zh - zl)) in three dependent operations and no test of the result:
// q = RN(a*zh + RN(a*zl + RN(a*zll))).  The idea of multiplying by a reciprocal
// in more than one word is N. Brisebarre, J.-M. Muller and S. K. Raina,
// "Accelerating correctly rounded floating-point division when the divisor is
// known in advance" (IEEE Trans. Computers 53, 2004); the third word removes
// their exceptional divisors.  Scaled to 1 <= a, b < 2: |zl| <= 2^-54, so the
// correction is below 2^-53 and its rounding error at most 2^-107 (+ 2^-158 for
// the rest), while a/b keeps 2^-106/b > 2^-107 from every midpoint of two
// doubles (2^-105/b when a >= b): the last rounding gives RN(a/b).  Divisors
// within 2^-20 of twice a power of two, where the margin closes, and those
// outside [2^-50, 2^51) are not covered (div_rn_3_covers).  The dividend has
// to be in [2^-900, 2^901) or zero (div_rn_3_takes); a zero quotient's sign is
// not kept.
__device__ __forceinline__ double div_rn_3(double a, double zh, double zl, double zll) {
  return fma(a, zh, fma(a, zl, a * zll));
}
__device__ __forceinline__ bool div_rn_3_covers(double b) {
  return exp_in<-50, 50, false>(b) && ((unsigned)__double2hiint(b) & 0xfffffu) != 0xfffffu;
}
__device__ __forceinline__ bool div_rn_3_takes(double a) {
  const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
  constexpr unsigned LO = (1023u - 900u) << 20, HI = (1023u + 901u) << 20;
  return h - LO < HI - LO || (h | (unsigned)__double_as_longlong(a)) == 0u;
}

}  // namespace a3g
