// Host build of the uncertified quotients of volcano-ash3d_b200/csrc/
// exact_div.cuh (test infrastructure): quot_rn with a reciprocal estimate off
// by up to 2^-19 in the limiter's range |a| < 2|b|, and div_rn_3 over the
// reciprocal's three words, against the host's IEEE division (the sign of a
// zero quotient aside, which div_rn_3 does not keep).
// usage: quotients_host <pairs per case> <seed>; prints one line per case,
// "<func> <family> pairs <n> mismatches <m> refused <r>"
#include <math.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
static inline long long __double_as_longlong(double x) {
  long long u;
  std::memcpy(&u, &x, 8);
  return u;
}
static inline double __longlong_as_double(long long u) {
  double x;
  std::memcpy(&x, &u, 8);
  return x;
}
static inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
#define A3G_HOST_TEST
#include "../volcano-ash3d_b200/csrc/exact_div.cuh"

static std::mt19937_64 g_est(7);
double a3g::host_rcp_estimate(double b) {  // 20 leading bits, as the hardware's
  std::uniform_real_distribution<double> u(-0x1p-19, 0x1p-19);
  return 1.0 / b * (1.0 + u(g_est));
}
long &a3g::host_fallback_count() {
  static long n = 0;
  return n;
}

static double mantissa(std::mt19937_64 &r, int fam) {  // in [1, 2)
  uint64_t m = r() & 0x000fffffffffffffULL;
  if (fam == 1) m |= 0x000fffff00000000ULL & ~((r() & 3) << 32);                     // just below 2
  if (fam == 2) m = (r() & 1) ? (r() & 15) : (0x000fffffffffffffULL - (r() & 15));  // a few ulps from 1 or 2
  if (fam == 3) m &= 0x000ffff000000000ULL;                                          // short: exact quotients
  return __longlong_as_double((long long)(0x3ff0000000000000ULL | m));
}

int main(int argc, char **argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 200000;
  std::mt19937_64 r(argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1);
  const char *fams[] = {"any", "below_two", "edges", "short", "tails"};
  int bad_total = 0;
  for (int f = 0; f < 2; f++)
    for (int fam = 0; fam < 5; fam++) {
      long bad = 0, refused = 0;
      for (long t = 0; t < n; t++) {
        double b = mantissa(r, fam), a = mantissa(r, fam == 1 && (r() & 1) ? 0 : fam);
        if (r() & 1) a = -a;
        double q;
        if (f == 0) {  // limiter: |a| < 2|b|, either sign
          b = std::ldexp(b, (int)(r() % 420) - 210);
          a *= std::fabs(b) / 2.0 * (r() & 1 ? 1.0 : std::ldexp(1.0, -(int)(r() % (fam == 4 ? 700 : 40))));
          if (r() & 1) b = -b;
          if (!(std::fabs(a) < 2.0 * std::fabs(b))) continue;
          if (!a3g::quot_rn(a, b, &q)) {
            refused++;
            continue;
          }
        } else {  // pivots
          b = std::ldexp(b, (int)(r() % 8));
          a = std::ldexp(a, fam == 4 ? -(int)(r() % 1090) : (int)(r() % 200) - 100);
          if (!a3g::div_rn_3_covers(b) || !a3g::div_rn_3_takes(a)) {
            refused++;
            continue;
          }
          const double zh = 1.0 / b, e = fma(-b, zh, 1.0), zl = e / b, zll = fma(-b, zl, e) / b;
          q = a3g::div_rn_3(a, zh, zl, zll);
        }
        const double want = a / b;
        if (std::memcmp(&q, &want, 8) != 0 && !(q == 0.0 && want == 0.0)) {  // a zero's sign is not kept
          if (bad++ < 5) std::printf("MISMATCH %s a=%a b=%a got=%a want=%a\n", fams[fam], a, b, q, want);
        }
      }
      std::printf("%s %s pairs %ld mismatches %ld refused %ld\n", f ? "div_rn_3" : "quot_rn", fams[fam], n, bad,
                  refused);
      bad_total += bad != 0;
    }
  return bad_total ? 1 : 0;
}
