// Host build of volcano-ash3d_b200/csrc/lim_coef.cuh (test infrastructure)
// against the oracle's orc_lim_coef, which divides: the same a and b (a NaN for a
// NaN) for every limiter, over general operands, short mantissas (ratios on
// the class bounds), operands an ulp off a bound, subnormals and tails, huge
// operands, infinities and NaN, and differences below EPS_THRESH (NOCYCLE).
// usage: lim_coef_host <pairs per case>; prints "<limiter> <family> mismatches <m>"
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
#include "../include/ash3d_b200.h"
#include "../volcano-ash3d_b200/csrc/exact_div.cuh"
double a3g::host_rcp_estimate(double b) { return 1.0 / b * (1.0 + 0x1p-20); }
long &a3g::host_fallback_count() {
  static long n = 0;
  return n;
}
namespace a3g {
static inline double fmx(double a, double b) { return a > b ? a : b; }
static inline double fmn(double a, double b) { return a < b ? a : b; }
}  // namespace a3g
#include "../volcano-ash3d_b200/csrc/lim_coef.cuh"

extern "C" void orc_lim_coef(int lim, double dq, double dqu, double eps, double *a, double *b);

static const double EPS = 1.0e-10;
static bool same(double x, double y) { return x == y || (x != x && y != y); }

template <int LIM>
static int run(const char *name, long n) {
  const char *fams[] = {"any", "short", "ulps", "tails", "huge", "nonfinite", "small"};
  int bad_total = 0;
  std::mt19937_64 r(11 + LIM);
  auto unit = [&]() { return 1.0 + (double)(r() >> 11) * 0x1p-53; };
  auto any = [&](int lo, int hi) { return std::ldexp(unit(), lo + (int)(r() % (uint64_t)(hi - lo + 1))); };
  const double odd[] = {INFINITY, NAN, 0.0, 1.0, 0x1p-1074, 0x1p1023, 3.0, 1.0e-5};
  for (int fam = 0; fam < 7; fam++) {
    long bad = 0;
    for (long t = 0; t < n; t++) {
      double dq, dqu;
      if (fam == 0) {
        dq = any(-30, 30);
        dqu = dq * any(-4, 3);
      } else if (fam == 1) {
        dq = std::ldexp((double)(1 + r() % 16), (int)(r() % 20) - 10);
        dqu = std::ldexp((double)(r() % 33), (int)(r() % 20) - 10);
      } else if (fam == 2) {
        dq = any(-30, 30);
        dqu = std::ldexp(dq, (int)(r() % 4) - 1);
        for (int k = (int)(r() % 3); k > 0; k--) dqu = std::nextafter(dqu, (r() & 1) ? INFINITY : 0.0);
      } else if (fam == 3) {
        dq = any(-30, 299);
        dqu = any(-1074, -600);
      } else if (fam == 4) {
        dq = any(250, 1023);
        dqu = any(-100, 1023);
      } else if (fam == 5) {
        dq = (r() & 1) ? odd[r() % 8] : any(-1000, 1000);
        dqu = odd[r() % 8];
      } else {
        dq = any(-1074, -34);  // below EPS_THRESH
        dqu = (r() % 8) ? any(-1074, 10) : 0.0;
      }
      if (r() & 1) dq = -dq;
      if (r() & 1) dqu = -dqu;
      // the sign of 3 from a NaN product is the machine's
      if ((dq != dq || dqu != dqu) && std::fabs(dq) < EPS) continue;
      double a, b, ra, rb;
      a3g::lim_coef<LIM>(dq, dqu, EPS, a, b);
      orc_lim_coef(LIM, dq, dqu, EPS, &ra, &rb);
      if (!(same(a, ra) && same(b, rb)) && bad++ < 3)
        std::printf("MISMATCH %s %s dq=%a dqu=%a got (%g, %g) want (%g, %g)\n", name, fams[fam], dq, dqu, a, b, ra, rb);
    }
    std::printf("%s %s mismatches %ld\n", name, fams[fam], bad);
    bad_total += bad != 0;
  }
  return bad_total;
}

int main(int argc, char **argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 200000;
  int bad = 0;
  bad += run<A3G_LIM_LAXWEN>("laxwen", n);
  bad += run<A3G_LIM_BW>("bw", n);
  bad += run<A3G_LIM_FROMM>("fromm", n);
  bad += run<A3G_LIM_MINMOD>("minmod", n);
  bad += run<A3G_LIM_SUPERBEE>("superbee", n);
  bad += run<A3G_LIM_MC>("mc", n);
  return bad ? 1 : 0;
}
