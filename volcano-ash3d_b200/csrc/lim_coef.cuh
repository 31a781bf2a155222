// lim_coef.cuh -- the limiter's frozen branch for the discrete adjoint and the
// tangent-linear sweeps.  Needs fmx and fmn, the A3G_LIM_* values and
// exact_div.cuh; the CPU test builds it for the host.
#pragma once

namespace a3g {

// d(ldq) = a*d(dq) + b*d(dqu) on the branch the forward limiter takes.
template <int LIM>
__device__ __forceinline__ void lim_coef(double dq, double dqu, double eps, double &a, double &b) {
  if (LIM == A3G_LIM_LAXWEN) { a = 1.0; b = 0.0; return; }
  if (LIM == A3G_LIM_BW) { a = 0.0; b = 1.0; return; }
  const double u = fabs(dqu), d = fabs(dq);
  if (LIM == A3G_LIM_SUPERBEE && u < 0x1p300 && d < 0x1p300) {
    // the branch by comparison, without the quotient: (a, b) is (0, 0) for
    // theta < 0, (0, 1) at 0, (0, 2) on (0, 1/2], (1, 0) between 1/2 and 1,
    // (0, 1) on [1, 2] and (2, 0) above.  RN(dqu/dq) equals 1/2, 1 or 2 only
    // when the exact quotient does, and lies on the same side of them; it is 0
    // for a dqu that is not only where the quotient underflows, which below
    // 2^300 takes a dqu below 2^-700.  Larger operands, infinities and NaN go
    // by the quotient.
    const bool same = (__double2hiint(dqu) ^ __double2hiint(dq)) >= 0;
    if (d < eps) {  // no cycle (NOCYCLE): the clamp
      a = same ? 2.0 : 0.0;
      b = 0.0;
      return;
    }
    const bool le_half = u + u <= d, lt1 = u < d, le2 = u <= d + d;
    a = le_half ? 0.0 : lt1 ? 1.0 : le2 ? 0.0 : 2.0;
    b = le_half ? 2.0 : lt1 ? 0.0 : le2 ? 1.0 : 0.0;
    if (!same) a = b = 0.0;
    if (u < 0x1p-700 && (u == 0.0 || dqu / dq == 0.0)) b = 1.0;
    return;
  }
  const bool clamp = u > 3.0 * d || d < eps;
  const double th = clamp ? copysign(3.0, dqu * dq) : div_rn(dqu, dq);
  double phi, dphi;
  if (LIM == A3G_LIM_FROMM) {
    phi = 0.5 * (1.0 + th); dphi = 0.5;
  } else if (LIM == A3G_LIM_MINMOD) {
    const double m = fmn(1.0, th), dm = (1.0 < th) ? 0.0 : 1.0;
    phi = fmx(0.0, m); dphi = (0.0 > m) ? 0.0 : dm;
  } else if (LIM == A3G_LIM_MC) {
    const double m1 = fmn((1.0 + th) / 2.0, 2.0), dm1 = ((1.0 + th) / 2.0 < 2.0) ? 0.5 : 0.0;
    const double m2 = fmn(m1, 2.0 * th), dm2 = (m1 < 2.0 * th) ? dm1 : 2.0;
    phi = fmx(0.0, m2); dphi = (0.0 > m2) ? 0.0 : dm2;
  } else {  // superbee
    const double m1 = fmn(1.0, 2.0 * th), dm1 = (1.0 < 2.0 * th) ? 0.0 : 2.0;
    const double a1 = fmx(0.0, m1), da1 = (0.0 > m1) ? 0.0 : dm1;
    const double m2 = fmn(2.0, th), dm2 = (2.0 < th) ? 0.0 : 1.0;
    phi = fmx(a1, m2); dphi = (a1 > m2) ? da1 : dm2;
  }
  if (clamp) dphi = 0.0;
  a = phi - th * dphi;
  b = dphi;
}

}  // namespace a3g
