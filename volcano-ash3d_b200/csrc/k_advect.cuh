#pragma once
// k_advect.cuh -- the forward advection sweeps (kernels and launch
// templates), shared by k_advect_x.cu, k_advect_y.cu and k_advect_z.cu, which
// instantiate one direction each, and by k_advect.cu (dt/kappa, adjoint).
//
// limited-upwind (DCU) advection sweeps on the device.
//
// Restates the row algorithm of advect_x / advect_y (src/AdvectionHorz_DCU.f90
// :68-305 / :322-556) and advect_z (src/AdvectionVert_DCU.f90:100-323):
// interface flux areas usig = 0.5*(v_{I-1}+v_I)*sigma_I, slopes dq, the
// limited second-order flux fss (superbee and the other LIM_* choices), the
// first-order fluctuations fs_r/fs_l with the divergence correction, and
// update = -dt/kappa*(fs_l(I+1)+fs_r(I)+fss(I+1)-fss(I)).  Every expression
// keeps the reference's operation order; the library is compiled with
// --fmad=false so that each product and sum rounds on its own, as the CPU
// build does, and divisions are IEEE (div.rn).  Terms that do not depend on
// the grain (flux areas, dt/kappa, 0.5|u|(1-dt/kappa|u|), the divergence
// corrections) are formed once per interface and shared by the grains a
// thread carries, which leaves each grain with one division (the limiter's
// theta) and about 25 other FP64 operations per cell.
//
// Mapping: a thread owns one line (a row along i, or a column along j or k)
// of GC grains and marches along a segment of it with a sliding register
// window (q, dq, fluxes); ghost values are generated at the line ends.  The
// y and z sweeps put neighbouring i on neighbouring lanes (coalesced); the x
// sweep puts neighbouring rows on lanes and relies on L1 to serve the four
// steps that share a 32-byte sector.  No shared memory, no barriers; the
// interior of a segment runs a branch-free step.
// Cells outside the active box and grains not aloft are written as zero: the
// zero-then-copy-back of the reference (AdvectionHorz_DCU.f90:122,302-303).
#include "a3g_internal.cuh"
#include "exact_div.cuh"
#include "tma.cuh"

#include <cstring>

namespace a3g {

// Fortran MAX/MIN of two reals as one FP64 min/max instruction.  For the
// non-NaN operands of this path they return the same value as the
// reference; at most the sign of an exact zero can differ, which no later
// operation of the sweep can turn into a different non-zero value.
__device__ __forceinline__ double dmx(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ double dmn(double a, double b) { return fmin(a, b); }

// Limited slope of one interface (src/AdvectionHorz_DCU.f90:179-226); *skip
// is set when the reference "cycle"s on |dq| <= EPS_THRESH (fss stays 0).
template <int LIM>
__device__ __forceinline__ double dcu_ldq(double dqm, double dq, double dqp, bool upw_left,
                                          double eps, int nocycle, bool &skip) {
  skip = false;
  if (!nocycle && fabs(dq) <= eps) {
    skip = true;
    return 0.0;
  }
  if (LIM == A3G_LIM_LAXWEN) return dq;
  const double dqu = upw_left ? dqm : dqp;
  double theta;
  if (fabs(dqu) > 3.0 * fabs(dq) || fabs(dq) < eps)
    theta = copysign(3.0, dqu * dq);
  else
    theta = div_rn(dqu, dq);  // == dqu/dq, see exact_div.cuh
  if (LIM == A3G_LIM_BW) return dqu;
  if (LIM == A3G_LIM_FROMM) return dq * (0.5 * (1.0 + theta));
  if (LIM == A3G_LIM_MINMOD) return dq * dmx(0.0, dmn(1.0, theta));
  if (LIM == A3G_LIM_MC) return dq * dmx(0.0, dmn(dmn((1.0 + theta) / 2.0, 2.0), 2.0 * theta));
  return dq * dmx(dmx(0.0, dmn(1.0, 2.0 * theta)), dmn(2.0, theta));
}

// Grain-independent quantities of one interface.
struct Iface {
  double usp, usm;      // max(0,usig), min(0,usig)
  double divp, divm;    // divu_p, divu_m (:245-246)
  double cf;            // 0.5*|usig|*(1 - dt_vol(I)*|usig|)  (:227-230)
  bool up;              // usig > 0 (upwind on the left)
  bool fss_ok, fs_ok;   // I in [rmin, rmax+1] / [rmin-1, rmax+1]
};

__device__ __forceinline__ Iface make_iface(double us_m, double us, double us_p, double dtv, bool fss_ok,
                                            bool fs_ok) {
  Iface f;
  f.usp = dmx(0.0, us);
  f.usm = dmn(0.0, us);
  f.divp = dmx(0.0, us) - dmx(0.0, us_m);
  f.divm = dmn(0.0, us_p) - dmn(0.0, us);
  const double aus = fabs(us);
  f.cf = 0.5 * aus * (1.0 - dtv * aus);
  f.up = us > 0.0;
  f.fss_ok = fss_ok;
  f.fs_ok = fs_ok;
  return f;
}

// fss, fs_r, fs_l of one interface for one grain (:179-249).
template <int LIM>
__device__ __forceinline__ void iface_grain(const Iface &f, double dqm, double dq, double dqp, double qm,
                                            double q, double eps, int nocycle, double &fss, double &fsr,
                                            double &fsl) {
  fss = 0.0;
  if (LIM != A3G_LIM_NONE && f.fss_ok) {
    bool skip;
    const double ldq = dcu_ldq<LIM>(dqm, dq, dqp, f.up, eps, nocycle, skip);
    if (!skip) fss = f.cf * ldq;
  }
  if (f.fs_ok) {
    fsr = f.usp * dq;
    fsl = f.usm * dq;
    fsr = fsr + q * f.divm;
    fsl = fsl + qm * f.divp;
  } else {
    fsr = 0.0;
    fsl = 0.0;
  }
}

// update of a cell from its two interfaces (:264-281)
__device__ __forceinline__ double cell_update(double dtv, double fsl_r, double fsr_l, double fss_r,
                                              double fss_l) {
  return -(dtv * (fsl_r + fsr_l + fss_r - fss_l));
}

// ---------------------------------------------------------------------------
// Marching sweep.  DIR 0: along i (lanes j, other index k); DIR 1: along j
// (lanes i, other k); DIR 2: along k (lanes i, other j).  Block (32, 4):
// threadIdx.x the lane, threadIdx.y the other index.  blockIdx.x = lane block
// * ngroups + grain group (the groups of one region run together and share
// the wind loads through L2); blockIdx.z = segment along the sweep.
// For DIR 0 the lanes are rows: each load touches one 32-byte sector per row,
// which serves the next three steps from L1.
// ---------------------------------------------------------------------------
struct LineGeo {        // a ghosted geometry line: value at sweep index c is p[(c+1)*s]
  const double *p;
  long s;
  __device__ __forceinline__ double at(int c) const { return p[(long)(c + 1) * s]; }
  __device__ __forceinline__ double ldg(int c) const { return __ldg(p + (long)(c + 1) * s); }
};

template <int DIR>
__device__ __forceinline__ LineGeo line_of(const Geo3 &g, int a, int o) {
  LineGeo r;
  if (DIR == 0) { r.p = g.p + (long)(a + 1) * g.sj + (long)(o + 1) * g.sk; r.s = g.si; }
  else if (DIR == 1) { r.p = g.p + (long)(a + 1) * g.si + (long)(o + 1) * g.sk; r.s = g.sj; }
  else { r.p = g.p + (long)(a + 1) * g.si + (long)(o + 1) * g.sj; r.s = g.sk; }
  return r;
}

// stride of a broadcast geometry array along sweep direction DIR (0: constant along the line)
template <int DIR>
inline long along(const Geo3 &g) { return DIR == 0 ? g.si : DIR == 1 ? g.sj : g.sk; }

struct CkT { static constexpr bool value = true; };     // step with range checks
struct FastT { static constexpr bool value = false; };  // interior step

template <int DIR, int LIM, int GC, bool PER, bool TOPO>
__global__ void __launch_bounds__(128, 1) k_advect_march(Layout L, Box box, int nocycle, double eps, int seg,
                                                      int ngroups, const double *__restrict__ cin,
                                                      double *__restrict__ cout,
                                                      const double *__restrict__ vel,
                                                      const double *__restrict__ vghost,
                                                      const double *__restrict__ deld, Geo4 vf, Geo3 sig,
                                                      Geo3 dtvt, const int32_t *__restrict__ aloft,
                                                      DevScalars *sc, double *__restrict__ out1,
                                                      double *__restrict__ out2) {
  // flux areas are grain independent except in z (settling speed per grain)
  constexpr int NU = (DIR == 2) ? GC : 1;
  const int gg = blockIdx.x % ngroups;
  const int a = (blockIdx.x / ngroups) * 32 + threadIdx.x + 1;   // lane index
  const int o = blockIdx.y * 4 + threadIdx.y + 1;                // other index
  const int na = (DIR == 0) ? L.ny : L.nx;
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  const int nother = (DIR == 2) ? L.ny : L.nz;
  if (a > na || o > nother) return;  // no barriers below
  const int g0 = gg * GC;
  const int s0 = 1 + blockIdx.z * seg;
  const int s1 = min(n, s0 + seg - 1);
  const int rmin = (DIR == 0) ? box.imin : (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 0) ? box.imax : (DIR == 1) ? box.jmax : box.kmax;
  const int ncells = rmax - rmin + 1;
  const long st = (DIR == 0) ? 1 : (DIR == 1) ? L.P : L.PY;
  const long base = (DIR == 0) ? L.cell(1, a, o) : (DIR == 1) ? L.cell(a, 1, o) : L.cell(a, o, 1);
  bool lane_active;
  if (DIR == 0) lane_active = a >= box.jmin && a <= box.jmax && o >= box.kmin && o <= box.kmax;
  else if (DIR == 1) lane_active = a >= box.imin && a <= box.imax && o >= box.kmin && o <= box.kmax;
  else lane_active = a >= box.imin && a <= box.imax && o >= box.jmin && o <= box.jmax;
  bool gval[GC], gal[GC];
  const double *pq[GC];
  double *po[GC];
  const double *pvf[GC];
  bool any = false;
#pragma unroll
  for (int q = 0; q < GC; q++) {
    const int g = g0 + q;
    gval[q] = g < L.ns;
    gal[q] = gval[q] && lane_active && aloft[g] != 0;
    pq[q] = cin + (long)(gval[q] ? g : 0) * L.PG + base;
    po[q] = cout + (long)(gval[q] ? g : 0) * L.PG + base;
    // vf line of this grain at sweep index c: pvf[q][(c+1)*vf.sk] (z only)
    pvf[q] = vf.p + (long)(a + 1) * vf.si + (long)(o + 1) * vf.sj + (long)(gval[q] ? g : 0) * vf.sg;
    any = any || gal[q];
  }
  if (!any) {  // nothing to advect here: the reference leaves zeros
#pragma unroll
    for (int q = 0; q < GC; q++)
      if (gval[q])
        for (int c = s0; c <= s1; c++) po[q][(long)(c - 1) * st] = 0.0;
    return;
  }
  const LineGeo gsig = line_of<DIR>(sig, a, o);
  const LineGeo gdtv = line_of<DIR>(dtvt, a, o);  // dt/kappa of this step
  const double *pv = vel + base;
  const double *pvg = vghost + base;  // ghost levels of z: plain vz (no vh)
  // DelDonD_cc(c) of this line (ZScaling_ID 2, :163-166; 0 outside
  // rmin-1..rmax+1): x row (j = a) at (c+1) + (a+1)*(nx+4), y column (i = a)
  // at (a+1) + (c+1)*(nx+4)
  const long dst = (DIR == 0) ? 1 : (long)(L.nx + 4);
  const double *pd = TOPO ? ((DIR == 0) ? deld + 1 + (long)(a + 1) * (L.nx + 4) : deld + (a + 1) + (L.nx + 4))
                          : nullptr;
  // top-outflow cell: n+1 for x and y; update_cc(ncells+1) for z (:309-311)
  const int ctop = (DIR == 2) ? ncells + 1 : rmax + 1;
  if (DIR == 2 && rmax == n && ctop < rmin - 1) raise_error(sc, A3G_ERR_UNSUPPORTED, 311);
  const bool out_lo = !PER && rmin == 1;
  const bool out_hi = !PER && rmax == n;
  const int cs = (s0 == 1 && out_lo) ? 0 : s0;
  const int ce = (s1 == n && out_hi) ? n + 1 : s1;
  const long oo_base = (long)(o - 1) * na + (a - 1);
  const long oslab = (long)na * nother;

  // ghost-aware loads (Set_BC(1): zero concentration, edge or periodic winds)
  auto wrap = [&](int c) { return c < 1 ? c + n : (c > n ? c - n : c); };
  auto qload = [&](int q, int c) -> double {
    if (c < rmin - 2 || c > rmax + 2) return 0.0;
    if (c >= 1 && c <= n) return pq[q][(long)(c - 1) * st];
    if (PER) return pq[q][(long)(wrap(c) - 1) * st];
    return 0.0;
  };
  auto vload = [&](int c) -> double {
    const int cl = PER ? wrap(c) : (c < 1 ? 1 : (c > n ? n : c));
    const double *src = (DIR == 2 && (c < 1 || c > n)) ? pvg : pv;
    return src[(long)(cl - 1) * st];
  };
  auto dload = [&](int c) -> double {
    return (c >= rmin - 1 && c <= rmax + 1) ? pd[(long)c * dst] : 0.0;
  };
  auto vfload = [&](int q, int c) -> double {
    const int cl = c < 1 ? 1 : (c > n ? n : c);
    return pvf[q][(long)(cl + 1) * vf.sk];
  };
  auto fs_ok = [&](int I) { return I >= rmin - 1 && I <= rmax + 1; };
  auto fss_ok = [&](int I) { return I >= rmin && I <= rmax + 1; };

  // ---- prologue at cell cs: interface cs, window q(cs), q(cs+1) ----------
  double q0[GC], q1[GC], d0[GC], d1[GC], fss0[GC], fsr0[GC];
  double usA[NU], usB[NU], vB[NU];  // us(c), us(c+1), vel(c+1) (+vf for z)
  double dtv0 = gdtv.at(cs);
  // topography term T(c) = 0.5*vel(c)*(sig(c)+sig(c+1))*q(c)*DelDonD(c) of
  // :251-257 (fs_r(I) += T(I), fs_l(I) -= T(I-1)): tp = T(c) per grain,
  // sB = sig(c+1) unmasked
  double tp[GC], sB = 0.0;
  {
    const double vm2 = vload(cs - 2), vm1 = vload(cs - 1), v0 = vload(cs), v1 = vload(cs + 1);
    const double sm1 = fs_ok(cs - 1) ? gsig.at(cs - 1) : 0.0;
    const double s0_ = fs_ok(cs) ? gsig.at(cs) : 0.0;
    const double s1_ = fs_ok(cs + 1) ? gsig.at(cs + 1) : 0.0;
    double usm1[NU];
#pragma unroll
    for (int u = 0; u < NU; u++) {
      double va = vm2, vb = vm1, vc = v0, vd = v1;
      if (DIR == 2) {
        va = va + vfload(u, cs - 2);
        vb = vb + vfload(u, cs - 1);
        vc = vc + vfload(u, cs);
        vd = vd + vfload(u, cs + 1);
      }
      usm1[u] = fs_ok(cs - 1) ? 0.5 * (va + vb) * sm1 : 0.0;
      usA[u] = fs_ok(cs) ? 0.5 * (vb + vc) * s0_ : 0.0;
      usB[u] = fs_ok(cs + 1) ? 0.5 * (vc + vd) * s1_ : 0.0;
      vB[u] = vd;
    }
#pragma unroll
    for (int q = 0; q < GC; q++) {
      const int u = (DIR == 2) ? q : 0;
      const double qm2 = qload(q, cs - 2), qm1 = qload(q, cs - 1);
      q0[q] = qload(q, cs);
      q1[q] = qload(q, cs + 1);
      const double dm = qm1 - qm2;
      d0[q] = q0[q] - qm1;
      d1[q] = q1[q] - q0[q];
      const Iface f = make_iface(usm1[u], usA[u], usB[u], dtv0, fss_ok(cs), fs_ok(cs));
      double fsl_unused;
      iface_grain<LIM>(f, dm, d0[q], d1[q], qm1, q0[q], eps, nocycle, fss0[q], fsr0[q], fsl_unused);
      if (TOPO) {
        const double t0 = (((0.5 * v0) * (gsig.at(cs) + gsig.at(cs + 1))) * q0[q]) * dload(cs);
        if (fs_ok(cs)) fsr0[q] = fsr0[q] + t0;
        tp[q] = t0;
      }
    }
    if (TOPO) sB = gsig.at(cs + 1);
  }

  // ---- one march step: interface c+1 and the update of cell c -------------
  // The values at the leading edge (q(c+2), vel(c+2), sigma(c+2), vf(c+2),
  // dt/kappa(c+1)) are passed in, so that the interior loop can load them
  // PF steps ahead.
  auto step = [&](int c, auto checked, const double *q2v, double vn, double sI2raw, double dtv1,
                  const double *vf2) {
    constexpr bool CK = decltype(checked)::value;
    const int I = c + 1;
    const bool fsok2 = CK ? fs_ok(c + 2) : true;
    const bool fsok1 = CK ? fs_ok(I) : true;
    const bool fssok1 = CK ? fss_ok(I) : true;
    const double sI2 = fsok2 ? sI2raw : 0.0;
    const bool own = CK ? (c >= s0 && c <= s1) : true;
    const bool inbox = CK ? (c >= rmin && c <= rmax) : true;
    const double vc1 = vB[0];                     // vel(c+1) (x, y)
    const double dcur = TOPO ? dload(I) : 0.0;    // DelDonD(c+1)
    Iface f[NU];
#pragma unroll
    for (int u = 0; u < NU; u++) {
      double vnq = vn;
      if (DIR == 2) vnq = vnq + vf2[u];
      const double usC = fsok2 ? 0.5 * (vB[u] + vnq) * sI2 : 0.0;
      vB[u] = vnq;
      f[u] = make_iface(usA[u], usB[u], usC, dtv1, fssok1, fsok1);
      usA[u] = usB[u];
      usB[u] = usC;
    }
#pragma unroll
    for (int q = 0; q < GC; q++) {
      const double q2 = q2v[q];
      const double d2 = q2 - q1[q];
      double fss1, fsr1, fsl1;
      iface_grain<LIM>(f[(DIR == 2) ? q : 0], d0[q], d1[q], d2, q0[q], q1[q], eps, nocycle, fss1, fsr1,
                       fsl1);
      if (TOPO) {
        const double t1 = (((0.5 * vc1) * (sB + sI2raw)) * q1[q]) * dcur;
        if (fsok1) {
          fsr1 = fsr1 + t1;
          fsl1 = fsl1 - tp[q];
        }
        tp[q] = t1;
      }
      const double upd = cell_update(dtv0, fsl1, fsr0[q], fss1, fss0[q]);
      if (gval[q]) {
        if (own) po[q][(long)(c - 1) * st] = (gal[q] && inbox) ? q0[q] + upd : 0.0;
        if (gal[q]) {
          if (CK && out_lo && c == 0) out1[(long)(g0 + q) * oslab + oo_base] += upd;
          if (out_hi && c == ctop) out2[(long)(g0 + q) * oslab + oo_base] += upd;
        }
      }
      fss0[q] = fss1;
      fsr0[q] = fsr1;
      q0[q] = q1[q];
      q1[q] = q2;
      d0[q] = d1[q];
      d1[q] = d2;
    }
    dtv0 = dtv1;
    if (TOPO) sB = sI2raw;
  };
  auto checked_step = [&](int c) {
    double q2v[GC], vf2[NU];
#pragma unroll
    for (int q = 0; q < GC; q++) q2v[q] = qload(q, c + 2);
#pragma unroll
    for (int u = 0; u < NU; u++) vf2[u] = (DIR == 2) ? vfload(u, c + 2) : 0.0;
    // unmasked for the topography term (sigma is ghosted to n+2)
    const double sraw = (TOPO ? (c + 2 <= n + 2) : fs_ok(c + 2)) ? gsig.at(c + 2) : 0.0;
    step(c, CkT{}, q2v, vload(c + 2), sraw, gdtv.at(c + 1), vf2);
  };
  // cells whose step needs no range checks: c >= rmin, c+2 <= min(n, rmax+1)
  int fa = max(cs, max(rmin, s0)), fb = min(ce, min(rmax - 1, n - 2));
  if (fb < fa) { fa = ce + 1; fb = ce; }
  int c = cs;
  for (; c < fa; c++) checked_step(c);
  if (fa <= fb) {
    // interior: leading-edge values come from a PF-deep ring loaded ahead;
    // loads stay inside the fast range (position <= fb+2 for q, vel, sigma,
    // vf; <= fb+1 for dt/kappa)
    constexpr int PF = 4;
    double rq[PF][GC], rv[PF], rs[PF], rd[PF], rf[PF][NU];
    auto fill = [&](int r, int cc) {  // leading-edge values of step cc into slot r
      const bool okq = cc + 2 <= fb + 2;
#pragma unroll
      for (int q = 0; q < GC; q++) rq[r][q] = okq ? pq[q][(long)(cc + 1) * st] : 0.0;
      rv[r] = okq ? pv[(long)(cc + 1) * st] : 0.0;
      rs[r] = okq ? gsig.at(cc + 2) : 0.0;
      rd[r] = okq ? gdtv.at(cc + 1) : 0.0;
#pragma unroll
      for (int u = 0; u < NU; u++) rf[r][u] = (DIR == 2 && okq) ? pvf[u][(long)(cc + 3) * vf.sk] : 0.0;
    };
#pragma unroll
    for (int r = 0; r < PF; r++) fill(r, fa + r);
    for (; c + PF - 1 <= fb; c += PF) {
#pragma unroll
      for (int r = 0; r < PF; r++) {
        double q2v[GC], vf2[NU];
#pragma unroll
        for (int q = 0; q < GC; q++) q2v[q] = rq[r][q];
#pragma unroll
        for (int u = 0; u < NU; u++) vf2[u] = rf[r][u];
        const double vn = rv[r], sr = rs[r], dd = rd[r];
        fill(r, c + r + PF);
        step(c + r, FastT{}, q2v, vn, sr, dd, vf2);
      }
    }
    // tail of the interior (fewer than PF steps); c - fa is a multiple of PF
#pragma unroll
    for (int r = 0; r < PF; r++) {
      if (c + r <= fb) {
        double q2v[GC], vf2[NU];
#pragma unroll
        for (int q = 0; q < GC; q++) q2v[q] = rq[r][q];
#pragma unroll
        for (int u = 0; u < NU; u++) vf2[u] = rf[r][u];
        step(c + r, FastT{}, q2v, rv[r], rs[r], rd[r], vf2);
      }
    }
    c = fb + 1;
  }
  for (; c <= ce; c++) checked_step(c);
}

// ---------------------------------------------------------------------------
// Block sweep: a thread computes V consecutive cells of one line for one
// grain with every input of the block loaded up front (q and the winds on
// cells c0-2 .. c0+V+1).  The V+1 interfaces of the block are independent
// straight-line code, which gives the scheduler V+1 limiter chains to
// interleave.  The limiter is written with selects (no divergent branches):
// the quotient is formed for every interface from safe operands and then
// selected.
// DIR 0: lanes are consecutive blocks along i of one row (contiguous memory,
// vector loads); DIR 1/2: lanes are consecutive i (coalesced).
// ---------------------------------------------------------------------------
template <int LIM>
__device__ __forceinline__ double fss_select(double dqm, double dq, double dqp, bool up, double cf,
                                             bool fss_ok, double eps, int nocycle) {
  if (LIM == A3G_LIM_NONE) return 0.0;
  const double adq = fabs(dq);
  const bool skip = (!nocycle && adq <= eps) || !fss_ok;  // :183 "cycle" (fss stays 0)
  double ldq;
  if (LIM == A3G_LIM_LAXWEN) {
    ldq = dq;
  } else {
    const double dqu = up ? dqm : dqp;
    const bool clamp = fabs(dqu) > 3.0 * adq || adq < eps;
    const bool use_div = !(skip || clamp);
    const double th = div_rn(use_div ? dqu : 1.0, use_div ? dq : 1.0);
    const double theta = clamp ? copysign(3.0, dqu * dq) : th;
    if (LIM == A3G_LIM_BW) ldq = dqu;
    else if (LIM == A3G_LIM_FROMM) ldq = dq * (0.5 * (1.0 + theta));
    else if (LIM == A3G_LIM_MINMOD) ldq = dq * dmx(0.0, dmn(1.0, theta));
    else if (LIM == A3G_LIM_MC) ldq = dq * dmx(0.0, dmn(dmn((1.0 + theta) / 2.0, 2.0), 2.0 * theta));
    else ldq = dq * dmx(dmx(0.0, dmn(1.0, 2.0 * theta)), dmn(2.0, theta));
  }
  return skip ? 0.0 : cf * ldq;
}

template <int DIR, int LIM, int V, bool PER, bool CK, bool LC>
__device__ __forceinline__ void block_body(const Layout &L, const Box &box, int nocycle, double eps,
                                           const double *__restrict__ line, double *__restrict__ oline,
                                           long st, const double *__restrict__ pv,
                                           const double *__restrict__ pvg, const double *pvf,
                                           long vfs, const LineGeo &gsig, const LineGeo &gdtv, int c0,
                                           int n, bool lane_active, bool al, double *o1, double *o2,
                                           DevScalars *sc) {
  const int rmin = (DIR == 0) ? box.imin : (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 0) ? box.imax : (DIR == 1) ? box.jmax : box.kmax;
  const int ncells = rmax - rmin + 1;
  const bool out_lo = !PER && rmin == 1;
  const bool out_hi = !PER && rmax == n;
  const int ctop = (DIR == 2) ? ncells + 1 : rmax + 1;
  auto wrap = [&](int c) { return c < 1 ? c + n : (c > n ? c - n : c); };
  // window w[m] = q(c0-2+m), vw[m] = vel(c0-2+m) (+vf for z), m = 0..V+3
  double w[V + 4], vw[V + 4];
  if (!CK && DIR == 0) {
    const double2 *p2 = reinterpret_cast<const double2 *>(line + (c0 - 3));
    const double2 *v2 = reinterpret_cast<const double2 *>(pv + (c0 - 3));
#pragma unroll
    for (int m = 0; m < (V + 4) / 2; m++) {
      const double2 a = p2[m], b = v2[m];
      w[2 * m] = a.x; w[2 * m + 1] = a.y;
      vw[2 * m] = b.x; vw[2 * m + 1] = b.y;
    }
  } else {
#pragma unroll
    for (int m = 0; m < V + 4; m++) {
      const int c = c0 - 2 + m;
      if (CK) {
        double q = 0.0;
        if (c >= rmin - 2 && c <= rmax + 2) {
          if (c >= 1 && c <= n) q = line[(long)(c - 1) * st];
          else if (PER) q = line[(long)(wrap(c) - 1) * st];
        }
        w[m] = q;
        const int cl = PER ? wrap(c) : (c < 1 ? 1 : (c > n ? n : c));
        vw[m] = ((DIR == 2 && (c < 1 || c > n)) ? pvg : pv)[(long)(cl - 1) * st];
      } else {
        w[m] = line[(long)(c - 1) * st];
        vw[m] = pv[(long)(c - 1) * st];
      }
    }
  }
  // LC: sigma, dt/kappa and (z) the fall speed do not vary along the line
  // (zero broadcast stride), so one load of each serves every index
  const double sig_c = LC ? gsig.p[0] : 0.0, dtv_c = LC ? gdtv.p[0] : 0.0;
  if (DIR == 2) {
    const double vf_c = LC ? pvf[0] : 0.0;
#pragma unroll
    for (int m = 0; m < V + 4; m++) {
      const int c = c0 - 2 + m;
      const int cl = CK ? (c < 1 ? 1 : (c > n ? n : c)) : c;
      vw[m] = vw[m] + (LC ? vf_c : pvf[(long)(cl + 1) * vfs]);
    }
  }
  auto fs_ok = [&](int I) { return !CK || (I >= rmin - 1 && I <= rmax + 1); };
  auto fss_ok = [&](int I) { return !CK || (I >= rmin && I <= rmax + 1); };
  // flux areas us(I), I = c0-1 .. c0+V+1  (us index u = I - (c0-1))
  double us[V + 3];
#pragma unroll
  for (int u = 0; u < V + 3; u++) {
    const int I = c0 - 1 + u;
    us[u] = fs_ok(I) ? 0.5 * (vw[u] + vw[u + 1]) * (LC ? sig_c : gsig.at(I)) : 0.0;
  }
  double dtv[V + 1];
#pragma unroll
  for (int m = 0; m <= V; m++) dtv[m] = LC ? dtv_c : gdtv.at(c0 + m);
  // interfaces I = c0+m, m = 0..V
  double fss[V + 1], fsr[V + 1], fsl[V + 1];
#pragma unroll
  for (int m = 0; m <= V; m++) {
    const int I = c0 + m;
    const Iface f = make_iface(us[m], us[m + 1], us[m + 2], dtv[m], fss_ok(I), fs_ok(I));
    const double dqm = w[m + 1] - w[m], dq = w[m + 2] - w[m + 1], dqp = w[m + 3] - w[m + 2];
    fss[m] = fss_select<LIM>(dqm, dq, dqp, f.up, f.cf, f.fss_ok, eps, nocycle);
    if (f.fs_ok) {
      fsr[m] = f.usp * dq;
      fsl[m] = f.usm * dq;
      fsr[m] = fsr[m] + w[m + 2] * f.divm;
      fsl[m] = fsl[m] + w[m + 1] * f.divp;
    } else {
      fsr[m] = 0.0;
      fsl[m] = 0.0;
    }
  }
  double outv[V];
#pragma unroll
  for (int v = 0; v < V; v++) {
    const int c = c0 + v;
    const double upd = cell_update(dtv[v], fsl[v + 1], fsr[v], fss[v + 1], fss[v]);
    const bool inbox = !CK || (c >= rmin && c <= rmax);
    outv[v] = (al && inbox) ? w[v + 2] + upd : 0.0;
    if (CK && al && out_hi && c == n) {  // cell n+1 (x, y; z when kmin == 1)
      const double updh = cell_update(dtv[v + 1], 0.0, fsr[v + 1], 0.0, fss[v + 1]);
      if (ctop == n + 1) *o2 += updh;
    }
    if (al && out_hi && c == ctop && c <= n) *o2 += upd;  // z quirk: ctop inside the column
  }
  if (CK && al && out_lo && c0 == 1) {
    // cell 0 from interfaces 0 and 1; fss(0) = 0 since rmin = 1
    const double us_m1 = 0.0;  // interface -1 is outside [rmin-1, rmax+1]
    const double dtv0 = LC ? dtv_c : gdtv.at(0);
    const Iface f0 = make_iface(us_m1, us[0], us[1], dtv0, false, true);
    const double dq0 = w[1] - w[0];
    const double fsr0 = f0.usp * dq0 + w[1] * f0.divm;
    const double upd0 = cell_update(dtv0, fsl[0], fsr0, fss[0], 0.0);
    *o1 += upd0;
  }
  if (DIR == 2 && CK && out_hi && ctop < rmin - 1) raise_error(sc, A3G_ERR_UNSUPPORTED, 311);
  // store own cells
  if (!CK && DIR == 0) {
    double2 *po = reinterpret_cast<double2 *>(oline + (c0 - 1));
#pragma unroll
    for (int v = 0; v < V / 2; v++) po[v] = make_double2(outv[2 * v], outv[2 * v + 1]);
  } else {
#pragma unroll
    for (int v = 0; v < V; v++) {
      const int c = c0 + v;
      if (!CK || c <= n) oline[(long)(c - 1) * st] = outv[v];
    }
  }
}

template <int DIR, int LIM, int V, bool PER, bool LC>
// 7 blocks of 128 per SM (at most 72 registers, a few spilled to L1): more
// warps in flight beat the spills (C2 z sweep 2.15 -> 1.81 ms on B200)
__global__ void __launch_bounds__(128, 7) k_advect_block(Layout L, Box box, int nocycle, double eps, int nblk,
                                                      const double *__restrict__ cin,
                                                      double *__restrict__ cout,
                                                      const double *__restrict__ vel,
                                                      const double *__restrict__ vghost, Geo4 vf, Geo3 sig,
                                                      Geo3 dtvt, const int32_t *__restrict__ aloft,
                                                      DevScalars *sc, double *__restrict__ out1,
                                                      double *__restrict__ out2) {
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  int a, o, blk, g;  // lane index (i or j), other index, block, grain
  if (DIR == 0) {
    blk = blockIdx.x * 32 + threadIdx.x;
    a = blockIdx.y * 4 + threadIdx.y + 1;  // j
    o = (int)(blockIdx.z % L.nz) + 1;      // k
    g = (int)(blockIdx.z / L.nz);
    if (blk >= nblk || a > L.ny) return;
  } else {
    a = blockIdx.x * 32 + threadIdx.x + 1;  // i
    const int w = blockIdx.y * 4 + threadIdx.y;
    blk = w % nblk;
    o = w / nblk + 1;
    g = blockIdx.z;
    const int nother = (DIR == 1) ? L.nz : L.ny;
    if (a > L.nx || o > nother) return;
  }
  const int c0 = 1 + blk * V;
  const long base = (DIR == 0) ? L.cell(1, a, o) : (DIR == 1) ? L.cell(a, 1, o) : L.cell(a, o, 1);
  const long st = (DIR == 0) ? 1 : (DIR == 1) ? L.P : L.PY;
  bool lane_active;
  if (DIR == 0) lane_active = a >= box.jmin && a <= box.jmax && o >= box.kmin && o <= box.kmax;
  else if (DIR == 1) lane_active = a >= box.imin && a <= box.imax && o >= box.kmin && o <= box.kmax;
  else lane_active = a >= box.imin && a <= box.imax && o >= box.jmin && o <= box.jmax;
  const bool al = lane_active && aloft[g] != 0;
  double *oline = cout + (long)g * L.PG + base;
  if (!al) {  // the reference leaves zeros
    for (int v = 0; v < V; v++)
      if (c0 + v <= n) oline[(long)(c0 + v - 1) * st] = 0.0;
    return;
  }
  const double *line = cin + (long)g * L.PG + base;
  const double *pv = vel + base;
  const double *pvg = vghost + base;
  const double *pvf = vf.p + (long)(((DIR == 0) ? 0 : a) + 1) * vf.si +
                      (long)(((DIR == 2) ? o : 0) + 1) * vf.sj + (long)g * vf.sg;
  const LineGeo gsig = line_of<DIR>(sig, a, o);
  const LineGeo gdtv = line_of<DIR>(dtvt, a, o);
  const int rmin = (DIR == 0) ? box.imin : (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 0) ? box.imax : (DIR == 1) ? box.jmax : box.kmax;
  const long na = (DIR == 0) ? L.ny : L.nx;
  const long nother = (DIR == 2) ? L.ny : L.nz;
  const long oo = (long)g * na * nother + (long)(o - 1) * na + (a - 1);
  const bool fast = c0 >= 3 && c0 >= rmin && c0 + V <= rmax && c0 + V <= n - 1;
  if (fast)
    block_body<DIR, LIM, V, PER, false, LC>(L, box, nocycle, eps, line, oline, st, pv, pvg, pvf, vf.sk, gsig, gdtv,
                                        c0, n, lane_active, al, out1 + oo, out2 + oo, sc);
  else
    block_body<DIR, LIM, V, PER, true, LC>(L, box, nocycle, eps, line, oline, st, pv, pvg, pvf, vf.sk, gsig, gdtv,
                                       c0, n, lane_active, al, out1 + oo, out2 + oo, sc);
}

// ---------------------------------------------------------------------------
// Warp-tiled x sweep.  A warp owns 32 x rows (row r = (g*nz + k-1)*ny + j-1
// starts at r*P; its winds at (r mod ny*nz)*P) and marches them side by side,
// one lane per row, over the whole row.  The leading-edge values of each
// step (q and the wind at cell c+2) come from shared-memory tiles of XA_TW
// columns that the warp fills with coalesced row segments, and the updated
// cells go out through a third tile the same way, so no lane touches global
// memory row-wise in the interior.  The arithmetic of a step is the march's
// (make_iface, iface_grain, cell_update in the same order), so the results
// are the same bits.  No lane returns early: lanes of rows past the end, of
// rows outside the box or of grains not aloft take part in the tile traffic
// and write zeros (or nothing past the last row).
// ---------------------------------------------------------------------------
constexpr int XA_TW = 16;        // tile width (cells)
constexpr int XA_S = XA_TW + 1;  // tile row stride (odd: conflict-free per-lane reads)
constexpr int XA_WARPS = 2;

template <int LIM, bool PER>
__global__ void __launch_bounds__(32 * XA_WARPS) k_advect_xt(Layout L, Box box, int nocycle, double eps,
                                                           const double *__restrict__ cin,
                                                           double *__restrict__ cout,
                                                           const double *__restrict__ vel, Geo3 sig,
                                                           Geo3 dtvt, const int32_t *__restrict__ aloft,
                                                           double *__restrict__ out1,
                                                           double *__restrict__ out2) {
  __shared__ double tq[XA_WARPS][32 * XA_S], tv[XA_WARPS][32 * XA_S], to[XA_WARPS][32 * XA_S];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long nrows = (long)L.ny * L.nz * L.ns;
  const long r0 = ((long)blockIdx.x * XA_WARPS + w) * 32;
  if (r0 >= nrows) return;  // uniform over the warp
  double *const sq = tq[w], *const sv = tv[w], *const so = to[w];
  const long plane = (long)L.ny * L.nz;
  const long r = r0 + lane;
  const bool valid = r < nrows;
  const long rc = valid ? r : nrows - 1;
  const int j = (int)(rc % L.ny) + 1;
  const int k = (int)((rc / L.ny) % L.nz) + 1;
  const int g = (int)(rc / plane);
  const int n = L.nx;
  const int rmin = box.imin, rmax = box.imax;
  const bool lane_active = j >= box.jmin && j <= box.jmax && k >= box.kmin && k <= box.kmax;
  const bool al = valid && lane_active && aloft[g] != 0;
  const long P = L.P;
  const double *pq = cin + rc * P;          // own row
  const double *pv = vel + (rc % plane) * P;
  const LineGeo gsig = line_of<0>(sig, j, k);
  const LineGeo gdtv = line_of<0>(dtvt, j, k);
  const bool out_lo = !PER && rmin == 1;
  const bool out_hi = !PER && rmax == n;
  const int ctop = rmax + 1;
  const long oo = (long)g * L.ny * L.nz + (long)(k - 1) * L.ny + (j - 1);
  auto wrap = [&](int c) { return c < 1 ? c + n : (c > n ? c - n : c); };
  // ghost-aware values of cell c of a row (Set_BC(1): zero concentration,
  // edge or periodic winds); cells beyond the reach of any step give 0
  auto qval = [&](const double *row, int c) -> double {
    if (c < rmin - 2 || c > rmax + 2 || c < -1 || c > n + 2) return 0.0;
    if (c >= 1 && c <= n) return row[c - 1];
    return PER ? row[wrap(c) - 1] : 0.0;
  };
  auto vval = [&](const double *row, int c) -> double {
    if (c < -1 || c > n + 2) return 0.0;
    const int cl = PER ? wrap(c) : (c < 1 ? 1 : (c > n ? n : c));
    return row[cl - 1];
  };
  // tile of cells t0 .. t0+XA_TW-1 for the warp's 32 rows
  auto load_tiles = [&](int t0) {
#pragma unroll 4
    for (int it = 0; it < 32 * XA_TW / 32; it++) {
      const int row = it * (32 / XA_TW) + lane / XA_TW, col = lane % XA_TW;
      const long rr = r0 + row;
      double a = 0.0, b = 0.0;
      if (rr < nrows) {
        a = qval(cin + rr * P, t0 + col);
        b = vval(vel + (rr % plane) * P, t0 + col);
      }
      sq[row * XA_S + col] = a;
      sv[row * XA_S + col] = b;
    }
    __syncwarp();
  };
  // output tile of cells o0 .. o0+XA_TW-1 (only cells 1..n are stored)
  auto flush = [&](int o0) {
    __syncwarp();
#pragma unroll 4
    for (int it = 0; it < 32 * XA_TW / 32; it++) {
      const int row = it * (32 / XA_TW) + lane / XA_TW, col = lane % XA_TW;
      const long rr = r0 + row;
      const int c = o0 + col;
      if (rr < nrows && c >= 1 && c <= n) cout[rr * P + (c - 1)] = so[row * XA_S + col];
    }
    __syncwarp();
  };
  auto fs_ok = [&](int I) { return I >= rmin - 1 && I <= rmax + 1; };
  auto fss_ok = [&](int I) { return I >= rmin && I <= rmax + 1; };
  const int cs = out_lo ? 0 : 1;
  const int ce = out_hi ? n + 1 : n;

  // ---- prologue at cell cs: interface cs, window q(cs), q(cs+1) ----
  double q0, q1, d0, d1, fss0, fsr0, usA, usB, vB;
  double dtv0 = gdtv.at(cs);
  {
    const double vm2 = vval(pv, cs - 2), vm1 = vval(pv, cs - 1), v0 = vval(pv, cs), v1 = vval(pv, cs + 1);
    const double sm1 = fs_ok(cs - 1) ? gsig.at(cs - 1) : 0.0;
    const double s0_ = fs_ok(cs) ? gsig.at(cs) : 0.0;
    const double s1_ = fs_ok(cs + 1) ? gsig.at(cs + 1) : 0.0;
    const double usm1 = fs_ok(cs - 1) ? 0.5 * (vm2 + vm1) * sm1 : 0.0;
    usA = fs_ok(cs) ? 0.5 * (vm1 + v0) * s0_ : 0.0;
    usB = fs_ok(cs + 1) ? 0.5 * (v0 + v1) * s1_ : 0.0;
    vB = v1;
    const double qm2 = qval(pq, cs - 2), qm1 = qval(pq, cs - 1);
    q0 = qval(pq, cs);
    q1 = qval(pq, cs + 1);
    const double dm = qm1 - qm2;
    d0 = q0 - qm1;
    d1 = q1 - q0;
    const Iface f = make_iface(usm1, usA, usB, dtv0, fss_ok(cs), fs_ok(cs));
    double fsl_unused;
    iface_grain<LIM>(f, dm, d0, d1, qm1, q0, eps, nocycle, fss0, fsr0, fsl_unused);
  }
  // steps that need no range checks: c >= rmin, c+2 <= min(n, rmax+1)
  const int fa = max(cs, rmin), fb = min(ce, min(rmax - 1, n - 2));
  int t0 = cs + 2;  // q/vel tile holds cells t0 .. t0+XA_TW-1 (the c+2 of steps c)
  load_tiles(t0);
  int o0 = 1;       // output tile holds cells o0 .. o0+XA_TW-1
  for (int c = cs; c <= ce; c++) {
    if (c + 2 >= t0 + XA_TW) {  // uniform: every lane is at the same c
      t0 += XA_TW;
      __syncwarp();
      load_tiles(t0);
    }
    const int ti = lane * XA_S + (c + 2 - t0);
    const double q2 = sq[ti], vn = sv[ti];
    const int I = c + 1;
    const bool fast = c >= fa && c <= fb;
    const bool fsok2 = fast || fs_ok(c + 2);
    const double sI2 = fsok2 ? gsig.at(c + 2) : 0.0;
    const double dtv1 = gdtv.at(I);
    const double usC = fsok2 ? 0.5 * (vB + vn) * sI2 : 0.0;
    vB = vn;
    const Iface f = make_iface(usA, usB, usC, dtv1, fast || fss_ok(I), fast || fs_ok(I));
    usA = usB;
    usB = usC;
    const double d2 = q2 - q1;
    double fss1, fsr1, fsl1;
    iface_grain<LIM>(f, d0, d1, d2, q0, q1, eps, nocycle, fss1, fsr1, fsl1);
    const double upd = cell_update(dtv0, fsl1, fsr0, fss1, fss0);
    if (c >= 1 && c <= n) {
      const bool inbox = c >= rmin && c <= rmax;
      so[lane * XA_S + (c - o0)] = (al && inbox) ? q0 + upd : 0.0;
      if (c == o0 + XA_TW - 1 || c == n) {
        flush(o0);
        o0 += XA_TW;
      }
    }
    if (al) {
      if (out_lo && c == 0) out1[oo] += upd;
      if (out_hi && c == ctop) out2[oo] += upd;
    }
    fss0 = fss1;
    fsr0 = fsr1;
    q0 = q1;
    q1 = q2;
    d0 = d1;
    d1 = d2;
    dtv0 = dtv1;
  }
}

template <int LIM>
static void launch_advect_xt(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  const long nrows = (long)L.ny * L.nz * L.ns;
  const long nwarps = (nrows + 31) / 32;
  const unsigned blocks = (unsigned)((nwarps + XA_WARPS - 1) / XA_WARPS);
  if (ctx->grid.periodic)
    k_advect_xt<LIM, true><<<blocks, 32 * XA_WARPS, 0, ctx->stream>>>(
        L, ctx->box, ctx->prm.nocycle, ctx->prm.eps_thresh, ctx->c0, ctx->c1, ctx->vx, ctx->snx, ctx->dtv,
        ctx->aloft, ctx->out_yz1, ctx->out_yz2);
  else
    k_advect_xt<LIM, false><<<blocks, 32 * XA_WARPS, 0, ctx->stream>>>(
        L, ctx->box, ctx->prm.nocycle, ctx->prm.eps_thresh, ctx->c0, ctx->c1, ctx->vx, ctx->snx, ctx->dtv,
        ctx->aloft, ctx->out_yz1, ctx->out_yz2);
}

// ---------------------------------------------------------------------------
// Warp-row x sweep.  A warp owns one x row (j, k) and a group of GC grains and
// walks the row in chunks of 32 cells with the lanes along i, so every global
// load and store is a coalesced row segment.  Lane l of the chunk starting at
// cell b loads cell i = b + l, forms the flux area us(i), and computes the
// fluxes of interface I = i - 1 (which needs q(I-2..I+1), us(I-1..I+1): the
// cells behind it come from per-warp shared-memory rings of 64 entries); it
// then updates cell c = I - 1 from interface I (its own) and interface c
// (lane l-1's, through the same rings).  Each interface is computed once, in
// the march's expressions (make_iface, iface_grain, cell_update), so the
// results are the same bits.  Nothing is carried in registers between
// chunks, which keeps the register count and the L1 traffic low.
// With TMA (rows whose geometry varies along i), the loads of the interior
// chunks (the ones without range checks) arrive by tensor copies instead: the warp's GC grains and the wind of the
// chunk, one chunk ahead, into one of two staging buffers, so that the
// lanes no longer wait on global loads there.  Same arithmetic, same bits.
// ---------------------------------------------------------------------------
constexpr int XW_WARPS = 4;

template <int LIM, int GC, bool PER, bool LC, bool TMA>
__global__ void __launch_bounds__(32 * XW_WARPS, 6) k_advect_xw(const __grid_constant__ CUtensorMap tq,
                                                          const __grid_constant__ CUtensorMap tv, Layout L,
                                                          Box box, int nocycle, double eps,
                                                          int ngroups, const double *__restrict__ cin,
                                                          double *__restrict__ cout,
                                                          const double *__restrict__ vel, Geo3 sig, Geo3 dtvt,
                                                          const int32_t *__restrict__ aloft, DevScalars *sc,
                                                          double *__restrict__ out1, double *__restrict__ out2) {
  __shared__ __align__(128) double s_st[TMA ? XW_WARPS : 1][2][(GC + 1) * 32];  // staged q (GC grains), v
  __shared__ __align__(8) uint64_t s_bar[XW_WARPS][2];
  __shared__ double s_q[XW_WARPS][GC][64];
  __shared__ double s_fss[XW_WARPS][GC][64];
  __shared__ double s_fsr[XW_WARPS][GC][64];
  __shared__ double s_v[XW_WARPS][64];
  __shared__ double s_u[XW_WARPS][64];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long w = (long)blockIdx.x * XW_WARPS + wid;
  if (w >= (long)L.ny * L.nz * ngroups) return;  // whole warps only; no block barrier below
  const int j = (int)(w % L.ny) + 1;
  const int k = (int)((w / L.ny) % L.nz) + 1;
  const int g0 = (int)(w / ((long)L.ny * L.nz)) * GC;
  const int n = L.nx;
  const int rmin = box.imin, rmax = box.imax;
  const bool row_active = j >= box.jmin && j <= box.jmax && k >= box.kmin && k <= box.kmax;
  const long base = L.cell(1, j, k);
  bool gval[GC], gal[GC];
  const double *pq[GC];
  double *po[GC];
  bool any = false;
#pragma unroll
  for (int q = 0; q < GC; q++) {
    const int g = g0 + q;
    gval[q] = g < L.ns;
    gal[q] = gval[q] && row_active && aloft[g] != 0;
    pq[q] = cin + (long)(gval[q] ? g : 0) * L.PG + base;
    po[q] = cout + (long)(gval[q] ? g : 0) * L.PG + base;
    any = any || gal[q];
  }
  if (!any) {  // the reference leaves zeros
#pragma unroll
    for (int q = 0; q < GC; q++)
      if (gval[q])
        for (int c = 1 + lane; c <= n; c += 32) po[q][c - 1] = 0.0;
    return;
  }
  const LineGeo gsig = line_of<0>(sig, j, k);
  const LineGeo gdtv = line_of<0>(dtvt, j, k);
  // LC: sigma and dt/kappa do not vary along the row (zero broadcast stride)
  const double sig_c = LC ? gsig.p[0] : 0.0, dtv_c = LC ? gdtv.p[0] : 0.0;
  const double *pv = vel + base;
  const bool out_lo = !PER && rmin == 1;
  const bool out_hi = !PER && rmax == n;
  const long oo = (long)(k - 1) * L.ny + (j - 1);
  const long oslab = (long)L.ny * L.nz;
  auto wrap = [&](int c) { return c < 1 ? c + n : (c > n ? c - n : c); };
  auto fs_ok = [&](int I) { return I >= rmin - 1 && I <= rmax + 1; };
  auto fss_ok = [&](int I) { return I >= rmin && I <= rmax + 1; };
  // ring slots of the chunk before the first (cells -4..-2): zero
#pragma unroll
  for (int q = 0; q < GC; q++) {
    s_q[wid][q][32 + lane] = 0.0;
    s_fss[wid][q][32 + lane] = 0.0;
    s_fsr[wid][q][32 + lane] = 0.0;
  }
  s_v[wid][32 + lane] = 0.0;
  s_u[wid][32 + lane] = 0.0;
  // chunk t covers loads i = 32t - 1 + lane and updates cells c = i - 2.  A
  // chunk whose loads all lie in [max(rmin+2, 1), min(n, rmax+1)] needs no
  // range check (its cells are inside the box, its interfaces and flux
  // areas inside [rmin, rmax+1], no ghost or outflow cell); the others take
  // the checked body.
  const int ilo = max(rmin + 2, 1), ihi = min(n, rmax + 1);
  auto chunk = [&](int t, auto checked, const double *stg) {
    constexpr bool CK = decltype(checked)::value;
    __syncwarp();
    const int i = 32 * t - 1 + lane;
    const int sl = (32 * t + lane) & 63;
    const int sl1 = (sl + 63) & 63, sl2 = (sl + 62) & 63, sl3 = (sl + 61) & 63;
    double qi[GC];
#pragma unroll
    for (int q = 0; q < GC; q++) {
      double v = 0.0;
      if (!CK) {
        v = TMA ? stg[q * 32 + lane] : pq[q][i - 1];
      } else if (i >= rmin - 2 && i <= rmax + 2) {  // ghost cells of Set_BC(1): zero, or wrapped
        if (i >= 1 && i <= n) v = pq[q][i - 1];
        else if (PER) v = pq[q][wrap(i) - 1];
      }
      qi[q] = v;
      s_q[wid][q][sl] = v;
    }
    double vi = 0.0;  // vel(i) is read by us(i) and us(i+1) only
    if (!CK) vi = TMA ? stg[GC * 32 + lane] : pv[i - 1];
    else if (i >= rmin - 2 && i <= rmax + 1) vi = pv[(PER ? wrap(i) : (i < 1 ? 1 : (i > n ? n : i))) - 1];
    s_v[wid][sl] = vi;
    __syncwarp();
    const double usi = (!CK || fs_ok(i)) ? 0.5 * (s_v[wid][sl1] + vi) * (LC ? sig_c : gsig.at(i)) : 0.0;
    s_u[wid][sl] = usi;
    __syncwarp();
    const int I = i - 1;
    const double dtvI = (!CK || (I >= -1 && I <= n + 2)) ? (LC ? dtv_c : gdtv.at(I)) : 0.0;
    const Iface f = make_iface(s_u[wid][sl2], s_u[wid][sl1], usi, dtvI, !CK || fss_ok(I), !CK || fs_ok(I));
    double qm[GC], fsl[GC], fss[GC];
#pragma unroll
    for (int q = 0; q < GC; q++) {
      const double q3 = s_q[wid][q][sl3], q2 = s_q[wid][q][sl2], q1 = s_q[wid][q][sl1];
      double fsr;
      iface_grain<LIM>(f, q2 - q3, q1 - q2, qi[q] - q1, q2, q1, eps, nocycle, fss[q], fsr, fsl[q]);
      qm[q] = q2;
      s_fss[wid][q][sl] = fss[q];
      s_fsr[wid][q][sl] = fsr;
    }
    __syncwarp();
    const int c = I - 1;
    if (!CK || (c >= 0 && c <= n + 1)) {
      const double dtvc = LC ? dtv_c : gdtv.at(c);
      const bool inbox = !CK || (c >= rmin && c <= rmax);
#pragma unroll
      for (int q = 0; q < GC; q++) {
        const double upd = cell_update(dtvc, fsl[q], s_fsr[wid][q][sl1], fss[q], s_fss[wid][q][sl1]);
        if (gval[q]) {
          if (!CK || (c >= 1 && c <= n)) po[q][c - 1] = (gal[q] && inbox) ? qm[q] + upd : 0.0;
          if (CK && gal[q]) {
            if (out_lo && c == 0) out1[(long)(g0 + q) * oslab + oo] += upd;
            if (out_hi && c == rmax + 1) out2[(long)(g0 + q) * oslab + oo] += upd;
          }
        }
      }
    }
  };
  // the interior chunks form the run tf0..tf1
  const int tf0 = (ilo + 32) / 32, tf1 = ihi >= 30 ? (ihi - 30) / 32 : -1;
  uint32_t ph = 0u;  // bit b: the parity of staging buffer b's barrier
  auto issue = [&](int t) {  // chunk t's loads i = 32t-1 .. 32t+30 (x from 32t-2 >= 0, even)
    const int bi = (t - tf0) & 1;
    if (lane == 0) {
      mbar_arrive_expect_tx(&s_bar[wid][bi], (GC + 1) * 32 * 8);
      tma_load_4d(s_st[wid][bi], &tq, &s_bar[wid][bi], 32 * t - 2, j - 1, k - 1, g0);
      tma_load_4d(s_st[wid][bi] + GC * 32, &tv, &s_bar[wid][bi], 32 * t - 2, j - 1, k - 1, 0);
    }
  };
  if (TMA) {
    if (lane == 0) {
      mbar_init(&s_bar[wid][0], 1);
      mbar_init(&s_bar[wid][1], 1);
      mbar_init_fence();
    }
    __syncwarp();
    if (tf0 <= tf1) issue(tf0);
  }
  for (int t = 0; 32 * t - 3 <= n + 1; t++) {
    if (t >= tf0 && t <= tf1) {
      if (TMA) {
        const int bi = (t - tf0) & 1;
        if (t + 1 <= tf1) issue(t + 1);
        if (!mbar_wait(&s_bar[wid][bi], (ph >> bi) & 1u)) {
          if (lane == 0) raise_error(sc, A3G_ERR_TIMEOUT, 4);
          return;
        }
        ph ^= 1u << bi;
        chunk(t, FastT{}, s_st[wid][bi]);
      } else {
        chunk(t, FastT{}, nullptr);
      }
    } else {
      chunk(t, CkT{}, nullptr);
    }
  }
}

template <int LIM>
static void launch_advect_xw(a3g_ctx *ctx, bool tma) {
  const Layout &L = ctx->L;
  const int gc = (L.ns >= 2) ? 2 : 1;
  const int ngroups = (L.ns + gc - 1) / gc;
  const long nwarps = (long)L.ny * L.nz * ngroups;
  const unsigned blocks = (unsigned)((nwarps + XW_WARPS - 1) / XW_WARPS);
  const bool lc = along<0>(ctx->snx) == 0 && along<0>(ctx->dtv) == 0;
  CUtensorMap tq, tv;
  std::memset(&tq, 0, sizeof(tq));
  std::memset(&tv, 0, sizeof(tv));
  if (tma && !(tensor_map(ctx, ctx->c0, gc == 2 ? TM_ADV_QX2 : TM_ADV_QX1, &tq) &&
               tensor_map(ctx, ctx->vx, TM_ADV_VX, &tv)))
    tma = false;
#define A3G_XW(GC_, PER_, LC_, TMA_)                                                                        \
  k_advect_xw<LIM, GC_, PER_, LC_, TMA_><<<blocks, 32 * XW_WARPS, 0, ctx->stream>>>(                        \
      tq, tv, L, ctx->box, ctx->prm.nocycle, ctx->prm.eps_thresh, ngroups, ctx->c0, ctx->c1, ctx->vx,        \
      ctx->snx, ctx->dtv, ctx->aloft, ctx->sc, ctx->out_yz1, ctx->out_yz2)
  // rows of constant geometry come here where they are few (launch_dir_lim) or without tensor maps
#define A3G_XW_LC(GC_, PER_)                      \
  if (lc) { A3G_XW(GC_, PER_, true, false); }     \
  else if (tma) { A3G_XW(GC_, PER_, false, true); } \
  else { A3G_XW(GC_, PER_, false, false); }
  if (gc == 2) {
    if (ctx->grid.periodic) { A3G_XW_LC(2, true); } else { A3G_XW_LC(2, false); }
  } else {
    if (ctx->grid.periodic) { A3G_XW_LC(1, true); } else { A3G_XW_LC(1, false); }
  }
#undef A3G_XW_LC
#undef A3G_XW
}

// the vertical wind of the z sweep: vz + vh once terrain is bound
static inline const double *dir_vel(a3g_ctx *ctx, int dir) {
  return (dir == 0) ? ctx->vx : (dir == 1) ? ctx->vy : (ctx->topo_on ? ctx->vzh : ctx->vz);
}
static inline const double *dir_vghost(a3g_ctx *ctx, int dir) {
  return (dir == 0) ? ctx->vx : (dir == 1) ? ctx->vy : ctx->vz;
}

// ---------------------------------------------------------------------------
// Column march for the y and z sweeps (DIR 1, 2): one thread per line and
// grain, lanes along i (every load and store a coalesced 256-byte row
// segment), marching the whole line with a rolling window so that each
// interface is formed once (the block kernel forms V+1 interfaces for V
// cells and loads a V+4 window).  Offsets along the line are 32-bit strides
// from per-line base pointers, the grain's fall speed is loaded once when it
// is the same in every cell (VFC), and the interior of the line runs without
// range checks.  The arithmetic of every interface and cell is block_body's
// (make_iface, fss_select, the fs_r/fs_l order, cell_update), so the results
// are the same bits.  Not periodic (only x can be), no ZScaling_ID 2 terms.
// ---------------------------------------------------------------------------
template <int DIR, int LIM, bool VFC>
__global__ void __launch_bounds__(128, 5) k_advect_col(Layout L, Box box, int nocycle, double eps,
                                                    const double *__restrict__ cin,
                                                    double *__restrict__ cout,
                                                    const double *__restrict__ vel,
                                                    const double *__restrict__ vghost, Geo4 vf, Geo3 sig,
                                                    Geo3 dtvt, const int32_t *__restrict__ aloft,
                                                    DevScalars *sc, double *__restrict__ out1,
                                                    double *__restrict__ out2) {
  static_assert(DIR == 1 || DIR == 2, "lanes along i: y and z sweeps only");
  const int a = blockIdx.x * 32 + threadIdx.x + 1;  // i
  const int o = blockIdx.y * 4 + threadIdx.y + 1;   // k (y sweep) or j (z sweep)
  const int g = blockIdx.z;
  const int nother = (DIR == 1) ? L.nz : L.ny;
  if (a > L.nx || o > nother) return;  // no barriers below
  const int n = (DIR == 1) ? L.ny : L.nz;
  const int rmin = (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 1) ? box.jmax : box.kmax;
  const int ncells = rmax - rmin + 1;
  const int st = (DIR == 1) ? (int)L.P : (int)L.PY;
  const long base = (DIR == 1) ? L.cell(a, 1, o) : L.cell(a, o, 1);
  const bool lane_active = (DIR == 1) ? (a >= box.imin && a <= box.imax && o >= box.kmin && o <= box.kmax)
                                      : (a >= box.imin && a <= box.imax && o >= box.jmin && o <= box.jmax);
  const bool al = lane_active && aloft[g] != 0;
  double *po = cout + (long)g * L.PG + base;
  if (!al) {  // the reference leaves zeros
    for (int c = 1; c <= n; c++) po[(c - 1) * st] = 0.0;
    return;
  }
  const double *pq = cin + (long)g * L.PG + base;
  const double *pv = vel + base;
  const double *pvg = vghost + base;
  const LineGeo gsig = line_of<DIR>(sig, a, o);
  const LineGeo gdtv = line_of<DIR>(dtvt, a, o);
  // fall speed of this grain along the line (z only): vf(c) at pvf[(c+1)*vfs]
  const double *pvf = vf.p + (long)(a + 1) * vf.si + (long)(((DIR == 2) ? o : 0) + 1) * vf.sj + (long)g * vf.sg;
  const long vfs = vf.sk;
  const double vf0 = (DIR == 2 && VFC) ? pvf[0] : 0.0;
  const bool out_lo = rmin == 1;
  const bool out_hi = rmax == n;
  const int ctop = (DIR == 2) ? ncells + 1 : rmax + 1;  // update_cc(ncells+1) for z (:309-311)
  if (DIR == 2 && out_hi && ctop < rmin - 1) raise_error(sc, A3G_ERR_UNSUPPORTED, 311);
  const long na = L.nx;
  const long oo = (long)g * na * nother + (long)(o - 1) * na + (a - 1);
  auto fs_ok = [&](int I) { return I >= rmin - 1 && I <= rmax + 1; };
  auto fss_ok = [&](int I) { return I >= rmin && I <= rmax + 1; };
  // ghost-aware loads (Set_BC(1): zero concentration, edge winds; the z
  // ghost levels read the plain vertical wind)
  auto qload = [&](int c) -> double {
    return (c >= rmin - 2 && c <= rmax + 2 && c >= 1 && c <= n) ? pq[(c - 1) * st] : 0.0;
  };
  auto vload = [&](int c) -> double {
    const int cl = c < 1 ? 1 : (c > n ? n : c);
    double v = ((DIR == 2 && (c < 1 || c > n)) ? pvg : pv)[(cl - 1) * st];
    if (DIR == 2) v = v + (VFC ? vf0 : pvf[(long)(cl + 1) * vfs]);
    return v;
  };
  const int cs = out_lo ? 0 : 1;
  const int ce = out_hi ? n + 1 : n;
  // ---- interface cs and the window at cs ----------------------------------
  double q0 = qload(cs), q1 = qload(cs + 1);
  double d0 = q0 - qload(cs - 1), d1 = q1 - q0;
  double usA, usB, vB, dtv0 = gdtv.at(cs), fss0, fsr0;
  {
    const double vm2 = vload(cs - 2), vm1 = vload(cs - 1), v0 = vload(cs);
    vB = vload(cs + 1);
    const double usm1 = fs_ok(cs - 1) ? 0.5 * (vm2 + vm1) * gsig.at(cs - 1) : 0.0;
    usA = fs_ok(cs) ? 0.5 * (vm1 + v0) * gsig.at(cs) : 0.0;
    usB = fs_ok(cs + 1) ? 0.5 * (v0 + vB) * gsig.at(cs + 1) : 0.0;
    const double qm1 = qload(cs - 1);
    const double dm = qm1 - qload(cs - 2);
    const Iface f = make_iface(usm1, usA, usB, dtv0, fss_ok(cs), fs_ok(cs));
    fss0 = fss_select<LIM>(dm, d0, d1, f.up, f.cf, f.fss_ok, eps, nocycle);
    fsr0 = f.fs_ok ? (f.usp * d0) + q0 * f.divm : 0.0;
  }
  // ---- one step: interface c+1 and the update of cell c --------------------
  auto step = [&](int c, auto checked, double q2, double vn, double s2, double dtv1) {
    constexpr bool CK = decltype(checked)::value;
    const int I = c + 1;
    const bool fsok2 = !CK || fs_ok(c + 2);
    const double usC = fsok2 ? 0.5 * (vB + vn) * s2 : 0.0;
    vB = vn;
    const Iface f = make_iface(usA, usB, usC, dtv1, !CK || fss_ok(I), !CK || fs_ok(I));
    usA = usB;
    usB = usC;
    const double d2 = q2 - q1;
    const double fss1 = fss_select<LIM>(d0, d1, d2, f.up, f.cf, f.fss_ok, eps, nocycle);
    double fsr1 = 0.0, fsl1 = 0.0;
    if (f.fs_ok) {
      fsr1 = f.usp * d1;
      fsl1 = f.usm * d1;
      fsr1 = fsr1 + q1 * f.divm;
      fsl1 = fsl1 + q0 * f.divp;
    }
    const double upd = cell_update(dtv0, fsl1, fsr0, fss1, fss0);
    if (!CK || (c >= 1 && c <= n)) {
      const bool inbox = !CK || (c >= rmin && c <= rmax);
      po[(c - 1) * st] = inbox ? q0 + upd : 0.0;
    }
    if (CK && out_lo && c == 0) out1[oo] += upd;
    if (out_hi && c == ctop) out2[oo] += upd;
    fss0 = fss1;
    fsr0 = fsr1;
    q0 = q1;
    q1 = q2;
    d0 = d1;
    d1 = d2;
    dtv0 = dtv1;
  };
  auto checked_step = [&](int c) {
    step(c, CkT{}, qload(c + 2), vload(c + 2), fs_ok(c + 2) ? gsig.at(c + 2) : 0.0, gdtv.at(c + 1));
  };
  // steps without range checks: c >= rmin, c+2 <= min(n, rmax+1)
  int fa = max(cs, rmin), fb = min(n - 2, rmax - 1);
  if (fb < fa) { fa = ce + 1; fb = ce; }
  int c = cs;
  for (; c < fa; c++) checked_step(c);
  if (fa <= fb) {
    const double *qn = pq + (fa + 1) * st;   // q(c+2)
    const double *vn = pv + (fa + 1) * st;   // vel(c+2)
    const double *sn = gsig.p + (long)(fa + 3) * gsig.s;   // sigma(c+2)
    const double *dn = gdtv.p + (long)(fa + 2) * gdtv.s;   // dt/kappa(c+1)
    const double *fn = pvf + (long)(fa + 3) * vfs;         // vf(c+2)
    const int ss = (int)gsig.s, ds = (int)gdtv.s, fs = (int)vfs;
#pragma unroll 4
    for (; c <= fb; c++) {
      double v = *vn;
      if (DIR == 2) v = v + (VFC ? vf0 : *fn);
      step(c, FastT{}, *qn, v, *sn, *dn);
      qn += st;
      vn += st;
      sn += ss;
      dn += ds;
      if (DIR == 2 && !VFC) fn += fs;
    }
  }
  for (; c <= ce; c++) checked_step(c);
}

template <int DIR, int LIM>
static void launch_col(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  const int nother = (DIR == 1) ? L.nz : L.ny;
  dim3 grid((L.nx + 31) / 32, (nother + 3) / 4, L.ns);
  const bool vfc = ctx->vf.si == 0 && ctx->vf.sj == 0 && ctx->vf.sk == 0;
#define A3G_COL(VFC_)                                                                                     \
  k_advect_col<DIR, LIM, VFC_><<<grid, dim3(32, 4), 0, ctx->stream>>>(                                  \
      L, ctx->box, ctx->prm.nocycle, ctx->prm.eps_thresh, ctx->c0, ctx->c1, dir_vel(ctx, DIR),           \
      dir_vghost(ctx, DIR), ctx->vf, (DIR == 1) ? ctx->sny : ctx->snz, ctx->dtv, ctx->aloft, ctx->sc,    \
      (DIR == 1) ? ctx->out_xz1 : ctx->out_xy1, (DIR == 1) ? ctx->out_xz2 : ctx->out_xy2)
  if (DIR == 2 && !vfc) A3G_COL(false); else A3G_COL(true);
#undef A3G_COL
}

// ---------------------------------------------------------------------------
// The marching step that the TMA-fed sweeps share.
// ---------------------------------------------------------------------------
// max(0, x) and min(0, x); both 0 for a NaN, as dmx and dmn give them, so that
// a missing wind carries no first-order flux whichever kernel sweeps its cell.
__device__ __forceinline__ double pos_part(double x) { return x > 0.0 ? x : 0.0; }
__device__ __forceinline__ double neg_part(double x) { return x < 0.0 ? x : 0.0; }
// The same of a number, by the sign bit (a NaN stays one in either): 9
// instructions a cell fewer in the y march's steps.
__device__ __forceinline__ double pos_bits(double x) {
  const int h = __double2hiint(x), m = ~(h >> 31);
  return __hiloint2double(h & m, __double2loint(x) & m);
}
__device__ __forceinline__ double neg_bits(double x) {
  const int h = __double2hiint(x), m = h >> 31;
  return __hiloint2double(h & m, __double2loint(x) & m);
}
__device__ __forceinline__ bool finite_bits(double x) { return (__double2hiint(x) & 0x7fffffff) < 0x7ff00000; }

// Second-order flux of one interface, cf*ldq (0 where the reference cycles),
// the same value as fss_select's, cf = 0.5*aus*(1 - dtv*aus).  Superbee's factor
// is 0 for ratios dqu/dq <= 0, 2 from 2 up, 1 on [1/2, 1], and 2*theta or theta in
// between, and rounding to nearest cannot move a quotient across those bounds,
// so the class comes from comparisons of dqu, with dq's sign taken off, with |dq|
// and 2|dq|, the quotient is needed in two classes only, and it is divided by the
// operator only where one of those lanes holds operands out of quot_rn's
// range.  A ratio that is NaN is in the class of 2 (fmin and fmax pass it
// over).  ANY: aus may be NaN (a missing wind), which reaches every interface
// that does not cycle, and no other.  `up` may be either for usig = 0, where
// cf = 0.  NOCYCLE, which no reference build sets, goes by the general rule.
static __device__ __noinline__ double ieee_theta(double dqu, double dq, bool twice) {
  const double th = dqu / dq;
  return twice ? th + th : th;
}

template <int LIM>
static __device__ __noinline__ double fss_nocycle(double dqm, double dq, double dqp, bool up, double cf, double eps) {
  return fss_select<LIM>(dqm, dq, dqp, up, cf, true, eps, 1);
}

template <int LIM, bool ANY>
__device__ __forceinline__ double fss_step(double dqm, double dq, double dqp, bool up, double aus, double dtv,
                                           double eps, bool nocycle) {
  if (LIM == A3G_LIM_NONE) return 0.0;
  if (LIM != A3G_LIM_SUPERBEE)
    return fss_select<LIM>(dqm, dq, dqp, up, 0.5 * aus * (1.0 - dtv * aus), true, eps, nocycle);
  if (nocycle) return fss_nocycle<LIM>(dqm, dq, dqp, up, 0.5 * aus * (1.0 - dtv * aus), eps);
  const double dqu = up ? dqm : dqp, b = fabs(dq);
  const double s = __hiloint2double(__double2hiint(dqu) ^ (__double2hiint(dq) & (int)0x80000000), __double2loint(dqu));
  const bool lt = s + s < b, gt = s > b, ge2 = !(s < b + b), skip = b <= eps, none = skip || s <= 0.0;
  const bool need = !none && !ge2 && (lt || gt);
  double th;
  const bool ok = quot_rn(dqu, dq, &th);
  int hi = __double2hiint(th) + (lt ? 1 << 20 : 0), lo = __double2loint(th);  // 2*theta of a normal theta
  if (need && !ok) {
    th = ieee_theta(dqu, dq, lt);
    hi = __double2hiint(th);
    lo = __double2loint(th);
  }
  const int flat = none ? 0 : (ge2 ? 0x40000000 : 0x3ff00000);  // 0, 2 or 1
  const double phi = __hiloint2double(need ? hi : flat, need ? lo : 0);
  const double cf = 0.5 * aus * (1.0 - dtv * aus);
  return ANY && skip ? 0.0 : cf * (dq * phi);
}

// The values a march carries from cell c to cell c+1.
struct March {
  double q0, q1, d0, d1;   // q(c), q(c+1), q(c)-q(c-1), q(c+1)-q(c)
  double us, vB;           // usig(c+1), vel(c+1)
  double upA, upB, unB;    // max(0,usig(c)), max(0,usig(c+1)), min(0,usig(c+1))
  double fss0, fsr0, dtv0; // fss(c), fs_r(c), dt/kappa(c)
};

// One interior step (no range checks): interface c+1 from q2 = q(c+2), d2 =
// q2 - q(c+1), vn = vel(c+2), hs = sigma(c+2)/2 and dtv1 = dt/kappa(c+1).
// Returns the sum whose product with dt/kappa(c) is taken off q(c) (:264-281).
// usig = 0.5*(v+v')*sigma is (v+v')*(sigma/2): halving is exact.  QUIET: the
// caller knows that |dq| <= EPS_THRESH at this interface; ANY: it does not know
// that the winds are numbers.
template <int LIM, bool QUIET, bool ANY>
__device__ __forceinline__ double march_step(March &m, double q2, double d2, double vn, double hs, double dtv1,
                                             double eps, bool nocycle) {
  const double usC = (m.vB + vn) * hs;
  const double upC = ANY ? pos_part(usC) : pos_bits(usC), unC = ANY ? neg_part(usC) : neg_bits(usC);
  double fss1 = 0.0;
  if (!QUIET && LIM != A3G_LIM_NONE) {
    fss1 = fss_step<LIM, ANY>(m.d0, m.d1, d2, __double2hiint(m.us) >= 0, fabs(m.us), dtv1, eps, nocycle);
  }
  double fsr1 = m.upB * m.d1;
  double fsl1 = m.unB * m.d1;
  fsr1 = fsr1 + m.q1 * (unC - m.unB);
  fsl1 = fsl1 + m.q0 * (m.upB - m.upA);
  const double sum = fsl1 + m.fsr0 + fss1 - m.fss0;
  m.us = usC;
  m.vB = vn;
  m.upA = m.upB;
  m.upB = upC;
  m.unB = unC;
  m.fss0 = fss1;
  m.fsr0 = fsr1;
  m.q0 = m.q1;
  m.q1 = q2;
  m.d0 = m.d1;
  m.d1 = d2;
  return sum;
}

// ---------------------------------------------------------------------------
// Column march fed by TMA chunks (y and z sweeps).  One warp per 32 lines of
// 32 consecutive i at one (other index, grain), lanes along i, marching the
// line with each interface formed once and the values of block_body (the same
// bits).  The concentration and the wind of cell c+2 come from shared memory:
// chunks of ACH cells of both arrive by two tensor loads into one of two
// buffers per warp, the next chunk in flight while the lanes march through
// the current one, and the geometry of the chunk's cells (sigma/2, dt/kappa:
// the same for the warp's lines) is staged beside them.  Every cell of the
// line takes the same unchecked step: concentrations beyond the line arrive
// as the zeros of Set_BC(1), the wind beyond its last cell is written into
// the last chunk, and the flux areas beyond the box are zero because their
// sigma is staged as zero.  The interface the line starts from and the two
// outflow cells are formed outside the loop.  Warps are ordered
// grain-fastest, so the grains of a tile run side by side and share its wind
// rows through L2.  Taken when the geometry is constant along i and the fall
// speed is one value per grain.
//
// Bound by instruction issue (68 % of cycles on 720x120x60, 10 grains) and the
// FP64 pipe (50 %).  march_step() forms an interface in about 100 instructions
// where block_body's expressions and the checked steps at the line ends took
// 190, and a chunk whose differences are all within EPS_THRESH on every lane --
// the air around a cloud -- takes steps without the limiter: 720x360x60, 10
// grains, ash in every cell, y 1.12 -> 0.71 ms and z 1.22 -> 0.77 ms a sweep.
// Lines are cut into segments of `seg` cells where whole lines would leave
// the chip short of warps (launch_colt); a segment repeats one interface.
// ---------------------------------------------------------------------------
constexpr int ACT_WARPS = 2;
constexpr int ACT_MINB = 8;  // 128 registers, none spilled: 9 and 10 blocks spill and run 5 % slower
constexpr int ACT_U = 4;     // steps unrolled: 4 measured faster than 8 (instruction cache) and than 2
// doubles per warp: two buffers of (q, v) chunks and two of staged geometry
constexpr int ACT_WARP_D = 2 * 2 * ACH * 32 + 2 * 2 * ACH;
static_assert((ACT_WARP_D * 8) % 128 == 0, "warp regions stay 128-byte aligned");
struct TrueT { static constexpr bool value = true; };
struct FalseT { static constexpr bool value = false; };

// VAR: geometry that varies along i (terrain); each lane loads its own
// sigma and dt/kappa, ACT_U cells at a time, in place of the staged pairs
// (z on 201x151x41, 5 grains: 90 us in the block kernel, 54 here).
template <int DIR, int LIM, bool VAR>
__global__ void __launch_bounds__(32 * ACT_WARPS, VAR ? ACT_MINB - 2 : ACT_MINB) k_advect_colt(
    const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tv, Layout L, Box box, Box cov,
    int nocycle, double eps, int nseg, int seg, const double *__restrict__ cin, double *__restrict__ cout,
    const double *__restrict__ vel, const double *__restrict__ vghost, Geo4 vf, Geo3 sig, Geo3 dtvt,
    const int32_t *__restrict__ aloft, DevScalars *sc, double *__restrict__ out1, double *__restrict__ out2) {
  static_assert(DIR == 1 || DIR == 2, "lanes along i: y and z sweeps only");
  extern __shared__ __align__(128) unsigned char act_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t *bar = reinterpret_cast<uint64_t *>(act_smem) + 2 * wid;
  double *wsm = reinterpret_cast<double *>(act_smem + 128) + (long)wid * ACT_WARP_D;
  // buffer b: q chunk at wsm + b*2*ACH*32, v chunk after it; geometry of
  // buffer b at wsm + 4*ACH*32 + b*2*ACH: pairs (sigma(c+2)/2, dt/kappa(c+1))
  const int nother = (DIR == 1) ? L.nz : L.ny;
  // lines of the cover: 32-column tiles it0.., other index o0.., sweep index l0..l1
  const int it0 = (cov.imin - 1) >> 5, nti = ((cov.imax - 1) >> 5) - it0 + 1;
  const int o0 = (DIR == 1) ? cov.kmin : cov.jmin, no = ((DIR == 1) ? cov.kmax : cov.jmax) - o0 + 1;
  const int l0 = (DIR == 1) ? cov.jmin : cov.kmin, l1 = (DIR == 1) ? cov.jmax : cov.kmax;
  const unsigned t = blockIdx.x * ACT_WARPS + wid;  // 32-bit: a 64-bit division costs a small grid a microsecond
  const unsigned ns = L.ns, rr = t / ns, ro = rr / (unsigned)nti;
  if (ro >= (unsigned)(no * nseg)) return;  // whole warps only; no block barrier below
  const int g = (int)(t - rr * ns);
  const int it = it0 + (int)(rr - ro * (unsigned)nti);
  const int sg_ = (int)(ro / (unsigned)no);
  const int o = o0 + (int)ro - sg_ * no;  // k (y sweep) or j (z sweep)
  const int s0 = l0 + sg_ * seg;
  const int a = (it << 5) + lane + 1;  // i
  const bool valid = a <= L.nx;
  const int n = (DIR == 1) ? L.ny : L.nz;
  const int s1 = min(l1, s0 + seg - 1);
  const int rmin = (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 1) ? box.jmax : box.kmax;
  const int st = (DIR == 1) ? (int)L.P : (int)L.PY;
  const int ac = valid ? a : 1;
  const bool lane_active = (DIR == 1) ? (a >= box.imin && a <= box.imax && o >= box.kmin && o <= box.kmax)
                                      : (a >= box.imin && a <= box.imax && o >= box.jmin && o <= box.jmax);
  const bool al = valid && lane_active && aloft[g] != 0;
  double *po = cout + (long)g * L.PG + ((DIR == 1) ? L.cell(ac, 1, o) : L.cell(ac, o, 1));
  const int c0 = max(s0, rmin), c1 = min(s1, rmax);  // the cells marched
  // the reference leaves zeros outside the box and for grains not aloft
  if (valid) {
    const int z0 = (al && c0 <= c1) ? c0 : s1 + 1;
    for (int c = s0; c < z0; c++) po[(c - 1) * st] = 0.0;
    for (int c = max(c1 + 1, z0); c <= s1; c++) po[(c - 1) * st] = 0.0;
  }
  if (c0 > c1 || !__any_sync(0xffffffffu, al)) return;
  const bool out_hi = rmax == n;
  // update_cc(ncells+1) for z (:309-311): cell n+1 of a box on the ground
  const int ctop = (DIR == 2) ? rmax - rmin + 2 : rmax + 1;
  if (DIR == 2 && out_hi && ctop < rmin - 1 && lane == 0) raise_error(sc, A3G_ERR_UNSUPPORTED, 311);
  const int nchunk = (c1 - c0) / ACH + 1;
  // chunk k holds cells C0(k) .. C0(k)+ACH-1, C0(k) = c0+2+k*ACH: the cell
  // c+2 of the steps c = c0+k*ACH ..
  auto issue = [&](int k) {
    double *qb = wsm + (k & 1) * 2 * ACH * 32;
    const int C0 = c0 + 2 + k * ACH;
    if (lane == 0) {
      uint64_t *b = &bar[k & 1];
      mbar_arrive_expect_tx(b, 2u * ACH * 32u * 8u);
      if (DIR == 1) {
        tma_load_4d(qb, &tq, b, it << 5, C0 - 1, o - 1, g);
        tma_load_4d(qb + ACH * 32, &tv, b, it << 5, C0 - 1, o - 1, 0);
      } else {
        tma_load_4d(qb, &tq, b, it << 5, o - 1, C0 - 1, g);
        tma_load_4d(qb + ACH * 32, &tv, b, it << 5, o - 1, C0 - 1, 0);
      }
    }
    if (VAR) return;
    const LineGeo gsig = line_of<DIR>(sig, 1, o), gdtv = line_of<DIR>(dtvt, 1, o);  // constant along i
    double2 *gb = reinterpret_cast<double2 *>(wsm + 4 * ACH * 32 + (k & 1) * 2 * ACH);
    const int I = C0 + lane;
    if (lane < ACH && I <= n + 2) gb[lane] = make_double2(I <= rmax + 1 ? 0.5 * gsig.at(I) : 0.0, gdtv.at(I - 1));
  };
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
  }
  __syncwarp();
  issue(0);
  const double vf0 = (DIR == 2) ? vf.p[(long)g * vf.sg] : 0.0;  // one fall speed per grain
  const long oo = (long)g * L.nx * nother + (long)(o - 1) * L.nx + (ac - 1);
  // ---- interface c0 and the window at c0; vedge: the wind beyond the line ----
  March m;
  double vedge;
  {
    const long base = (DIR == 1) ? L.cell(ac, 1, o) : L.cell(ac, o, 1);
    const double *pq = cin + (long)g * L.PG + base;
    const double *pv = vel + base, *pvg = vghost + base;
    const LineGeo gsig = line_of<DIR>(sig, VAR ? ac : 1, o), gdtv = line_of<DIR>(dtvt, VAR ? ac : 1, o);
    auto qload = [&](int c) -> double {
      return (c >= rmin - 2 && c <= rmax + 2 && c >= 1 && c <= n) ? pq[(c - 1) * st] : 0.0;
    };
    auto vload = [&](int c) -> double {  // edge winds; the z ghost levels read the plain vertical wind
      const int cl = c < 1 ? 1 : (c > n ? n : c);
      const double v = ((DIR == 2 && (c < 1 || c > n)) ? pvg : pv)[(cl - 1) * st];
      return (DIR == 2) ? v + vf0 : v;
    };
    vedge = ((DIR == 2) ? pvg : pv)[(n - 1) * st];
    m.q0 = qload(c0);
    m.q1 = qload(c0 + 1);
    const double qm1 = qload(c0 - 1), qm2 = qload(c0 - 2);
    m.d0 = m.q0 - qm1;
    m.d1 = m.q1 - m.q0;
    m.dtv0 = gdtv.at(c0);
    const double vm2 = vload(c0 - 2), vm1 = vload(c0 - 1), v0 = vload(c0);
    m.vB = vload(c0 + 1);
    const double usm1 = 0.5 * (vm2 + vm1) * gsig.at(c0 - 1);
    const double usA = 0.5 * (vm1 + v0) * gsig.at(c0);
    m.us = 0.5 * (v0 + m.vB) * gsig.at(c0 + 1);
    const double dm = qm1 - qm2;
    const Iface f = make_iface(usm1, usA, m.us, m.dtv0, true, true);
    m.fss0 = fss_select<LIM>(dm, m.d0, m.d1, f.up, f.cf, true, eps, nocycle);
    m.fsr0 = f.usp * m.d0;
    m.fsr0 = m.fsr0 + m.q0 * f.divm;
    // cell rmin-1: the low outflow of a box at the edge (or the z quirk's cell)
    if (c0 == rmin && (rmin == 1 || (DIR == 2 && out_hi && ctop == rmin - 1))) {
      double fsl = f.usm * m.d0;
      fsl = fsl + qm1 * f.divp;
      double fsr = pos_part(usm1) * dm;
      fsr = fsr + qm1 * (neg_part(usA) - neg_part(usm1));
      const double upd = cell_update(gdtv.at(c0 - 1), fsl, fsr, m.fss0, 0.0);
      if (al) (rmin == 1 ? out1 : out2)[oo] += upd;
    }
    m.upA = pos_part(usA);
    m.upB = pos_part(m.us);
    m.unB = neg_part(m.us);
  }
  const bool nocyc = nocycle != 0;
  const int eps_hi = nocyc ? 0 : __double2hiint(eps);  // |d| < eps for certain, by its high word alone
  po += (long)(c0 - 1) * st;                           // cell c's place from here on
  const LineGeo lsig = line_of<DIR>(sig, ac, o), ldtv = line_of<DIR>(dtvt, ac, o);
  // sigma(I)/2 and dt/kappa(I-1), I = c+2 the cell at slot e of the chunk
  auto geo = [&](const double2 *gb, int e, int I) {
    return VAR ? make_double2(I <= rmax + 1 ? 0.5 * lsig.ldg(I) : 0.0, ldtv.ldg(I - 1)) : gb[e];
  };
  // the step c from the values of cell c+2 at slot e of the chunk
  auto step = [&](auto quiet, auto any, const double *qv, double2 sd, int e) {
    const double q0 = m.q0, q2 = qv[e * 32];
    const double vn = (DIR == 2) ? qv[(ACH + e) * 32] + vf0 : qv[(ACH + e) * 32];
    const double sum = march_step<LIM, decltype(quiet)::value, decltype(any)::value>(m, q2, q2 - m.q1, vn, sd.x, sd.y,
                                                                                     eps, nocyc);
    const double upd = m.dtv0 * sum;
    if (al) *po = q0 - upd;
    po += st;
    m.dtv0 = sd.y;
    return upd;
  };
  uint32_t ph = 0u;
  for (int k = 0, c = c0; k < nchunk; k++) {
    const int bi = k & 1;
    if (k + 1 < nchunk) issue(k + 1);
    if (!mbar_wait(&bar[bi], (ph >> bi) & 1u)) {
      if (lane == 0) raise_error(sc, A3G_ERR_TIMEOUT, 3);
      return;
    }
    ph ^= 1u << bi;
    double *qv = wsm + bi * 2 * ACH * 32 + lane;
    // cells of the chunk's steps; the wind of cell n+1 (only the last chunk holds it)
    const int cnt = min(ACH, c1 - c + 1);
    if (c + 2 <= n + 1 && n + 1 <= c + 1 + cnt) qv[(ACH + n - 1 - c) * 32] = vedge;
    __syncwarp();
    const double2 *gb = reinterpret_cast<const double2 *>(wsm + 4 * ACH * 32 + bi * 2 * ACH);
    int e = 0;
    // whether every wind that the chunk's interfaces take is a number: their sum is
    double sum = m.vB + m.us + vf0;
#pragma unroll
    for (int u = 0; u < ACH; u += 2) sum = sum + (qv[(ACH + u) * 32] + qv[(ACH + u + 1) * 32]);
    if (__any_sync(0xffffffffu, al && !finite_bits(sum))) {
      for (; e < cnt; e++) {
        const double upd = step(FalseT{}, TrueT{}, qv, geo(gb, e, c + e + 2), e);
        if (DIR == 2 && al && out_hi && c + e == ctop) out2[oo] -= upd;
      }
    } else if (!(DIR == 2 && out_hi && ctop <= rmax)) {  // the z sweep's ctop (a box off the ground) is the last loop's
      // the differences the chunk's interfaces limit: d1 and the first cnt-1 new ones
      int top = __double2hiint(m.d1) & 0x7fffffff;
      double prev = m.q1;
#pragma unroll
      for (int u = 0; u < ACH - 1; u++) {
        const double x = qv[u * 32];
        top = max(top, __double2hiint(x - prev) & 0x7fffffff);
        prev = x;
      }
      if (LIM == A3G_LIM_NONE || __all_sync(0xffffffffu, top < eps_hi || !al)) {
        for (; e + 2 <= cnt; e += 2) {
          const double2 sd0 = geo(gb, e, c + e + 2), sd1 = geo(gb, e + 1, c + e + 3);
          step(TrueT{}, FalseT{}, qv, sd0, e);
          step(TrueT{}, FalseT{}, qv, sd1, e + 1);
        }
      } else {
        for (; e + ACT_U <= cnt; e += ACT_U) {
          double2 sd[ACT_U];
          if (VAR) {
#pragma unroll
            for (int u = 0; u < ACT_U; u++) sd[u] = geo(gb, e + u, c + e + u + 2);
          }
#pragma unroll
          for (int u = 0; u < ACT_U; u++) step(FalseT{}, FalseT{}, qv, VAR ? sd[u] : gb[e + u], e + u);
        }
      }
    }
    for (; e < cnt; e++) {
      const double upd = step(FalseT{}, FalseT{}, qv, geo(gb, e, c + e + 2), e);
      if (DIR == 2 && al && out_hi && c + e == ctop) out2[oo] -= upd;
    }
    c += cnt;
    __syncwarp();
  }
  // cell n+1: interface n+2 lies outside the box and carries nothing
  if (al && s1 == n && out_hi && ctop == n + 1) out2[oo] += cell_update(m.dtv0, 0.0, m.fsr0, 0.0, m.fss0);
}

// Segments a marched line of n cells is cut into, given the warps that whole
// lines would make: the count with the least waves x cells per wave, where a
// wave is the 16 warps an SM's registers hold and a segment's start costs
// about eight cells (its loads, and the interface it repeats).  93x131x37, 2
// grains: y 56 -> 14 us, z 27 -> 14 us a sweep (whole lines 45, 22);
// 140x120x40, 4 grains: x 27.4 -> 24.6, y 20.3 -> 18.7 us against 20 warps an
// SM whatever the waves.  At most 32, or 128 where whole lines are less than 16
// warps (1000x20x10, 1 grain: x 12.3 -> 10.3, its transpose 16.4 -> 12.3 us; at
// 2000x100x10, 2 grains, 37 instead of 32 took the transpose from 42 to 52).
static inline int march_segments(int n, long warps) {
  const long wave = 148L * 16;
  const int most = warps < 16 ? 128 : 32;
  int best = 1;
  long least = 0;
  for (int s = 1; s == 1 || (s <= most && n / s >= 6); s++) {
    const long cost = ((warps * s + wave - 1) / wave) * ((n + s - 1) / s + 8);
    if (s == 1 || cost < least) {
      best = s;
      least = cost;
    }
  }
  return best;
}

// Launches the TMA-fed column march; false when its conditions do not hold
// (the caller takes another variant).
template <int DIR, int LIM>
static bool launch_colt(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  const Geo3 &sg = (DIR == 1) ? ctx->sny : ctx->snz;
  const bool var = sg.si != 0 || ctx->dtv.si != 0;
  if (DIR == 2 && (ctx->vf.si != 0 || ctx->vf.sj != 0 || ctx->vf.sk != 0)) return false;
  CUtensorMap tq, tv;
  const double *vel = dir_vel(ctx, DIR);
  if (!tensor_map(ctx, ctx->c0, DIR == 1 ? TM_ADV_QY : TM_ADV_QZ, &tq) ||
      !tensor_map(ctx, vel, DIR == 1 ? TM_ADV_VY : TM_ADV_VZ, &tv))
    return false;
  const size_t smem = 128 + (size_t)ACT_WARPS * ACT_WARP_D * sizeof(double);
  static_assert(128 + ACT_WARPS * ACT_WARP_D * 8 <= 48 * 1024, "fits the default dynamic limit");
  const Box cov = cover_box(ctx);
  const int n = (DIR == 1) ? cov.jmax - cov.jmin + 1 : cov.kmax - cov.kmin + 1;
  const int nother = (DIR == 1) ? cov.kmax - cov.kmin + 1 : cov.jmax - cov.jmin + 1;
  const long nlw = (long)((cov.imax - 1) / 32 - (cov.imin - 1) / 32 + 1) * nother * L.ns;  // warps of whole lines
  const int nseg = march_segments(n, nlw);
  const int seg = (n + nseg - 1) / nseg;
  const long nw = nlw * ((n + seg - 1) / seg);
  auto run = [&](auto kernel) {
    kernel<<<(unsigned)((nw + ACT_WARPS - 1) / ACT_WARPS), 32 * ACT_WARPS, smem, ctx->stream>>>(
        tq, tv, L, ctx->box, cov, ctx->prm.nocycle, ctx->prm.eps_thresh, (n + seg - 1) / seg, seg, ctx->c0, ctx->c1, vel,
        dir_vghost(ctx, DIR), ctx->vf, sg, ctx->dtv, ctx->aloft, ctx->sc, (DIR == 1) ? ctx->out_xz1 : ctx->out_xy1,
        (DIR == 1) ? ctx->out_xz2 : ctx->out_xy2);
  };
  if (var) run(k_advect_colt<DIR, LIM, true>);
  else run(k_advect_colt<DIR, LIM, false>);
  return true;
}

// ---------------------------------------------------------------------------
// Row march fed by TMA chunks (x sweep).  A warp owns 32 rows of one grain
// (row r = (k-1)*ny + j-1 of the plane) with one row per lane, and marches
// them with march_step() as the column march does: no exchange between lanes
// and no ring in shared memory.  Chunks of 8 cells x 32 rows of the
// concentration and the wind arrive by tensor loads in the 64-byte swizzle,
// under which the lanes' 16-byte reads of their own rows meet no bank twice;
// the new cells replace the chunk's old ones in place, two cells behind, and
// leave by a tensor store.  Chunk t holds the cells s0+2+8t .. of a segment
// that starts at s0 = 1 (mod 8), so that loads start on an even cell and
// stores on a multiple of 8 (the 16-byte rule).  Three concentration buffers
// turn: one being marched, one loading, one being stored.  A tile whose 32
// rows are not all this plane's (the last of a grain) is stored by the lanes.
// Taken when sigma and dt/kappa do not vary along the row.
//
// Bound, like the column march, by issue (65 % of cycles on 720x120x60, 10
// grains, 16 warps per SM by registers) and the FP64 pipe (48 %).  720x360x60, 10
// grains, ash in every cell: 1.26 -> 0.70 ms a sweep against the warp-row kernel,
// whose lanes pass each value on through shared-memory rings (188 instructions a
// cell against 97).
// ---------------------------------------------------------------------------
constexpr int AXM_WARPS = 2;
constexpr int AXM_BUF = 32 * 8 * 8;                    // bytes of a chunk
constexpr int AXM_WARP_B = 5 * AXM_BUF;                // 3 concentration and 2 wind buffers
constexpr int AXM_SMEM = 512 + 512 + AXM_WARPS * AXM_WARP_B;  // barriers, room to align, buffers

template <int LIM, bool PER>
__global__ void __launch_bounds__(32 * AXM_WARPS, ACT_MINB) k_advect_xm(
    const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tv,
    const __grid_constant__ CUtensorMap to, Layout L, Box box, RowCover cov, int nocycle, double eps, int nseg, int seg,
    const double *__restrict__ cin, double *__restrict__ cout, const double *__restrict__ vel, Geo3 sig, Geo3 dtvt,
    const int32_t *__restrict__ aloft, DevScalars *sc, double *__restrict__ out1, double *__restrict__ out2) {
  extern __shared__ unsigned char axm_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned char *const sm = axm_smem + ((512u - (smem_u32(axm_smem) & 511u)) & 511u);  // the swizzle's period
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm) + 2 * wid;
  unsigned char *const qbuf = sm + 512 + wid * AXM_WARP_B, *const vbuf = qbuf + 3 * AXM_BUF;
  const unsigned t = blockIdx.x * AXM_WARPS + wid, ns = L.ns, rr = t / ns, rs = rr / (unsigned)cov.ntile;
  if (rs >= (unsigned)nseg) return;  // whole warps only; no block barrier below
  const int g = (int)(t - rr * ns);
  int r0, nrows;  // the tile's first row, the end of its run of rows
  cov.tile((int)(rr - rs * (unsigned)cov.ntile), &r0, &nrows);
  const int s0 = cov.x0 + (int)rs * seg;
  const int n = L.nx, s1 = min(cov.x1, s0 + seg - 1);
  const int r = min(r0 + lane, nrows - 1);
  const int j = r % L.ny + 1, k = r / L.ny + 1;
  const int rmin = box.imin, rmax = box.imax;
  const bool al = r0 + lane < nrows && j >= box.jmin && j <= box.jmax && k >= box.kmin && k <= box.kmax &&
                  aloft[g] != 0;
  const long grow = (long)g * L.ny * L.nz;  // this grain's first row in the level
  double *const po = cout + (grow + r0) * L.P;
  auto zero = [&](int ca, int cb) {   // cells ca..cb of the tile's rows: the reference leaves zeros
    for (int row = 0; row < min(32, nrows - r0); row++)
      for (int c = ca + lane; c <= cb; c += 32) po[(long)row * L.P + (c - 1)] = 0.0;
  };
  const int c0 = max(s0, rmin), c1 = min(s1, rmax);  // the cells marched
  if (c0 > c1 || !__any_sync(0xffffffffu, al)) {
    zero(s0, s1);
    return;
  }
  const int t0 = (c0 - s0) >> 3, t1 = (c1 - s0) >> 3;
  zero(s0, s0 + 8 * t0 - 1);
  zero(s0 + 8 * t1 + 8, s1);
  auto issue = [&](int c) {  // chunk c; its concentration buffer was stored from two chunks ago
    if (lane == 0) {
      uint64_t *b = &bar[c & 1];
      bulk_wait_read1();
      mbar_arrive_expect_tx(b, 2u * AXM_BUF);
      tma_load_2d(qbuf + (c % 3) * AXM_BUF, &tq, b, s0 + 1 + 8 * c, (int)(grow + r0));
      tma_load_2d(vbuf + (c & 1) * AXM_BUF, &tv, b, s0 + 1 + 8 * c, r0);
    }
  };
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
  }
  __syncwarp();
  issue(t0);
  const double *const pv = vel + (long)r * L.P;
  const double *const pq = cin + (grow + r) * L.P;
  // ghost-aware loads (Set_BC(1): zero or wrapped concentration, edge or wrapped winds)
  auto qload = [&](int c) -> double {
    if (c < rmin - 2 || c > rmax + 2) return 0.0;
    if (c >= 1 && c <= n) return pq[c - 1];
    return PER ? pq[(c < 1 ? c + n : c - n) - 1] : 0.0;
  };
  auto vload = [&](int c) -> double {
    if (PER) return pv[(c < 1 ? c + n : c > n ? c - n : c) - 1];
    return pv[(c < 1 ? 1 : c > n ? n : c) - 1];
  };
  // sigma and dt/kappa of the row
  const double sg = sig.p[(long)(j + 1) * sig.sj + (long)(k + 1) * sig.sk], hs = 0.5 * sg;
  const double dtv = dtvt.p[(long)(j + 1) * dtvt.sj + (long)(k + 1) * dtvt.sk];
  // ---- interface c0 and the window at c0 -------------------------------------
  March m;
  {
    m.q0 = qload(c0);
    m.q1 = qload(c0 + 1);
    const double qm1 = qload(c0 - 1), qm2 = qload(c0 - 2);
    m.d0 = m.q0 - qm1;
    m.d1 = m.q1 - m.q0;
    const double vm2 = vload(c0 - 2), vm1 = vload(c0 - 1), v0 = vload(c0);
    m.vB = vload(c0 + 1);
    const double usm1 = 0.5 * (vm2 + vm1) * sg;
    const double usA = 0.5 * (vm1 + v0) * sg;
    m.us = 0.5 * (v0 + m.vB) * sg;
    const double dm = qm1 - qm2;
    const Iface f = make_iface(usm1, usA, m.us, dtv, true, true);
    m.fss0 = fss_select<LIM>(dm, m.d0, m.d1, f.up, f.cf, true, eps, nocycle);
    m.fsr0 = f.usp * m.d0;
    m.fsr0 = m.fsr0 + m.q0 * f.divm;
    if (!PER && c0 == 1 && al) {  // the low outflow, cell 0
      double fsl = f.usm * m.d0;
      fsl = fsl + qm1 * f.divp;
      double fsr = pos_part(usm1) * dm;
      fsr = fsr + qm1 * (neg_part(usA) - neg_part(usm1));
      out1[grow + r] += cell_update(dtv, fsl, fsr, m.fss0, 0.0);
    }
    m.upA = pos_part(usA);
    m.upB = pos_part(m.us);
    m.unB = neg_part(m.us);
  }
  const bool nocyc = nocycle != 0;
  const int eps_hi = nocyc ? 0 : __double2hiint(eps);  // |d| < eps for certain, by its high word alone
  // this lane's row of a buffer: cells 2p, 2p+1 at pair(p), cell e at cell(e)
  const int row_b = lane << 6, row_s = ((lane >> 1) & 3) << 4;
  auto pair = [&](unsigned char *b, int p) { return reinterpret_cast<double2 *>(b + row_b + ((p << 4) ^ row_s)); };
  auto cell = [&](unsigned char *b, int e) { return reinterpret_cast<double *>(pair(b, e >> 1)) + (e & 1); };
  auto step = [&](auto quiet, auto any, double q2, double vn) {
    const double q0 = m.q0;
    const double sum =
        march_step<LIM, decltype(quiet)::value, decltype(any)::value>(m, q2, q2 - m.q1, vn, hs, dtv, eps, nocyc);
    const double upd = dtv * sum;
    return q0 - upd;
  };
  auto two = [&](auto quiet, unsigned char *qb, unsigned char *vb, int p) {  // cells 2p, 2p+1 of the chunk
    double2 *q = pair(qb, p);
    const double2 x = *q, v = *pair(vb, p);
    double2 y;
    y.x = step(quiet, FalseT{}, x.x, v.x);
    y.y = step(quiet, FalseT{}, x.y, v.y);
    *q = y;
  };
  const bool whole = r0 + 32 <= nrows, all_al = __all_sync(0xffffffffu, al);
  uint32_t ph = 0u;
  for (int c = t0; c <= t1; c++) {
    if (c < t1) issue(c + 1);
    if (!mbar_wait(&bar[c & 1], (ph >> (c & 1)) & 1u)) {
      if (lane == 0) {
        raise_error(sc, A3G_ERR_TIMEOUT, 4);
        bulk_wait0();
      }
      return;
    }
    ph ^= 1u << (c & 1);
    unsigned char *const qb = qbuf + (c % 3) * AXM_BUF, *const vb = vbuf + (c & 1) * AXM_BUF;
    const int cb = s0 + 8 * c;                       // slot e: the step of cell cb+e, holding cell cb+e+2
    const int e0 = max(c0 - cb, 0), e1 = min(c1 - cb, 7);
    if (cb + 9 > n) {                                // the ghosts beyond the row's end
#pragma unroll
      for (int x = n + 1; x <= n + 2; x++) {
        const int e = x - cb - 2;
        if (e >= 0 && e < 8) {
          if (PER) *cell(qb, e) = qload(x);
          *cell(vb, e) = vload(x);
        }
      }
    }
    // the differences the chunk's interfaces limit: d1 and the first 7 new ones;
    // and whether every wind they take is a number: their sum is
    int top = __double2hiint(m.d1) & 0x7fffffff;
    double sum = m.vB + m.us;
    {
      double prev = m.q1;
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const double2 x = *pair(qb, p), v = *pair(vb, p);
        sum = sum + (v.x + v.y);
        top = max(top, __double2hiint(x.x - prev) & 0x7fffffff);
        if (p < 3) top = max(top, __double2hiint(x.y - x.x) & 0x7fffffff);
        prev = x.y;
      }
    }
    const bool quiet = LIM == A3G_LIM_NONE || __all_sync(0xffffffffu, top < eps_hi || !al);
    const bool any = __any_sync(0xffffffffu, al && !finite_bits(sum));
    if (e0 == 0 && e1 == 7 && !any) {
      if (quiet) {
        for (int p = 0; p < 4; p++) two(TrueT{}, qb, vb, p);
      } else {
        for (int p = 0; p < 4; p += ACT_U / 2) {
#pragma unroll
          for (int u = 0; u < ACT_U / 2; u++) two(FalseT{}, qb, vb, p + u);
        }
      }
    } else {
      for (int e = 0; e < 8; e++) {
        double *q = cell(qb, e);
        double y = 0.0;  // outside the box
        if (e >= e0 && e <= e1) y = step(FalseT{}, TrueT{}, *q, *cell(vb, e));
        *q = y;
      }
    }
    if (!all_al && !al) {
#pragma unroll
      for (int p = 0; p < 4; p++) *pair(qb, p) = make_double2(0.0, 0.0);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (whole) {
      if (lane == 0) {
        tma_store_2d(&to, qb, cb - 1, (int)(grow + r0));
        bulk_commit();
      }
    } else {
      const int e = lane & 7, x = cb + e;
#pragma unroll
      for (int h = 0; h < 8; h++) {
        const int row = 4 * h + (lane >> 3);
        if (r0 + row < nrows && x <= n)
          po[(long)row * L.P + (x - 1)] = *reinterpret_cast<const double *>(
              qb + (row << 6) + ((((e >> 1) ^ ((row >> 1) & 3)) << 4) | ((e & 1) << 3)));
      }
      __syncwarp();
    }
  }
  // cell n+1: interface n+2 lies outside the box and carries nothing
  if (!PER && al && s1 == n && rmax == n) out2[grow + r] += cell_update(dtv, 0.0, m.fsr0, 0.0, m.fss0);
  if (lane == 0) bulk_wait0();
}

// Launches the TMA-fed row march; false when its conditions do not hold.
template <int LIM>
static bool launch_advect_xm(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  if (along<0>(ctx->snx) != 0 || along<0>(ctx->dtv) != 0) return false;
  CUtensorMap tq, tv, to;
  if (!tensor_map(ctx, ctx->c0, TM_QROWS, &tq) || !tensor_map(ctx, ctx->vx, TM_VROWS, &tv) ||
      !tensor_map(ctx, ctx->c1, TM_QROWS, &to))
    return false;
  const RowCover cov = row_cover(L, cover_box(ctx));
  const int nxc = cov.x1 - cov.x0 + 1;
  const long nlw = (long)cov.ntile * L.ns;
  const int want = march_segments(nxc, nlw);
  const int seg = (nxc + want - 1) / want + 7 & ~7;  // whole chunks
  const int nseg = (nxc + seg - 1) / seg;
  const unsigned blocks = (unsigned)((nlw * nseg + AXM_WARPS - 1) / AXM_WARPS);
#define A3G_XM(PER_)                                                                                           \
  k_advect_xm<LIM, PER_><<<blocks, 32 * AXM_WARPS, AXM_SMEM, ctx->stream>>>(                                    \
      tq, tv, to, L, ctx->box, cov, ctx->prm.nocycle, ctx->prm.eps_thresh, nseg, seg, ctx->c0, ctx->c1, ctx->vx,     \
      ctx->snx, ctx->dtv, ctx->aloft, ctx->sc, ctx->out_yz1, ctx->out_yz2)
  if (ctx->grid.periodic) A3G_XM(true); else A3G_XM(false);
#undef A3G_XM
  return true;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// warps of k_advect_march in segments of 96 cells
template <int DIR>
static inline long march_warps(const Layout &L, int gc) {
  const long lines = (long)((((DIR == 0) ? L.ny : L.nx) + 31) / 32) * ((DIR == 2) ? L.ny : L.nz);
  return lines * ((L.ns + gc - 1) / gc) * ((((DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz) + 95) / 96);
}

template <int DIR, int LIM, int GC, bool PER, bool TOPO = false>
static void launch_march_gc(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  const int na = (DIR == 0) ? L.ny : L.nx;
  const int nother = (DIR == 2) ? L.ny : L.nz;
  // segments of about 96 cells (whole lines when they are short); over terrain
  // of 48 along rows, and along columns where 96 give an SM less than 32 warps
  const int len = TOPO && (DIR == 0 || march_warps<DIR>(L, GC) < 148 * 32) ? 48 : 96;
  const int nseg = (n + len - 1) / len;
  const int seg = (n + nseg - 1) / nseg;
  const int ngroups = (L.ns + GC - 1) / GC;
  dim3 grid(((na + 31) / 32) * ngroups, (nother + 3) / 4, (n + seg - 1) / seg);
  const long n2 = (long)(L.nx + 4) * (L.ny + 4);
  const double *deld = TOPO ? ctx->topo_buf + ((DIR == 0) ? 2 : 3) * n2 : nullptr;
  k_advect_march<DIR, LIM, GC, PER, TOPO><<<grid, dim3(32, 4), 0, ctx->stream>>>(
      L, ctx->box, ctx->prm.nocycle, ctx->prm.eps_thresh, seg, ngroups, ctx->c0, ctx->c1,
      dir_vel(ctx, DIR), dir_vghost(ctx, DIR), deld, ctx->vf,
      (DIR == 0) ? ctx->snx : (DIR == 1) ? ctx->sny : ctx->snz, ctx->dtv, ctx->aloft, ctx->sc,
      (DIR == 0) ? ctx->out_yz1 : (DIR == 1) ? ctx->out_xz1 : ctx->out_xy1,
      (DIR == 0) ? ctx->out_yz2 : (DIR == 1) ? ctx->out_xz2 : ctx->out_xy2);
}

template <int DIR, int LIM, int V, bool PER>
static void launch_block_v(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  const int nblk = (n + V - 1) / V;
  dim3 grid;
  if (DIR == 0) grid = dim3((nblk + 31) / 32, (L.ny + 3) / 4, L.nz * L.ns);
  else grid = dim3((L.nx + 31) / 32, (nblk * ((DIR == 1) ? L.nz : L.ny) + 3) / 4, L.ns);
  const Geo3 &sg = (DIR == 0) ? ctx->snx : (DIR == 1) ? ctx->sny : ctx->snz;
  const bool lc = along<DIR>(sg) == 0 && along<DIR>(ctx->dtv) == 0 && (DIR != 2 || ctx->vf.sk == 0);
#define A3G_BLK(LC_)                                                                                  \
  k_advect_block<DIR, LIM, V, PER, LC_><<<grid, dim3(32, 4), 0, ctx->stream>>>(                       \
      L, ctx->box, ctx->prm.nocycle, ctx->prm.eps_thresh, nblk, ctx->c0, ctx->c1,                     \
      dir_vel(ctx, DIR), dir_vghost(ctx, DIR), ctx->vf, sg, ctx->dtv, ctx->aloft, ctx->sc,            \
      (DIR == 0) ? ctx->out_yz1 : (DIR == 1) ? ctx->out_xz1 : ctx->out_xy1,                           \
      (DIR == 0) ? ctx->out_yz2 : (DIR == 1) ? ctx->out_xz2 : ctx->out_xy2)
  if (lc) A3G_BLK(true); else A3G_BLK(false);
#undef A3G_BLK
}

template <int DIR, int LIM>
static void launch_dir_lim(a3g_ctx *ctx) {
  const bool per = (DIR == 0) && ctx->grid.periodic;
  const int variant = ctx->tune_advect[DIR];
  if constexpr (DIR != 2) {
    // ZScaling_ID 2: the DelD*onD_cc terms live in the marching kernel only.
    // Along x two grains a thread share the row's winds, unless a missing second
    // one makes a sixth of the work or more; along y a grain a thread.  x with
    // segments of 48 and two grains, with 48 and one, and with 96 and two, us a
    // sweep of 201x151x41: 3 grains 89, 86, 122; 5 grains 135, 131, 148; 6: 146,
    // 161, 156; 8: 186, 200, 217; 10: 226, 246, 232; 402x301x50, 4 grains: 381,
    // 407, 403; 150x120x30, 2 grains: 35, 33, 61; 97x83x25, 8: 42, 54, 56.  y with
    // one and with two (segments of 96): 402x301x50, 10 grains, 746, 825;
    // 201x151x41, 5 grains, 102, 142.
    if (ctx->topo_on && ctx->prm.zscaling_id == 2) {
      if constexpr (DIR == 0) {
        const bool g2 = ctx->L.ns % 2 == 0 || ctx->L.ns > 6;
        if (per && g2) launch_march_gc<DIR, LIM, 2, true, true>(ctx);
        else if (per) launch_march_gc<DIR, LIM, 1, true, true>(ctx);
        else if (g2) launch_march_gc<DIR, LIM, 2, false, true>(ctx);
        else launch_march_gc<DIR, LIM, 1, false, true>(ctx);
      } else {
        launch_march_gc<DIR, LIM, 1, false, true>(ctx);
      }
      return;
    }
  }
  if constexpr (DIR == 0) {
    if (variant == 3) {
      launch_advect_xt<LIM>(ctx);
      return;
    }
    // A row per lane needs rows: with few and short ones a warp per row is
    // sooner done (50x50x23, 1 grain: 6.2 us a sweep, the march 8.2; 60x80x30, 2
    // grains: 9.3, 10.4; 200x100x20, 1 grain: 10.3, 12.3; but 400x3x40, 2 grains:
    // 17.9, 10.3; 30x200x20, 2 grains: 12.3, 10.3; 100x100x40, 2 grains: 18, 14).
    const bool few_rows = ctx->L.nx <= 224 && (long)ctx->L.ny * ctx->L.nz * ctx->L.ns < 5000;
    if (variant == 5 && !few_rows && launch_advect_xm<LIM>(ctx)) return;
    if (variant == 4 || variant == 5) {
      launch_advect_xw<LIM>(ctx, variant == 5);
      return;
    }
  }
  if constexpr (DIR != 0) {
    if (variant == 5) {
      launch_col<DIR, LIM>(ctx);
      return;
    }
    if (variant == 6) {
      if (!launch_colt<DIR, LIM>(ctx)) launch_block_v<DIR, LIM, 4, false>(ctx);
      return;
    }
  }
  if (variant == 1) {
    if (per) launch_block_v<DIR, LIM, 4, true>(ctx);
    else launch_block_v<DIR, LIM, 4, false>(ctx);
    return;
  }
  if (variant == 2) {
    if (per) launch_block_v<DIR, LIM, 8, true>(ctx);
    else launch_block_v<DIR, LIM, 8, false>(ctx);
    return;
  }
  if (ctx->L.ns >= 2) {
    if (per) launch_march_gc<DIR, LIM, 2, true>(ctx);
    else launch_march_gc<DIR, LIM, 2, false>(ctx);
  } else {
    if (per) launch_march_gc<DIR, LIM, 1, true>(ctx);
    else launch_march_gc<DIR, LIM, 1, false>(ctx);
  }
}

#define A3G_LIM_SWITCH(FN, ...)                                      \
  switch (ctx->prm.limiter) {                                        \
    case A3G_LIM_NONE: FN<__VA_ARGS__ A3G_LIM_NONE>(ctx); break;     \
    case A3G_LIM_LAXWEN: FN<__VA_ARGS__ A3G_LIM_LAXWEN>(ctx); break; \
    case A3G_LIM_BW: FN<__VA_ARGS__ A3G_LIM_BW>(ctx); break;         \
    case A3G_LIM_FROMM: FN<__VA_ARGS__ A3G_LIM_FROMM>(ctx); break;   \
    case A3G_LIM_MINMOD: FN<__VA_ARGS__ A3G_LIM_MINMOD>(ctx); break; \
    case A3G_LIM_MC: FN<__VA_ARGS__ A3G_LIM_MC>(ctx); break;         \
    default: FN<__VA_ARGS__ A3G_LIM_SUPERBEE>(ctx); break;           \
  }

}  // namespace a3g
