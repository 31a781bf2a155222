// k_advect.cu -- dt/kappa of the step and the discrete adjoint of the advection
// sweeps.  The forward sweeps are in k_advect.cuh.
#include "k_advect.cuh"
#include "lim_coef.cuh"

namespace a3g {

// dt/kappa of the current step on the compressed kappa layout (the reference
// forms dt_vol_cc = dt/kap_cc in every row, :155; the quotient is the same).
__global__ void k_dtv(const double *__restrict__ kap, long n, const DevScalars *__restrict__ sc,
                      double *__restrict__ dtv) {
  const double dt = sc->dt;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
    dtv[t] = dt / kap[t];
}

int refresh_dtv(a3g_ctx *ctx) {
  // recomputed whenever the step's dt may have changed
  if (ctx->dtv_valid && ctx->dtv_stamp == ctx->dt_stamp) return A3G_OK;
  const long n = (long)ctx->kappa_len;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  tbegin(ctx, A3G_K_OTHER);
  k_dtv<<<blocks, 256, 0, ctx->stream>>>(ctx->kappa.p, n, ctx->sc, const_cast<double *>(ctx->dtv.p));
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  ctx->dtv_valid = true;
  ctx->dtv_stamp = ctx->dt_stamp;
  return A3G_OK;
}

// ===========================================================================
// Discrete adjoint of one advection sweep (no counterpart in the reference).
//
// With the limiter branches fixed by the sweep's input state q, the limited
// slope is ldq = a*dq + b*dqu, so the sweep is linear; this kernel applies
// its transpose to lam (the adjoint of the sweep's output).  It is a gather:
// one thread per cell-grain, lanes along x in every direction (coalesced),
// each thread re-deriving the four interfaces m-1..m+2 that its cell feeds
// (limiter branch, flux-area terms) from q, winds and geometry.  With t(i) =
// -dt/kappa(i)*lam_u(i) (lam_u = lam inside the line, the deposit adjoint
// at the z bottom outflow, 0 at the other outflows):
//   lam_fsr(I) = t(I), lam_fsl(I) = t(I-1), lam_fss(I) = t(I-1) - t(I)
//   e(J) = 0.5|us|(1 - dtv|us|) * lam_fss(J)       (active fss interfaces)
//   lam_dq(I) = max(0,us)lam_fsr(I) + min(0,us)lam_fsl(I) + a(I)e(I)
//               + b(I+1)e(I+1) [us(I+1) > 0] + b(I-1)e(I-1) [us(I-1) <= 0]
//   lam_q(m)  = lam(m) + divu_m(m)lam_fsr(m) + divu_p(m+1)lam_fsl(m+1)
//               + lam_dq(m) - lam_dq(m+1)
// Ghost cells of Set_BC(1) are zero (their adjoint is dropped) except x-
// periodic wraps, whose adjoint is added back to the wrapped cells.  Full box
// only (the subgrid box depends on the state).
// ===========================================================================

template <int DIR, int LIM, bool PER>
__global__ void __launch_bounds__(256) k_adj_advect(Layout L, int nocycle, double eps,
                                                    const double *__restrict__ cq,
                                                    const double *__restrict__ lin,
                                                    double *__restrict__ lout,
                                                    const double *__restrict__ vel, Geo4 vf, Geo3 sig,
                                                    Geo3 dtvt, const int32_t *__restrict__ aloft,
                                                    const double *__restrict__ lam_lo) {
  const int i = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int k = (int)(blockIdx.z % L.nz) + 1;
  const int g = (int)(blockIdx.z / L.nz);
  if (i > L.nx || j > L.ny) return;
  const long cell = L.cell(i, j, k);
  const long gb = (long)g * L.PG;
  if (!aloft[g]) {
    lout[gb + cell] = 0.0;
    return;
  }
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  const int m = (DIR == 0) ? i : (DIR == 1) ? j : k;
  const long st = (DIR == 0) ? 1 : (DIR == 1) ? L.P : L.PY;
  const long lb = cell - (long)(m - 1) * st;  // sweep index 1 of this line
  const int la = (DIR == 0) ? j : i, lo_ = (DIR == 2) ? j : k;
  const LineGeo gsig = line_of<DIR>(sig, la, lo_);
  const LineGeo gdtv = line_of<DIR>(dtvt, la, lo_);
  const double *pq = cq + gb + lb;
  const double *pl = lin + gb + lb;
  const double *pv = vel + lb;
  const double *pvf = vf.p + (long)(i + 1) * vf.si + (long)(j + 1) * vf.sj + (long)g * vf.sg;
  auto wrap = [&](int c) { return c < 1 ? c + n : (c > n ? c - n : c); };
  auto Q = [&](int c) -> double {
    if (c < -1 || c > n + 2) return 0.0;
    if (c >= 1 && c <= n) return pq[(long)(c - 1) * st];
    return PER ? pq[(long)(wrap(c) - 1) * st] : 0.0;
  };
  auto V = [&](int c) -> double {
    const int cl = PER ? wrap(c) : (c < 1 ? 1 : (c > n ? n : c));
    double v = pv[(long)(cl - 1) * st];
    if (DIR == 2) v = v + pvf[(long)(cl + 1) * vf.sk];
    return v;
  };
  auto US = [&](int I) -> double {  // usig(I), zero outside [0, n+1]
    if (I < 0 || I > n + 1) return 0.0;
    return 0.5 * (V(I - 1) + V(I)) * gsig.at(I);
  };
  auto T = [&](int c) -> double {  // t(c) = -dtv(c)*lam_u(c)
    if (c < 0 || c > n + 1) return 0.0;
    double lu = 0.0;
    if (c >= 1 && c <= n) lu = pl[(long)(c - 1) * st];
    else if (c == 0 && lam_lo) lu = lam_lo[(long)g * L.nx * L.ny + (long)(j - 1) * L.nx + (i - 1)];
    return -(gdtv.at(c) * lu);
  };
  auto DQ = [&](int I) -> double { return (I < 0 || I > n + 2) ? 0.0 : Q(I) - Q(I - 1); };
  // lam_q at sweep index c (an interior cell or a ghost)
  auto lam_at = [&](int c) -> double {
    double us[6], tt[5], dq[6];
#pragma unroll
    for (int d = 0; d < 6; d++) us[d] = US(c - 2 + d);  // us(c-2 .. c+3)
#pragma unroll
    for (int d = 0; d < 5; d++) tt[d] = T(c - 2 + d);   // t(c-2 .. c+2)
#pragma unroll
    for (int d = 0; d < 6; d++) dq[d] = DQ(c - 2 + d);  // dq(c-2 .. c+3)
    // interfaces J = c-1 .. c+2 (index r = J-c+1): a*e, b*e, upwind side
    double ea[4], eb[4];
    bool up[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int J = c - 1 + r;
      const double u = us[r + 1];
      up[r] = u > 0.0;
      ea[r] = 0.0;
      eb[r] = 0.0;
      if (LIM != A3G_LIM_NONE && J >= 1 && J <= n + 1) {
        const double dqJ = dq[r + 1];
        if (nocycle || !(fabs(dqJ) <= eps)) {
          const double aus = fabs(u);
          const double w = 0.5 * aus * (1.0 - gdtv.at(J) * aus);
          const double e = w * (tt[r] - tt[r + 1]);  // t(J-1) - t(J)
          double a, b;
          lim_coef<LIM>(dqJ, up[r] ? dq[r] : dq[r + 2], eps, a, b);
          ea[r] = a * e;
          eb[r] = b * e;
        }
      }
    }
    // lam_dq(c) (r = 1) and lam_dq(c+1) (r = 2)
    double ldq[2];
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const int I = c + s, r = 1 + s;
      double v = 0.0;
      if (I >= 0 && I <= n + 2) {
        const double u = us[r + 1];
        const double lfsr = tt[r + 1];                          // t(I)
        const double lfsl = (I <= n + 1) ? tt[r] : 0.0;         // t(I-1)
        v = dmx(0.0, u) * lfsr + dmn(0.0, u) * lfsl + ea[r];
        if (up[r + 1]) v = v + eb[r + 1];
        if (!up[r - 1]) v = v + eb[r - 1];
      }
      ldq[s] = v;
    }
    double lam = (c >= 1 && c <= n) ? pl[(long)(c - 1) * st] : 0.0;
    if (c >= 0 && c <= n + 1) {  // divu_m(c)*lam_fsr(c)
      const double divm = dmn(0.0, us[3]) - dmn(0.0, us[2]);
      lam = lam + divm * tt[2];
    }
    if (c + 1 >= 0 && c + 1 <= n + 1) {  // divu_p(c+1)*lam_fsl(c+1)
      const double divp = dmx(0.0, us[3]) - dmx(0.0, us[2]);
      lam = lam + divp * tt[2];
    }
    return lam + ldq[0] - ldq[1];
  };
  double lam = lam_at(m);
  if (PER) {
    if (m <= 2) lam = lam + lam_at(m + n);
    if (m >= n - 1) lam = lam + lam_at(m - n);
  }
  lout[gb + cell] = lam;
}

// Block form of k_adj_advect: a thread takes V consecutive cells of a line
// and forms each of the V+3 interfaces they read (c0-1 .. c0+V+1) once,
// instead of the four a cell-per-thread gather forms for every cell; the
// expressions and their order are lam_at's, so the results are the same
// bits.  Runs where the marches below do not.  Not x-periodic (the wrapped ghosts stay with the gather kernel).
// DIR 0: lanes are consecutive blocks along i; DIR 1, 2: lanes along i.
template <int DIR, int LIM, int V, bool CK>
__device__ __forceinline__ void adj_block_body(const Layout &L, int nocycle, double eps, int n, int c0, long st,
                                               const double *__restrict__ pq, const double *__restrict__ pl,
                                               double *__restrict__ po, const double *__restrict__ pv,
                                               const double *__restrict__ pvf, long vfs, const LineGeo &gsig,
                                               const LineGeo &gdtv, double lam_lo0) {
  auto Q = [&](int c) -> double {
    if (CK && (c < 1 || c > n)) return 0.0;
    return pq[(long)(c - 1) * st];
  };
  auto VV = [&](int c) -> double {
    const int cl = CK ? (c < 1 ? 1 : (c > n ? n : c)) : c;
    double v = pv[(long)(cl - 1) * st];
    if (DIR == 2) v = v + pvf[(long)(cl + 1) * vfs];
    return v;
  };
  auto T = [&](int c) -> double {  // t(c) = -dtv(c)*lam_u(c)
    if (CK && (c < 0 || c > n + 1)) return 0.0;
    double lu = 0.0;
    if (!CK || (c >= 1 && c <= n)) lu = pl[(long)(c - 1) * st];
    else if (c == 0 && DIR == 2) lu = lam_lo0;
    return -(gdtv.at(c) * lu);
  };
  // window: q(c0-3 .. c0+V+2), vel(c0-3 .. c0+V+2), t(c0-2 .. c0+V+1)
  double q[V + 6], vv[V + 6], tt[V + 4];
#pragma unroll
  for (int m = 0; m < V + 6; m++) {
    q[m] = Q(c0 - 3 + m);
    vv[m] = VV(c0 - 3 + m);
  }
#pragma unroll
  for (int m = 0; m < V + 4; m++) tt[m] = T(c0 - 2 + m);
  // dq(c0-2 .. c0+V+2): dq(I) = q(I) - q(I-1), zero outside [0, n+2]
  double dq[V + 5];
#pragma unroll
  for (int m = 0; m < V + 5; m++) {
    const int I = c0 - 2 + m;
    dq[m] = (CK && (I < 0 || I > n + 2)) ? 0.0 : q[m + 1] - q[m];
  }
  // interfaces J = c0-1+r, r = 0 .. V+2: usig, upwind side, a*e, b*e
  double us[V + 3], ea[V + 3], eb[V + 3];
  bool up[V + 3];
#pragma unroll
  for (int r = 0; r < V + 3; r++) {
    const int J = c0 - 1 + r;
    const double u = (CK && (J < 0 || J > n + 1)) ? 0.0 : 0.5 * (vv[r + 1] + vv[r + 2]) * gsig.at(J);
    us[r] = u;
    up[r] = u > 0.0;
    ea[r] = 0.0;
    eb[r] = 0.0;
    if (LIM != A3G_LIM_NONE && (!CK || (J >= 1 && J <= n + 1))) {
      const double dqJ = dq[r + 1];
      if (nocycle || !(fabs(dqJ) <= eps)) {
        const double aus = fabs(u);
        const double w = 0.5 * aus * (1.0 - gdtv.at(J) * aus);
        const double e = w * (tt[r] - tt[r + 1]);  // t(J-1) - t(J)
        double a, b;
        lim_coef<LIM>(dqJ, up[r] ? dq[r] : dq[r + 2], eps, a, b);
        ea[r] = a * e;
        eb[r] = b * e;
      }
    }
  }
#pragma unroll
  for (int v = 0; v < V; v++) {
    const int c = c0 + v;
    if (CK && c > n) break;
    double ldq[2];
#pragma unroll
    for (int s2 = 0; s2 < 2; s2++) {
      const int I = c + s2, r = v + 1 + s2;
      double val = 0.0;
      if (!CK || (I >= 0 && I <= n + 2)) {
        const double u = us[r];
        const double lfsr = tt[v + 2 + s2];                              // t(I)
        const double lfsl = (!CK || I <= n + 1) ? tt[v + 1 + s2] : 0.0;  // t(I-1)
        val = dmx(0.0, u) * lfsr + dmn(0.0, u) * lfsl + ea[r];
        if (up[r + 1]) val = val + eb[r + 1];
        if (!up[r - 1]) val = val + eb[r - 1];
      }
      ldq[s2] = val;
    }
    double lam = pl[(long)(c - 1) * st];
    const double divm = dmn(0.0, us[v + 2]) - dmn(0.0, us[v + 1]);
    lam = lam + divm * tt[v + 2];
    const double divp = dmx(0.0, us[v + 2]) - dmx(0.0, us[v + 1]);
    lam = lam + divp * tt[v + 2];
    po[(long)(c - 1) * st] = lam + ldq[0] - ldq[1];
  }
}

template <int DIR, int LIM, int V>
__global__ void __launch_bounds__(128) k_adj_advect_blk(Layout L, int nocycle, double eps, int nblk,
                                                        const double *__restrict__ cq,
                                                        const double *__restrict__ lin,
                                                        double *__restrict__ lout,
                                                        const double *__restrict__ vel, Geo4 vf, Geo3 sig,
                                                        Geo3 dtvt, const int32_t *__restrict__ aloft,
                                                        const double *__restrict__ lam_lo) {
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  int a, o, blk, g;  // lane index (i or j), other index, block, grain (k_advect_block's mapping)
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
  const long gb = (long)g * L.PG;
  double *po = lout + gb + base;
  if (!aloft[g]) {
    for (int v = 0; v < V; v++)
      if (c0 + v <= n) po[(long)(c0 + v - 1) * st] = 0.0;
    return;
  }
  const int i = (DIR == 0) ? 1 : a, j = (DIR == 1) ? 1 : (DIR == 0 ? a : o);
  const LineGeo gsig = line_of<DIR>(sig, a, o);
  const LineGeo gdtv = line_of<DIR>(dtvt, a, o);
  const double *pvf = vf.p + (long)(i + 1) * vf.si + (long)(j + 1) * vf.sj + (long)g * vf.sg;
  const double lam_lo0 = (DIR == 2 && lam_lo && c0 <= 2) ? lam_lo[(long)g * L.nx * L.ny + (long)(j - 1) * L.nx + (i - 1)]
                                                         : 0.0;
  const bool fast = c0 - 3 >= 1 && c0 + V + 2 <= n;
  if (fast)
    adj_block_body<DIR, LIM, V, false>(L, nocycle, eps, n, c0, st, cq + gb + base, lin + gb + base, po, vel + base,
                                       pvf, vf.sk, gsig, gdtv, lam_lo0);
  else
    adj_block_body<DIR, LIM, V, true>(L, nocycle, eps, n, c0, st, cq + gb + base, lin + gb + base, po, vel + base,
                                      pvf, vf.sk, gsig, gdtv, lam_lo0);
}

// ---------------------------------------------------------------------------
// Marched form of the adjoint sweep (the default; not x-periodic): a lane walks
// its line and forms each interface once, in lam_at's expressions, so the
// results are the same bits.  Reading cell x completes interface J = x-1
// (which needs q(J+1)), then lam_dq(J-1), then lam_q(J-2).
// ---------------------------------------------------------------------------
struct AdjMarch {
  double q, d0, dm;        // q(J), dq(J), dq(J-1)
  double v, vm;            // vel(J), vel(J-1)
  double lam, lamm, t;     // lam(J), lam(J-1), t(J-1)
  double pos, neg;         // max, min of 0 and usig(J-1)
  double e1, e2;           // b*e of J-1 and of J-2 where their upwind side is the right
  double base, ldq, L1;    // lam_dq(J-1) without its neighbours' terms, lam_dq(J-2), lam_q(J-2) without lam_dq
};

// Takes cell J+1 (its q, vel, lam) with sigma(J)/2 and dt/kappa(J); returns lam_q(J-2).
// ANY: the caller does not know that the winds are numbers.
template <int LIM, bool ANY>
__device__ __forceinline__ double adj_march_step(AdjMarch &m, double qx, double vx, double lx, double hs, double dtv,
                                                 double eps, int nocycle) {
  const double d1 = qx - m.q;
  const double us = (m.vm + m.v) * hs;
  const double p = ANY ? pos_part(us) : pos_bits(us), n = ANY ? neg_part(us) : neg_bits(us);
  const bool up = us > 0.0;
  const double tJ = -(dtv * m.lam);
  double ea = 0.0, eb = 0.0;
  if (LIM != A3G_LIM_NONE && (nocycle || !(fabs(m.d0) <= eps))) {
    const double aus = fabs(us);
    const double e = 0.5 * aus * (1.0 - dtv * aus) * (m.t - tJ);  // t(J-1) - t(J)
    double a, b;
    lim_coef<LIM>(m.d0, up ? m.dm : d1, eps, a, b);
    ea = a * e;
    eb = b * e;
  }
  const double ldq = m.base + (up ? eb : 0.0) + m.e2;  // lam_dq(J-1)
  const double out = m.L1 + m.ldq - ldq;
  m.L1 = m.lamm + (n - m.neg) * m.t + (p - m.pos) * m.t;
  m.base = p * tJ + n * m.t + ea;
  m.ldq = ldq;
  m.e2 = m.e1;
  m.e1 = up ? 0.0 : eb;
  m.pos = p;
  m.neg = n;
  m.lamm = m.lam;
  m.lam = lx;
  m.t = tJ;
  m.vm = m.v;
  m.v = vx;
  m.dm = m.d0;
  m.d0 = d1;
  m.q = qx;
  return out;
}

// State before cell x = s0 is taken (J = s0-1) from values by index.
template <class Q, class V, class T, class L>
__device__ __forceinline__ AdjMarch adj_march_start(int s0, Q q, V v, T t, L lam) {
  AdjMarch m;
  const double qa = q(s0 - 2);
  m.q = q(s0 - 1);
  m.d0 = m.q - qa;
  m.dm = qa - q(s0 - 3);
  m.v = v(s0 - 1);
  m.vm = v(s0 - 2);
  m.lam = lam(s0 - 1);
  m.lamm = 0.0;
  m.t = t(s0 - 2);
  m.pos = m.neg = m.e1 = m.e2 = m.base = m.ldq = m.L1 = 0.0;
  return m;
}

// Columns (y and z): k_advect_colt's mapping and chunks, with lam as a third
// array of the chunk.  140x120x40, 4 grains: y 48 -> 29 us, z 61 -> 29 us
// against blocks of four cells, which form 7 interfaces for 4 cells (and took
// a certified quotient for each).
constexpr int ADJ_WARPS = 2;
constexpr int ADJ_BUF_D = 3 * ACH * 32 + 2 * ACH;  // q, vel, lam; pairs (sigma/2, dt/kappa)

template <int DIR, int LIM>
__global__ void __launch_bounds__(32 * ADJ_WARPS, 8) k_adj_colt(
    const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tv,
    const __grid_constant__ CUtensorMap tl, Layout L, int nocycle, double eps, int nseg, int seg,
    const double *__restrict__ cq, const double *__restrict__ lin, double *__restrict__ lout,
    const double *__restrict__ vel, Geo4 vf, Geo3 sig, Geo3 dtvt, const int32_t *__restrict__ aloft, DevScalars *sc,
    const double *__restrict__ lam_lo) {
  extern __shared__ __align__(128) unsigned char adj_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t *bar = reinterpret_cast<uint64_t *>(adj_smem) + 2 * wid;
  double *wsm = reinterpret_cast<double *>(adj_smem + 128) + (long)wid * 2 * ADJ_BUF_D;
  const int nother = (DIR == 1) ? L.nz : L.ny;
  const int nti = (L.nx + 31) >> 5;
  const unsigned t = blockIdx.x * ADJ_WARPS + wid, ns = L.ns, rr = t / ns, ro = rr / (unsigned)nti;
  if (ro >= (unsigned)(nother * nseg)) return;  // whole warps only; no block barrier below
  const int g = (int)(t - rr * ns);
  const int it = (int)(rr - ro * (unsigned)nti);
  const int sg_ = (int)(ro / (unsigned)nother);
  const int o = (int)ro - sg_ * nother + 1;
  const int s0 = sg_ * seg + 1;
  const int a = (it << 5) + lane + 1;
  const bool valid = a <= L.nx;
  const int n = (DIR == 1) ? L.ny : L.nz;
  const int s1 = min(n, s0 + seg - 1);
  const int st = (DIR == 1) ? (int)L.P : (int)L.PY;
  const int ac = valid ? a : 1;
  const long base = (DIR == 1) ? L.cell(ac, 1, o) : L.cell(ac, o, 1);
  double *po = lout + (long)g * L.PG + base;
  if (!aloft[g]) {
    if (valid)
      for (int c = s0; c <= s1; c++) po[(c - 1) * st] = 0.0;
    return;
  }
  const LineGeo gsig = line_of<DIR>(sig, 1, o), gdtv = line_of<DIR>(dtvt, 1, o);  // constant along i
  // chunk k holds the cells s0+k*ACH .. and the geometry of the interfaces one before them
  const int nx_ = s1 + 3 - s0 + 1, nchunk = (nx_ + ACH - 1) / ACH;
  auto issue = [&](int k) {
    double *qb = wsm + (k & 1) * ADJ_BUF_D;
    const int X = s0 + k * ACH;
    if (lane == 0) {
      uint64_t *b = &bar[k & 1];
      mbar_arrive_expect_tx(b, 3u * ACH * 32u * 8u);
      const int y = (DIR == 1) ? X - 1 : o - 1, z = (DIR == 1) ? o - 1 : X - 1;
      tma_load_4d(qb, &tq, b, it << 5, y, z, g);
      tma_load_4d(qb + ACH * 32, &tv, b, it << 5, y, z, 0);
      tma_load_4d(qb + 2 * ACH * 32, &tl, b, it << 5, y, z, g);
    }
    const int J = X + lane - 1;
    if (lane < ACH && J <= n + 2)  // usig is zero outside interfaces 1 .. n+1
      reinterpret_cast<double2 *>(qb + 3 * ACH * 32)[lane] =
          make_double2(J >= 1 && J <= n + 1 ? 0.5 * gsig.at(J) : 0.0, gdtv.at(J));
  };
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
  }
  __syncwarp();
  issue(0);
  const double vf0 = (DIR == 2) ? vf.p[(long)g * vf.sg] : 0.0;  // one fall speed per grain
  const double *pq = cq + (long)g * L.PG + base, *pl = lin + (long)g * L.PG + base, *pv = vel + base;
  const double lam0 = (DIR == 2 && lam_lo) ? lam_lo[(long)g * L.nx * L.ny + (long)(o - 1) * L.nx + (ac - 1)] : 0.0;
  auto Q = [&](int c) { return c >= 1 && c <= n ? pq[(c - 1) * st] : 0.0; };
  auto V = [&](int c) { return pv[((c < 1 ? 1 : c) - 1) * st] + vf0; };
  auto Lm = [&](int c) { return c >= 1 ? pl[(c - 1) * st] : c == 0 ? lam0 : 0.0; };
  auto T = [&](int c) { return c < 0 ? 0.0 : -(gdtv.at(c) * Lm(c)); };
  AdjMarch m = adj_march_start(s0, Q, V, T, Lm);
  const double vedge = pv[(n - 1) * st];  // the wind beyond the line
  po += (long)(s0 - 1) * st;              // cell x-3's place, once x-3 >= s0
  uint32_t ph = 0u;
  for (int k = 0, x = s0; k < nchunk; k++) {
    const int bi = k & 1;
    if (k + 1 < nchunk) issue(k + 1);
    if (!mbar_wait(&bar[bi], (ph >> bi) & 1u)) {
      if (lane == 0) raise_error(sc, A3G_ERR_TIMEOUT, 6);
      return;
    }
    ph ^= 1u << bi;
    double *qv = wsm + bi * ADJ_BUF_D + lane;
    if (x <= n + 1 && n + 1 < x + ACH) qv[(ACH + n + 1 - x) * 32] = vedge;
    __syncwarp();
    const double2 *gb = reinterpret_cast<const double2 *>(wsm + bi * ADJ_BUF_D + 3 * ACH * 32);
    const int cnt = min(ACH, s1 + 3 - x + 1);
    // whether every wind that the chunk's interfaces take is a number: their sum is
    double sum = m.vm + m.v + vf0;
#pragma unroll
    for (int u = 0; u < ACH; u += 2) sum = sum + (qv[(ACH + u) * 32] + qv[(ACH + u + 1) * 32]);
    auto step = [&](auto any, int e) {
      const double2 sd = gb[e];
      const double y = adj_march_step<LIM, decltype(any)::value>(m, qv[e * 32], qv[(ACH + e) * 32] + vf0, qv[(2 * ACH + e) * 32], sd.x, sd.y,
                                           eps, nocycle);
      if (x + e - 3 >= s0) {
        if (valid) *po = y;
        po += st;
      }
    };
    int e = 0;
    if (__any_sync(0xffffffffu, !finite_bits(sum)))
      for (; e < cnt; e++) step(TrueT{}, e);
    for (; e + 2 <= cnt; e += 2) {
      step(FalseT{}, e);
      step(FalseT{}, e + 1);
    }
    if (e < cnt) step(FalseT{}, e);
    x += ACH;
    __syncwarp();
  }
}

// Rows (x): k_advect_xm's mapping and swizzled chunks, a row per lane.  Chunk
// k holds the cells s0+8k ..; the new lam of cell x-4 takes the place of cell
// x's old one, so that a chunk's new values start on an even cell; the first
// and last chunk of a segment, which also hold other segments' cells, are
// stored by the lanes.  140x120x40, 4 grains: 133 -> 31 us (the blocks' lanes
// were four cells apart, a sector each).
constexpr int AJX_WARP_B = 7 * AXM_BUF;  // 2 concentration, 2 wind, 3 lam buffers
constexpr int AJX_SMEM = 512 + 512 + ADJ_WARPS * AJX_WARP_B;

template <int LIM>
__global__ void __launch_bounds__(32 * ADJ_WARPS, 8) k_adj_xm(
    const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tv,
    const __grid_constant__ CUtensorMap tl, const __grid_constant__ CUtensorMap to, Layout L, int nocycle, double eps,
    int nseg, int seg, const double *__restrict__ cq, const double *__restrict__ lin, double *__restrict__ lout,
    const double *__restrict__ vel, Geo3 sig, Geo3 dtvt, const int32_t *__restrict__ aloft, DevScalars *sc) {
  extern __shared__ unsigned char ajx_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned char *const sm = ajx_smem + ((512u - (smem_u32(ajx_smem) & 511u)) & 511u);  // the swizzle's period
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm) + 2 * wid;
  unsigned char *const qbuf = sm + 512 + wid * AJX_WARP_B, *const vbuf = qbuf + 2 * AXM_BUF,
                *const lbuf = vbuf + 2 * AXM_BUF;
  const int nrows = L.ny * L.nz;
  const int ntile = (nrows + 31) >> 5;
  const unsigned t = blockIdx.x * ADJ_WARPS + wid, ns = L.ns, rr = t / ns, rs = rr / (unsigned)ntile;
  if (rs >= (unsigned)nseg) return;  // whole warps only; no block barrier below
  const int g = (int)(t - rr * ns);
  const int r0 = (int)(rr - rs * (unsigned)ntile) * 32;
  const int s0 = (int)rs * seg + 1;
  const int n = L.nx, s1 = min(n, s0 + seg - 1);
  const int r = min(r0 + lane, nrows - 1);
  const int j = r % L.ny + 1, k = r / L.ny + 1;
  const long grow = (long)g * nrows;
  double *const po = lout + (grow + r0) * L.P;
  if (!aloft[g]) {
    for (int row = 0; row < min(32, nrows - r0); row++)
      for (int c = s0 + lane; c <= s1; c += 32) po[(long)row * L.P + (c - 1)] = 0.0;
    return;
  }
  const int nchunk = (s1 + 4 - s0 + 8) >> 3;  // cells s0 .. s1+4
  auto issue = [&](int c) {  // chunk c; its lam buffer was stored from two chunks ago
    if (lane == 0) {
      uint64_t *b = &bar[c & 1];
      bulk_wait_read1();
      mbar_arrive_expect_tx(b, 3u * AXM_BUF);
      tma_load_2d(qbuf + (c & 1) * AXM_BUF, &tq, b, s0 - 1 + 8 * c, (int)(grow + r0));
      tma_load_2d(vbuf + (c & 1) * AXM_BUF, &tv, b, s0 - 1 + 8 * c, r0);
      tma_load_2d(lbuf + (c % 3) * AXM_BUF, &tl, b, s0 - 1 + 8 * c, (int)(grow + r0));
    }
  };
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
  }
  __syncwarp();
  issue(0);
  const double *const pq = cq + (grow + r) * L.P, *const pl = lin + (grow + r) * L.P, *const pv = vel + (long)r * L.P;
  const double hs = 0.5 * sig.p[(long)(j + 1) * sig.sj + (long)(k + 1) * sig.sk];
  const double dtv = dtvt.p[(long)(j + 1) * dtvt.sj + (long)(k + 1) * dtvt.sk];
  auto Q = [&](int c) { return c >= 1 && c <= n ? pq[c - 1] : 0.0; };
  auto V = [&](int c) { return pv[(c < 1 ? 1 : c) - 1]; };
  auto Lm = [&](int c) { return c >= 1 ? pl[c - 1] : 0.0; };
  auto T = [&](int c) { return -(dtv * Lm(c)); };
  AdjMarch m = adj_march_start(s0, Q, V, T, Lm);
  const int row_b = lane << 6, row_s = ((lane >> 1) & 3) << 4;
  auto pair = [&](unsigned char *b, int p) { return reinterpret_cast<double2 *>(b + row_b + ((p << 4) ^ row_s)); };
  auto cell = [&](unsigned char *b, int e) { return reinterpret_cast<double *>(pair(b, e >> 1)) + (e & 1); };
  double held = 0.0;  // lam_q of the cell behind the last one computed
  auto step = [&](auto any, double q, double v, double l, double h) {
    const double y = held;
    held = adj_march_step<LIM, decltype(any)::value>(m, q, v, l, h, dtv, eps, nocycle);
    return y;
  };
  const bool whole = r0 + 32 <= nrows;
  uint32_t ph = 0u;
  for (int c = 0; c < nchunk; c++) {
    if (c + 1 < nchunk) issue(c + 1);
    if (!mbar_wait(&bar[c & 1], (ph >> (c & 1)) & 1u)) {
      if (lane == 0) {
        raise_error(sc, A3G_ERR_TIMEOUT, 7);
        bulk_wait0();
      }
      return;
    }
    ph ^= 1u << (c & 1);
    unsigned char *const qb = qbuf + (c & 1) * AXM_BUF, *const vb = vbuf + (c & 1) * AXM_BUF,
                  *const lb = lbuf + (c % 3) * AXM_BUF;
    const int X = s0 + 8 * c;  // slot e: cell X+e in, cell X+e-4 out
    if (X + 7 > n) {           // the edge wind, and its negative beyond: usig(n+2) = 0
      for (int x = max(n + 1, X); x <= min(n + 2, X + 7); x++) *cell(vb, x - X) = x == n + 1 ? pv[n - 1] : -pv[n - 1];
    }
    // whether every wind that the chunk's interfaces take is a number: their sum is
    double sum = m.vm + m.v;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const double2 v = *pair(vb, p);
      sum = sum + (v.x + v.y);
    }
    if (X > 1 && !__any_sync(0xffffffffu, !finite_bits(sum))) {
#pragma unroll 2
      for (int p = 0; p < 4; p++) {
        double2 *l = pair(lb, p);
        const double2 q = *pair(qb, p), v = *pair(vb, p), w = *l;
        double2 y;
        y.x = step(FalseT{}, q.x, v.x, w.x, hs);
        y.y = step(FalseT{}, q.y, v.y, w.y, hs);
        *l = y;
      }
    } else {  // interface 0 carries nothing
      for (int e = 0; e < 8; e++)
        *cell(lb, e) = step(TrueT{}, *cell(qb, e), *cell(vb, e), *cell(lb, e), X == 1 && e == 0 ? 0.0 : hs);
    }
    fence_proxy_async_smem();
    __syncwarp();
    const int o0 = X - 4;  // first cell of the chunk's new values
    if (whole && o0 >= s0 && o0 + 7 <= s1) {
      if (lane == 0) {
        tma_store_2d(&to, lb, o0 - 1, (int)(grow + r0));
        bulk_commit();
      }
    } else {
      const int e = lane & 7, x = o0 + e;
#pragma unroll
      for (int h = 0; h < 8; h++) {
        const int row = 4 * h + (lane >> 3);
        if (r0 + row < nrows && x >= s0 && x <= s1)
          po[(long)row * L.P + (x - 1)] = *reinterpret_cast<const double *>(
              lb + (row << 6) + ((((e >> 1) ^ ((row >> 1) & 3)) << 4) | ((e & 1) << 3)));
      }
      __syncwarp();
    }
  }
  if (lane == 0) bulk_wait0();
}

// Launches the marched adjoint sweep; false where its conditions (those of the
// forward marches) do not hold.
template <int DIR, int LIM>
static bool launch_adj_march(a3g_ctx *ctx, const double *cq, const double *lin, double *lout, const double *lam_lo) {
  const Layout &L = ctx->L;
  CUtensorMap tq, tv, tl, to;
  if constexpr (DIR == 0) {
    if (along<0>(ctx->snx) != 0 || along<0>(ctx->dtv) != 0) return false;
    if (!tensor_map(ctx, cq, TM_QROWS, &tq) || !tensor_map(ctx, ctx->vx, TM_VROWS, &tv) ||
        !tensor_map(ctx, lin, TM_QROWS, &tl) || !tensor_map(ctx, lout, TM_QROWS, &to))
      return false;
    const long nlw = (long)(((long)L.ny * L.nz + 31) / 32) * L.ns;
    const int want = march_segments(L.nx, nlw);
    const int seg = (L.nx + want - 1) / want + 7 & ~7;
    const int nseg = (L.nx + seg - 1) / seg;
    k_adj_xm<LIM><<<(unsigned)((nlw * nseg + ADJ_WARPS - 1) / ADJ_WARPS), 32 * ADJ_WARPS, AJX_SMEM, ctx->stream>>>(
        tq, tv, tl, to, L, ctx->prm.nocycle, ctx->prm.eps_thresh, nseg, seg, cq, lin, lout, ctx->vx, ctx->snx,
        ctx->dtv, ctx->aloft, ctx->sc);
  } else {
    const Geo3 &sg = (DIR == 1) ? ctx->sny : ctx->snz;
    const double *vel = (DIR == 1) ? ctx->vy : ctx->vz;
    if (sg.si != 0 || ctx->dtv.si != 0) return false;
    if (DIR == 2 && (ctx->vf.si != 0 || ctx->vf.sj != 0 || ctx->vf.sk != 0)) return false;
    const int qk = DIR == 1 ? TM_ADV_QY : TM_ADV_QZ, vk = DIR == 1 ? TM_ADV_VY : TM_ADV_VZ;
    if (!tensor_map(ctx, cq, qk, &tq) || !tensor_map(ctx, vel, vk, &tv) || !tensor_map(ctx, lin, qk, &tl)) return false;
    const int n = (DIR == 1) ? L.ny : L.nz, nother = (DIR == 1) ? L.nz : L.ny;
    const long nlw = (long)((L.nx + 31) / 32) * nother * L.ns;
    const int want = march_segments(n, nlw);
    const int seg = (n + want - 1) / want, nseg = (n + seg - 1) / seg;
    const size_t smem = 128 + (size_t)ADJ_WARPS * 2 * ADJ_BUF_D * sizeof(double);
    k_adj_colt<DIR, LIM><<<(unsigned)((nlw * nseg + ADJ_WARPS - 1) / ADJ_WARPS), 32 * ADJ_WARPS, smem, ctx->stream>>>(
        tq, tv, tl, L, ctx->prm.nocycle, ctx->prm.eps_thresh, nseg, seg, cq, lin, lout, vel, ctx->vf, sg, ctx->dtv,
        ctx->aloft, ctx->sc, lam_lo);
  }
  return true;
}

template <int DIR, int LIM>
static void launch_adj_dir_lim(a3g_ctx *ctx, const double *cq, const double *lin, double *lout,
                               const double *lam_lo) {
  const Layout &L = ctx->L;
  dim3 grid((L.nx + 31) / 32, (L.ny + 7) / 8, L.nz * L.ns);
  const bool per = (DIR == 0) && ctx->grid.periodic;
  const double *vel = (DIR == 0) ? ctx->vx : (DIR == 1) ? ctx->vy : ctx->vz;
  const Geo3 &sig = (DIR == 0) ? ctx->snx : (DIR == 1) ? ctx->sny : ctx->snz;
  if (per) {
    k_adj_advect<DIR, LIM, true><<<grid, dim3(32, 8), 0, ctx->stream>>>(
        L, ctx->prm.nocycle, ctx->prm.eps_thresh, cq, lin, lout, vel, ctx->vf, sig, ctx->dtv, ctx->aloft,
        lam_lo);
  } else if (ctx->adj_gather) {
    k_adj_advect<DIR, LIM, false><<<grid, dim3(32, 8), 0, ctx->stream>>>(
        L, ctx->prm.nocycle, ctx->prm.eps_thresh, cq, lin, lout, vel, ctx->vf, sig, ctx->dtv, ctx->aloft,
        lam_lo);
  } else if (!launch_adj_march<DIR, LIM>(ctx, cq, lin, lout, lam_lo)) {
    constexpr int V = 4;
    const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
    const int nblk = (n + V - 1) / V;
    dim3 gb;
    if (DIR == 0) gb = dim3((nblk + 31) / 32, (L.ny + 3) / 4, L.nz * L.ns);
    else gb = dim3((L.nx + 31) / 32, (nblk * ((DIR == 1) ? L.nz : L.ny) + 3) / 4, L.ns);
    k_adj_advect_blk<DIR, LIM, V><<<gb, dim3(32, 4), 0, ctx->stream>>>(
        L, ctx->prm.nocycle, ctx->prm.eps_thresh, nblk, cq, lin, lout, vel, ctx->vf, sig, ctx->dtv, ctx->aloft,
        lam_lo);
  }
}

template <int DIR>
static void launch_adj_dir(a3g_ctx *ctx, const double *cq, const double *lin, double *lout,
                           const double *lam_lo) {
  switch (ctx->prm.limiter) {
    case A3G_LIM_NONE: launch_adj_dir_lim<DIR, A3G_LIM_NONE>(ctx, cq, lin, lout, lam_lo); break;
    case A3G_LIM_LAXWEN: launch_adj_dir_lim<DIR, A3G_LIM_LAXWEN>(ctx, cq, lin, lout, lam_lo); break;
    case A3G_LIM_BW: launch_adj_dir_lim<DIR, A3G_LIM_BW>(ctx, cq, lin, lout, lam_lo); break;
    case A3G_LIM_FROMM: launch_adj_dir_lim<DIR, A3G_LIM_FROMM>(ctx, cq, lin, lout, lam_lo); break;
    case A3G_LIM_MINMOD: launch_adj_dir_lim<DIR, A3G_LIM_MINMOD>(ctx, cq, lin, lout, lam_lo); break;
    case A3G_LIM_MC: launch_adj_dir_lim<DIR, A3G_LIM_MC>(ctx, cq, lin, lout, lam_lo); break;
    default: launch_adj_dir_lim<DIR, A3G_LIM_SUPERBEE>(ctx, cq, lin, lout, lam_lo); break;
  }
}

// lam_out <- J(cq)^T lam_in for the advection sweep along dir (0 x, 1 y, 2 z).
int launch_adj_advect(a3g_ctx *ctx, int dir, const double *cq, const double *lin, double *lout,
                      const double *lam_lo) {
  int rc = refresh_dtv(ctx);
  if (rc) return rc;
  tbegin(ctx, A3G_K_ADJOINT);
  if (dir == 0) launch_adj_dir<0>(ctx, cq, lin, lout, nullptr);
  else if (dir == 1) launch_adj_dir<1>(ctx, cq, lin, lout, nullptr);
  else launch_adj_dir<2>(ctx, cq, lin, lout, lam_lo);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// ===========================================================================
// Tangent-linear of one advection sweep (no counterpart in the reference).
//
// The same linear map k_adj_advect transposes: with the limiter branches
// fixed by the sweep's input state q (lim_coef: ldq = a*dq + b*dqu), a
// perturbation d of the input goes to
//   d_fss(I) = cf(I)*(a(I)*dd(I) + b(I)*dd_u(I))   (active fss interfaces)
//   d_fsr(I) = max(0,us)*dd(I) + d(I)*divu_m(I),  d_fsl(I) = min(0,us)*dd(I) + d(I-1)*divu_p(I)
//   d_out(m) = d(m) - dt/kappa(m)*(d_fsl(m+1) + d_fsr(m) + d_fss(m+1) - d_fss(m))
// with dd = the perturbation's slopes and Set_BC(1) ghosts (zero, x-periodic
// wrap).  The z sweep adds the perturbation of the bottom outflow (the
// deposit) to dep.  One thread per cell-grain, full box.
// ===========================================================================
template <int DIR, int LIM, bool PER>
__global__ void __launch_bounds__(256) k_tl_advect(Layout L, int nocycle, double eps,
                                                   const double *__restrict__ cq,
                                                   const double *__restrict__ din,
                                                   double *__restrict__ dout,
                                                   const double *__restrict__ vel, Geo4 vf, Geo3 sig,
                                                   Geo3 dtvt, const int32_t *__restrict__ aloft,
                                                   double *__restrict__ dep) {
  const int i = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int k = (int)(blockIdx.z % L.nz) + 1;
  const int g = (int)(blockIdx.z / L.nz);
  if (i > L.nx || j > L.ny) return;
  const long cell = L.cell(i, j, k);
  const long gb = (long)g * L.PG;
  if (!aloft[g]) {
    dout[gb + cell] = 0.0;
    return;
  }
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  const int m = (DIR == 0) ? i : (DIR == 1) ? j : k;
  const long st = (DIR == 0) ? 1 : (DIR == 1) ? L.P : L.PY;
  const long lb = cell - (long)(m - 1) * st;
  const int la = (DIR == 0) ? j : i, lo_ = (DIR == 2) ? j : k;
  const LineGeo gsig = line_of<DIR>(sig, la, lo_);
  const LineGeo gdtv = line_of<DIR>(dtvt, la, lo_);
  const double *pq = cq + gb + lb;
  const double *pd = din + gb + lb;
  const double *pv = vel + lb;
  const double *pvf = vf.p + (long)(i + 1) * vf.si + (long)(j + 1) * vf.sj + (long)g * vf.sg;
  auto wrap = [&](int c) { return c < 1 ? c + n : (c > n ? c - n : c); };
  auto ghosted = [&](const double *p, int c) -> double {
    if (c < -1 || c > n + 2) return 0.0;
    if (c >= 1 && c <= n) return p[(long)(c - 1) * st];
    return PER ? p[(long)(wrap(c) - 1) * st] : 0.0;
  };
  auto V = [&](int c) -> double {
    const int cl = PER ? wrap(c) : (c < 1 ? 1 : (c > n ? n : c));
    double v = pv[(long)(cl - 1) * st];
    if (DIR == 2) v = v + pvf[(long)(cl + 1) * vf.sk];
    return v;
  };
  auto US = [&](int I) -> double {  // usig(I), zero outside [0, n+1]
    if (I < 0 || I > n + 1) return 0.0;
    return 0.5 * (V(I - 1) + V(I)) * gsig.at(I);
  };
  // d_fss, d_fsr, d_fsl of interface I
  auto iface = [&](int I, double &dfss, double &dfsr, double &dfsl) {
    const double us = US(I), usm = US(I - 1), usp = US(I + 1);
    dfss = 0.0;
    dfsr = 0.0;
    dfsl = 0.0;
    if (I < 0 || I > n + 1) return;
    const double qm2 = ghosted(pq, I - 2), qm1 = ghosted(pq, I - 1), q0 = ghosted(pq, I), qp1 = ghosted(pq, I + 1);
    const double dm2 = ghosted(pd, I - 2), dm1 = ghosted(pd, I - 1), d0 = ghosted(pd, I), dp1 = ghosted(pd, I + 1);
    const double dq = q0 - qm1, ddq = d0 - dm1;
    const bool up = us > 0.0;
    if (LIM != A3G_LIM_NONE && I >= 1 && (nocycle || !(fabs(dq) <= eps))) {
      const double dqu = up ? qm1 - qm2 : qp1 - q0;
      const double ddqu = up ? dm1 - dm2 : dp1 - d0;
      double a, b;
      lim_coef<LIM>(dq, dqu, eps, a, b);
      const double aus = fabs(us);
      const double cf = 0.5 * aus * (1.0 - gdtv.at(I) * aus);
      dfss = cf * (a * ddq + b * ddqu);
    }
    const double divm = fmn(0.0, usp) - fmn(0.0, us);
    const double divp = fmx(0.0, us) - fmx(0.0, usm);
    dfsr = fmx(0.0, us) * ddq + d0 * divm;
    dfsl = fmn(0.0, us) * ddq + dm1 * divp;
  };
  double fssL, fsrL, fslL, fssR, fsrR, fslR;
  iface(m, fssL, fsrL, fslL);
  iface(m + 1, fssR, fsrR, fslR);
  const double dupd = -(gdtv.at(m) * (fslR + fsrL + fssR - fssL));
  dout[gb + cell] = pd[(long)(m - 1) * st] + dupd;
  if (DIR == 2 && dep && m == 1) {  // cell 0 (the bottom outflow): interfaces 0 and 1, fss(0) = 0
    double fss0, fsr0, fsl0;
    iface(0, fss0, fsr0, fsl0);
    const double d0upd = -(gdtv.at(0) * (fslL + fsr0 + fssL - 0.0));
    dep[(long)g * L.nx * L.ny + (long)(j - 1) * L.nx + (i - 1)] += d0upd;
  }
}

template <int DIR, int LIM>
static void launch_tl_dir_lim(a3g_ctx *ctx, const double *cq, const double *din, double *dout, double *dep) {
  const Layout &L = ctx->L;
  dim3 grid((L.nx + 31) / 32, (L.ny + 7) / 8, L.nz * L.ns);
  const bool per = (DIR == 0) && ctx->grid.periodic;
  const double *vel = (DIR == 0) ? ctx->vx : (DIR == 1) ? ctx->vy : ctx->vz;
  const Geo3 &sig = (DIR == 0) ? ctx->snx : (DIR == 1) ? ctx->sny : ctx->snz;
  if (per)
    k_tl_advect<DIR, LIM, true><<<grid, dim3(32, 8), 0, ctx->stream>>>(
        L, ctx->prm.nocycle, ctx->prm.eps_thresh, cq, din, dout, vel, ctx->vf, sig, ctx->dtv, ctx->aloft, dep);
  else
    k_tl_advect<DIR, LIM, false><<<grid, dim3(32, 8), 0, ctx->stream>>>(
        L, ctx->prm.nocycle, ctx->prm.eps_thresh, cq, din, dout, vel, ctx->vf, sig, ctx->dtv, ctx->aloft, dep);
}

template <int DIR>
static void launch_tl_dir(a3g_ctx *ctx, const double *cq, const double *din, double *dout, double *dep) {
  switch (ctx->prm.limiter) {
    case A3G_LIM_NONE: launch_tl_dir_lim<DIR, A3G_LIM_NONE>(ctx, cq, din, dout, dep); break;
    case A3G_LIM_LAXWEN: launch_tl_dir_lim<DIR, A3G_LIM_LAXWEN>(ctx, cq, din, dout, dep); break;
    case A3G_LIM_BW: launch_tl_dir_lim<DIR, A3G_LIM_BW>(ctx, cq, din, dout, dep); break;
    case A3G_LIM_FROMM: launch_tl_dir_lim<DIR, A3G_LIM_FROMM>(ctx, cq, din, dout, dep); break;
    case A3G_LIM_MINMOD: launch_tl_dir_lim<DIR, A3G_LIM_MINMOD>(ctx, cq, din, dout, dep); break;
    case A3G_LIM_MC: launch_tl_dir_lim<DIR, A3G_LIM_MC>(ctx, cq, din, dout, dep); break;
    default: launch_tl_dir_lim<DIR, A3G_LIM_SUPERBEE>(ctx, cq, din, dout, dep); break;
  }
}

// dout <- J(cq) din for the advection sweep along dir; dep (z only, may be
// null) gains the perturbation of the bottom outflow.
int launch_tl_advect(a3g_ctx *ctx, int dir, const double *cq, const double *din, double *dout, double *dep) {
  int rc = refresh_dtv(ctx);
  if (rc) return rc;
  tbegin(ctx, A3G_K_ADJOINT);
  if (dir == 0) launch_tl_dir<0>(ctx, cq, din, dout, nullptr);
  else if (dir == 1) launch_tl_dir<1>(ctx, cq, din, dout, nullptr);
  else launch_tl_dir<2>(ctx, cq, din, dout, dep);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

}  // namespace a3g
