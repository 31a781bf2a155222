// k_diffuse.cu -- explicit and Crank-Nicolson diffusion sweeps on the device.
//
// Explicit: diff_x/diff_y/diff_z, src/Diffusion.F90:266-650 (LeVeque eq. 4.11)
//   update(l) = dt*k_ds(l+1)*dq(l+1)*(sig(l+1)/kap(l)) - dt*k_ds(l)*dq(l)*(sig(l)/kap(l))
//   with k_ds = 0.5*(k_{l-1}+k_l) * 2*sig/(kap_{l-1}+kap_l) and Neumann ghosts
//   (periodic in x).  Where nothing varies along i, warps march along j (x and y
//   in one pass) and k with the factors that dt does not touch in a table; else,
//   and in z on small grids, one thread per cell takes all grains in a loop.
//
// Crank-Nicolson: diffCN_x/y/z, src/Diffusion.F90:671-1428 (eq. 4.13), each
// line solved by LAPACK dgtsv in the reference.  The matrices are strictly
// diagonally dominant (D >= 1, off-diagonals -Imp_fac*L <= 0), so dgtsv's
// partial pivoting never interchanges rows on them and its elimination
// reduces to: fact = DL(i)/D'(i); D'(i+1) = D(i+1) - fact*DU(i);
// B'(i+1) = B(i+1) - fact*B'(i); then x(n) = B'(n)/D'(n),
// x(i) = (B'(i) - DU(i)*x(i+1))/D'(i).  The factorisation (fact, D', DU) and
// the right-hand-side weights depend only on geometry, diffusivity and dt, so
// a table, rebuilt when dt changes, holds them once per distinct line geometry (a
// projected grid has one per k) and a lane solves one line of one grain.
// A line that would need a row interchange (or a zero pivot) raises
// A3G_ERR_PIVOT instead of silently diverging from dgtsv.
#include "a3g_internal.cuh"
#include "exact_div.cuh"
#include "tma.cuh"

namespace a3g {

// ---------------------------------------------------------------------------
// explicit diffusion
// ---------------------------------------------------------------------------
template <int DIR>
__global__ void __launch_bounds__(256) k_diff(Layout L, Box box, int periodic,
                                              const double *__restrict__ cin,
                                              double *__restrict__ cout, Geo3 sig, Geo3 kap,
                                              Geo3 kk, const int32_t *__restrict__ aloft,
                                              const DevScalars *__restrict__ sc) {
  const int i = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > L.nx || j > L.ny) return;
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  const int l = (DIR == 0) ? i : (DIR == 1) ? j : k;
  const int rmin = (DIR == 0) ? box.imin : (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 0) ? box.imax : (DIR == 1) ? box.jmax : box.kmax;
  const bool active = i >= box.imin && i <= box.imax && j >= box.jmin && j <= box.jmax &&
                      k >= box.kmin && k <= box.kmax;
  const long cell = L.cell(i, j, k);
  if (!active) {
    for (int g = 0; g < L.ns; g++) cout[(long)g * L.PG + cell] = 0.0;
    return;
  }
  const long st = (DIR == 0) ? 1 : (DIR == 1) ? L.P : L.PY;
  auto G = [&](const Geo3 &a, int m) {
    return (DIR == 0) ? a.at(m, j, k) : (DIR == 1) ? a.at(i, m, k) : a.at(i, j, m);
  };
  const double dt = sc->dt;
  // interface l+1 (right) and l (left), :351-360
  const double dsR = 2.0 * G(sig, l + 1) / (G(kap, l) + G(kap, l + 1));
  const double kdsR = 0.5 * (G(kk, l) + G(kk, l + 1)) * dsR;
  const double dsL = 2.0 * G(sig, l) / (G(kap, l - 1) + G(kap, l));
  const double kdsL = 0.5 * (G(kk, l - 1) + G(kk, l)) * dsL;
  const double aR = dt * kdsR, aL = dt * kdsL;
  const double sR = G(sig, l + 1) / G(kap, l), sL = G(sig, l) / G(kap, l);
  // neighbour offsets with the Neumann (or periodic x) ghosts, :317-327
  long offL = -st, offR = st;
  bool selfL = false, selfR = false;
  if (l - 1 < 1) {
    if (DIR == 0 && periodic) offL = (long)(n - 1);
    else selfL = true;
  }
  if (l + 1 > n) {
    if (DIR == 0 && periodic) offR = -(long)(n - 1);
    else selfR = true;
  }
  for (int g = 0; g < L.ns; g++) {
    const long a = (long)g * L.PG + cell;
    if (!aloft[g]) { cout[a] = 0.0; continue; }
    const double q = cin[a];
    const double qL = selfL ? q : cin[a + offL];
    const double qR = selfR ? q : cin[a + offR];
    const double LF = aR * (qR - q) * sR;
    const double RF = -(aL * (q - qL) * sL);
    cout[a] = (l >= rmin && l <= rmax) ? q + (LF + RF) : 0.0;
  }
}

// ---------------------------------------------------------------------------
// Explicit diffusion where nothing it uses varies along i (every projected or
// lon/lat grid with uniform diffusivities): the dt-independent factors come
// from a table per (j, k), and DiffuseHorz's two sweeps run as one.
// ---------------------------------------------------------------------------
// Row (j, k) of the table: the x factors k_ds and sigma/kappa (the same for
// both faces), then for y and for z k_ds of the face before the cell,
// sigma/kappa of the face after it and of the face before it.
struct DiffRow {
  double kx, sx, ky, syR, syL, kz, szR, szL;
};

// rows j = 1..ny+1, k = 1..nz+1 (the last ones for their ky and kz only)
__global__ void k_diff_table(Layout L, Geo3 snx, Geo3 sny, Geo3 snz, Geo3 kap, Geo3 kx, Geo3 ky, Geo3 kz,
                             DiffRow *__restrict__ tab) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (L.ny + 1) * (L.nz + 1)) return;
  const int j = t % (L.ny + 1) + 1, k = t / (L.ny + 1) + 1, i = 1;
  const double k0 = kap.at(i, j, k);
  DiffRow r;
  // :351-360 in the operations of k_diff
  r.kx = 0.5 * (kx.at(i, j, k) + kx.at(i + 1, j, k)) * (2.0 * snx.at(i + 1, j, k) / (k0 + kap.at(i + 1, j, k)));
  r.sx = snx.at(i + 1, j, k) / k0;
  r.ky = 0.5 * (ky.at(i, j - 1, k) + ky.at(i, j, k)) * (2.0 * sny.at(i, j, k) / (kap.at(i, j - 1, k) + k0));
  r.syR = sny.at(i, j + 1, k) / k0;
  r.syL = sny.at(i, j, k) / k0;
  r.kz = 0.5 * (kz.at(i, j, k - 1) + kz.at(i, j, k)) * (2.0 * snz.at(i, j, k) / (kap.at(i, j, k - 1) + k0));
  r.szR = snz.at(i, j, k + 1) / k0;
  r.szL = snz.at(i, j, k) / k0;
  tab[t] = r;
}

// One cell of a sweep from its neighbours; aL, aR: dt*k_ds of its faces, sL,
// sR: sigma/kappa of its faces.  A neighbour beyond the grid is the cell
// itself (Neumann) or the wrapped one.
__device__ __forceinline__ double diff_cell(double l, double q, double r, double aL, double aR, double sL, double sR) {
  const double LF = aR * (r - q) * sR;
  const double RF = -(aL * (q - l) * sL);
  return q + (LF + RF);
}
// Its transpose: own coefficients cL, cR, the left neighbour's cR and the right
// neighbour's cL; the ghosts' terms fold back last (k_adj_diff's order).
__device__ __forceinline__ double adj_diff_cell(double l, double q, double r, double cL, double cR, double cRm,
                                                double cLp, bool first, bool last) {
  double v = q - cR * q - cL * q;
  if (!first) v = v + cRm * l;
  if (!last) v = v + cLp * r;
  if (first) v = v + (cRm)*l;
  if (last) v = v + (cLp)*r;
  return v;
}

// DiffuseHorz (ADJ: its transpose) in one pass: XFIRST the x sweep, then the y
// sweep, else the other order.  A warp marches along j with a column per
// lane; the first and last lane hold the columns beside the warp's 30, so that
// every x neighbour is a shuffle away, and the rows beside a segment are taken
// again.  The sweep in between never reaches memory: 16 B a cell instead of 32,
// and the six divisions a cell that k_diff repeats every step are the table's.
// 360x161x40, 5 grains: x and y 200 -> 64 us together; 100x100x40, 4 grains: 40
// -> 15 us.
template <bool XFIRST, bool ADJ, bool PER>
__global__ void __launch_bounds__(128) k_diff_xy(Layout L, Box box, Box cov, int nseg, int seg,
                                                 const double *__restrict__ cin, double *__restrict__ cout,
                                                 const DiffRow *__restrict__ tab,
                                                 const int32_t *__restrict__ aloft,
                                                 const DevScalars *__restrict__ sc) {
  const int lane = threadIdx.x & 31;
  const int nti = (cov.imax - cov.imin + 30) / 30, nk = cov.kmax - cov.kmin + 1;
  const unsigned w = blockIdx.x * 4 + (threadIdx.x >> 5), wt = w / (unsigned)nti, ws = wt / (unsigned)nseg;
  const int g = (int)(ws / (unsigned)nk), k = (int)ws - g * nk + cov.kmin;
  if (g >= L.ns) return;  // whole warps
  const int it = (int)(w - wt * (unsigned)nti);
  const int s0 = (int)(wt - ws * (unsigned)nseg) * seg + cov.jmin, s1 = min(cov.jmax, s0 + seg - 1);
  const int i0 = cov.imin - 1 + it * 30 + lane;  // 1-based column of this lane: 0 and nx+1 are the ghosts
  const int i = i0 < 1 ? (PER ? L.nx : 1) : i0 > L.nx ? (PER ? (i0 - L.nx - 1) % L.nx + 1 : L.nx) : i0;
  const bool own = lane >= 1 && lane <= 30 && i0 <= cov.imax;
  const double *q0 = cin + (long)g * L.PG + (long)(k - 1) * L.PY + (i - 1);
  double *p0 = cout + (long)g * L.PG + (long)(k - 1) * L.PY + (i - 1);
  const bool col_in = i >= box.imin && i <= box.imax && k >= box.kmin && k <= box.kmax;
  if (!aloft[g] || !__any_sync(0xffffffffu, col_in)) {
    if (own)
      for (int j = s0; j <= s1; j++) p0[(long)(j - 1) * L.P] = 0.0;
    return;
  }
  const double dt = sc->dt;
  const DiffRow *T = tab + (long)(k - 1) * (L.ny + 1) - 1;  // row j at T[j]
  auto in = [&](int j) { return col_in && j >= box.jmin && j <= box.jmax; };
  auto xs = [&](double q, int j) {  // the x sweep of row j; lanes 0 and 31 give nothing of use
    const double l = __shfl_up_sync(0xffffffffu, q, 1), r = __shfl_down_sync(0xffffffffu, q, 1);
    const double a = dt * T[j].kx, s = T[j].sx;
    if (ADJ) {
      const double c = a * s;
      return adj_diff_cell(l, q, r, c, c, c, c, i == 1, i == L.nx);
    }
    return in(j) ? diff_cell(l, q, r, a, a, s, s) : 0.0;
  };
  auto ys = [&](double l, double q, double r, int j) {  // the y sweep at row j
    const double aL = dt * T[j].ky, aR = dt * T[j + 1].ky;
    if (ADJ) {
      const double cL = aL * T[j].syL, cR = aR * T[j].syR;
      const double cRm = j > 1 ? aL * T[j - 1].syR : cL, cLp = j < L.ny ? aR * T[j + 1].syL : cR;
      return adj_diff_cell(l, q, r, cL, cR, cRm, cLp, j == 1, j == L.ny);
    }
    return in(j) ? diff_cell(l, q, r, aL, aR, T[j].syL, T[j].syR) : 0.0;
  };
  auto at = [&](int j) { return q0[(long)((j < 1 ? 1 : j > L.ny ? L.ny : j) - 1) * L.P]; };
  // row j as the y sweep sees it, from row j as loaded
  auto row = [&](double q, int j) {
    const int jc = j < 1 ? 1 : j > L.ny ? L.ny : j;  // a ghost row is its neighbour's copy
    return XFIRST ? xs(q, jc) : q;
  };
  double a = row(at(s0 - 1), s0 - 1), b = row(at(s0), s0);
  double nq = at(s0 + 1);
#pragma unroll 4
  for (int j = s0; j <= s1; j++) {
    const double c = row(nq, j + 1);
    nq = at(j + 2);
    double y = ys(a, b, c, j);
    if (!XFIRST) y = xs(y, j);
    if (own) p0[(long)(j - 1) * L.P] = y;
    a = b;
    b = c;
  }
}

// DiffuseVert (ADJ: its transpose) marched along k, lanes along i, every cell
// read once.  360x161x40, 5 grains: 76 -> 56 us.
template <bool ADJ>
__global__ void __launch_bounds__(128) k_diff_z(Layout L, Box box, Box cov, int nseg, int seg, const double *__restrict__ cin,
                                                double *__restrict__ cout, const DiffRow *__restrict__ tab,
                                                const int32_t *__restrict__ aloft,
                                                const DevScalars *__restrict__ sc) {
  const int lane = threadIdx.x & 31;
  const int nti = (cov.imax - cov.imin + 32) >> 5, nj = cov.jmax - cov.jmin + 1;
  const unsigned w = blockIdx.x * 4 + (threadIdx.x >> 5), wt = w / (unsigned)nti, ws = wt / (unsigned)nseg;
  const int g = (int)(ws / (unsigned)nj), j = (int)ws - g * nj + cov.jmin;
  const int i = cov.imin + (int)(w - wt * (unsigned)nti) * 32 + lane;
  if (g >= L.ns || i > cov.imax) return;
  const int s0 = (int)(wt - ws * (unsigned)nseg) * seg + cov.kmin, s1 = min(cov.kmax, s0 + seg - 1);
  const double *q0 = cin + (long)g * L.PG + L.cell(i, j, 1);
  double *p0 = cout + (long)g * L.PG + L.cell(i, j, 1);
  if (!aloft[g] || i < box.imin || i > box.imax || j < box.jmin || j > box.jmax) {
    for (int k = s0; k <= s1; k++) p0[(long)(k - 1) * L.PY] = 0.0;
    return;
  }
  const double dt = sc->dt;
  const long TS = L.ny + 1;
  const DiffRow *T = tab + (j - 1) - TS;  // row k at T[k*TS]
  auto at = [&](int k) { return q0[(long)((k < 1 ? 1 : k > L.nz ? L.nz : k) - 1) * L.PY]; };
  double a = at(s0 - 1), b = at(s0), c = at(s0 + 1);
#pragma unroll 4
  for (int k = s0; k <= s1; k++) {
    const double next = at(k + 2);
    const DiffRow *t = T + k * TS;
    const double aL = dt * t->kz, aR = dt * t[TS].kz;
    double y;
    if (ADJ) {
      const double cL = aL * t->szL, cR = aR * t->szR;
      const double cRm = k > 1 ? aL * t[-TS].szR : cL, cLp = k < L.nz ? aR * t[TS].szL : cR;
      y = adj_diff_cell(a, b, c, cL, cR, cRm, cLp, k == 1, k == L.nz);
    } else {
      y = k >= box.kmin && k <= box.kmax ? diff_cell(a, b, c, aL, aR, t->szL, t->szR) : 0.0;
    }
    p0[(long)(k - 1) * L.PY] = y;
    a = b;
    b = c;
    c = next;
  }
}

// ---------------------------------------------------------------------------
// Crank-Nicolson line tables
// ---------------------------------------------------------------------------
// Per row of a distinct line: dgtsv's multiplier, the right-hand side's
// weights, the upper diagonal, the pivot D', and 1/D' as a sum of up to three
// doubles (exact_div.cuh, div_rn_3).  Two layouts:
//   by field, [field][row][line] (neighbouring lines in neighbouring words):
//     the x tables, whose solve runs a line per lane, and y or z tables whose
//     lines differ along i; without CN_ZL and CN_ZLL;
//   by row, [line][row][8] with D' behind it as [line][row]: the y and z
//     tables that a warp's 32 lines share, so that a chunk's rows are one
//     contiguous copy.
enum {
  CN_FACT = 0, CN_CL = 1, CN_CC = 2, CN_CR = 3, CN_DU = 4, CN_ZH = 5, CN_DP = 6, CN_NFX = 7,  // by field
  CN_ROW = 8, CN_ZL = 6, CN_ZLL = 7, CN_NF = 9                                               // by row
};

struct CnTab {
  const double *p;
  long F, U;  // rows x lines, lines
  int n;      // rows of a line
  bool byrow;
  __device__ __forceinline__ double at(int f, int l, long u) const {  // f: CN_FACT .. CN_ZH or CN_DP
    if (!byrow) return p[f * F + (long)l * U + u];
    const long r = u * n + l;
    return f == CN_DP ? p[CN_ROW * F + r] : p[CN_ROW * r + f];
  }
  // per line: the run [lo, hi] (below) and whether a pivot is one div_rn_3 does not cover
  __host__ __device__ __forceinline__ const double *runs() const { return p + (byrow ? CN_NF : CN_NFX) * F; }
};

// Constant runs.  Along a line whose geometry and diffusivity do not change
// (every x line of a lon/lat grid, every line of a projected grid with
// uniform spacing) the interior rows of the matrix are identical, and the
// elimination factors of dgtsv settle to a fixed point after a few rows, so
// the table rows become bit-identical.  Per distinct line the table keeps the
// run [lo, hi] of identical rows that ends at the last interior row
// (hi = ncells-2): row lo is stored, rows lo+1..hi of the x tables are not,
// and readers take them from registers.  The values are the same bits either
// way.
struct CnRun {
  int lo, hi;
  double v[CN_NFX];
};

__device__ __forceinline__ void cn_load_run(const CnTab &t, long u, CnRun &R) {
  const double *runs = t.runs();
  R.lo = (int)runs[u];
  R.hi = (int)runs[t.U + u];
#pragma unroll
  for (int f = 0; f < CN_NFX; f++) R.v[f] = t.p[f * t.F + (long)R.lo * t.U + u];
}

// Field f of row l of an x line: from the run registers inside (lo, hi], else from the table.
__device__ __forceinline__ double cn_coef(const CnTab &t, long u, const CnRun &R, int f, int l) {
  return (l > R.lo && l <= R.hi) ? R.v[f] : t.p[f * t.F + (long)l * t.U + u];
}

struct LineMap {  // distinct-line indexing for one sweep direction
  int na, nb;     // extents of the two fixed indices (a fastest)
  int da, db;     // 1 if the coefficients vary with a / b
  int ds;         // 1 if they vary along the sweep
  int U;          // number of distinct lines
  __host__ __device__ __forceinline__ int u(int a, int b) const {
    return (da ? a - 1 : 0) + (da ? na : 1) * (db ? b - 1 : 0);
  }
};

__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

// The tables of LPB lines per block (256 threads), in tiles of CN_TR rows:
//   the rows' coefficients (four IEEE divisions each) by all threads, then
//   the elimination -- fact = DL/D'(l-1), D' = D - fact*DU(l-1), the only
//   serial part -- by one lane per line, then the pivots' reciprocals by all.
// One thread per line doing all of it took 55 us a table on 317x211x53 (53
// lines) and 150 us on 201x151x41 over terrain; the chain of one division,
// product and difference per row is what is left.  A lane that reaches the
// fixed point of a line whose remaining interior rows have the same inputs
// stops; LPB = 1 (few lines, more rows per tile) or 32.
//
// The tables are kept between steps: st_old holds the dt this table was built
// for, and while that is the step's dt (and the host allows it, `may`: same
// box, geometry and diffusivity) the blocks return at once.  st_new is the
// slot the next launch reads, so that no block can see this launch's write.
struct CnTableJob {  // the table of one direction
  LineMap map;
  Geo3 sig, kk;
  const double *st_old;
  double *st_new, *tab;
  int may, byrow, lpb, blocks;  // blocks == 0: up to date, or no line to solve
};

template <int DIR, int LPB>
__device__ __forceinline__ void cn_table_block(const Layout &L, const Box &box, double imp, const Geo3 &kap,
                                               const CnTableJob &J, DevScalars *sc, int block, double *smem) {
  constexpr bool COMPRESS = (DIR == 0);
  constexpr int TR = LPB == 1 ? 256 : 32;  // rows per tile
  double *const sD = smem, *const sDL = sD + TR * LPB, *const sDU = sDL + TR * LPB, *const sF = sDU + TR * LPB,
                *const sP = sF + TR * LPB;
  __shared__ double cF[LPB], cP[LPB];      // fact and D' of the row before the tile
  __shared__ int sRun[LPB], sBad[LPB], sBrk;
  const LineMap &map = J.map;
  const Geo3 &sig = J.sig, &kk = J.kk;
  const int byrow = J.byrow;
  double *const __restrict__ tab = J.tab;
  const double dt = sc->dt;
  if (block == 0 && threadIdx.x == 0) *J.st_new = dt;
  if (J.may && *J.st_old == dt) return;
  const int u0 = block * LPB;
  const int tid = threadIdx.x;
  // representative fixed indices of a distinct line
  const int amin = (DIR == 0) ? box.jmin : box.imin;
  const int bmin = (DIR == 2) ? box.jmin : box.kmin;
  const int na1 = map.da ? map.na : 1;
  const int rmin = (DIR == 0) ? box.imin : (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 0) ? box.imax : (DIR == 1) ? box.jmax : box.kmax;
  const int n = rmax - rmin + 1;
  const long U = map.U, F = (long)n * U;
  auto G = [&](const Geo3 &g3, int u, int m) {
    const int a = map.da ? (u % na1) + 1 : amin, b = map.db ? (u / na1) + 1 : bmin;
    return (DIR == 0) ? g3.at(m, a, b) : (DIR == 1) ? g3.at(a, m, b) : g3.at(a, b, m);
  };
  auto put = [&](int u, int l, int f, double v) {
    if (!byrow) tab[f * F + (long)l * U + u] = v;
    else tab[CN_ROW * ((long)u * n + l) + f] = v;
  };
  if (tid == 0) sBrk = map.ds ? 0 : 1;
  if (tid < LPB) {
    sRun[tid] = n;  // first row of the final run, once known
    sBad[tid] = 0;
  }
  __syncthreads();
  if (map.ds) {  // the last interior row whose inputs differ from its predecessor's, over the block's lines
    int last = 1;
    if (LPB > 1) {
      last = n;
    } else {
      for (int l = n - 2 - tid; l >= 2 && last == 1; l -= 256) {
        const int c = rmin + l;
        bool same = true;
        for (int d = -1; d <= 1; d++)
          same = same && same_bits(G(kap, u0, c + d), G(kap, u0, c + d - 1)) &&
                 same_bits(G(kk, u0, c + d), G(kk, u0, c + d - 1)) &&
                 (d < 0 || same_bits(G(sig, u0, c + d), G(sig, u0, c + d - 1)));
        if (!same) last = l;
      }
    }
    atomicMax(&sBrk, last);
    __syncthreads();
  }
  const int brk = sBrk;
  double dp = 0.0, du = 0.0, fa = 0.0;  // of the row before (the serial lanes)
  for (int b0 = 0; b0 < n; b0 += TR) {
    const int cnt = min(TR, n - b0);
    // ---- coefficients (:794-811) ----
    for (int e = tid; e < cnt * LPB; e += 256) {
      const int ln = e % LPB, l = b0 + e / LPB, u = u0 + ln;
      if (u >= U || (l > sRun[ln] && l < n - 1 && COMPRESS)) continue;
      const int c = rmin + l;
      const double k0 = G(kap, u, c - 1), k1 = G(kap, u, c), k2 = G(kap, u, c + 1);
      const double sl = G(sig, u, c), sr = G(sig, u, c + 1);
      const double vavgL = 0.5 * (k0 + k1);
      const double kavgL = 0.5 * (G(kk, u, c - 1) + G(kk, u, c));
      const double dsL = sl / vavgL;
      const double kdsL = kavgL * dsL;
      const double vavgR = 0.5 * (k1 + k2);
      const double kavgR = 0.5 * (G(kk, u, c) + G(kk, u, c + 1));
      const double dsR = sr / vavgR;
      const double kdsR = kavgR * dsR;
      const double Lf = dt * kdsL * sl / k1;
      const double Rf = dt * kdsR * sr / k1;
      const double Cf = Lf + Rf;
      double D = 1.0 + imp * Cf;
      if (l == n - 1) D = D - imp * Rf;
      else if (l == 0) D = D - imp * Lf;
      const double DU = l == n - 1 ? 0.0 : -(imp * Rf);
      sD[e] = D;
      sDL[e] = -(imp * Lf);  // DL_d(l-1)
      sDU[e] = DU;
      put(u, l, CN_CL, (1.0 - imp) * Lf);
      put(u, l, CN_CC, 1.0 - (1.0 - imp) * Cf);
      put(u, l, CN_CR, (1.0 - imp) * Rf);
      put(u, l, CN_DU, DU);
    }
    __syncthreads();
    // ---- elimination ----
    if (tid < LPB) {
      cF[tid] = fa;
      cP[tid] = dp;
      if (u0 + tid < U) {
        int l = b0;
        if (sRun[tid] < n) l = max(l, n - 1);  // in the final run: only the last row is left
        for (; l < b0 + cnt; l++) {
          const int e = (l - b0) * LPB + tid;
          double f = 0.0, p = sD[e];
          if (l > 0) {
            f = div_rn(sDL[e], dp);
            p = p - f * du;
          }
          sF[e] = f;
          sP[e] = p;
          // (fact, D') repeat and so do all later inputs: the run that ends at row n-2
          if (l > brk && l < n - 2 && same_bits(p, dp) && same_bits(f, fa) && same_bits(sDU[e], du)) {
            sRun[tid] = l - 1;
            l = n - 2;  // the loop's next row is the last one, in this tile or a later one
          }
          dp = p;
          fa = f;
          if (l < n - 1) du = sDU[e];
        }
      }
    }
    __syncthreads();
    // ---- pivots and their reciprocals ----
    for (int e = tid; e < cnt * LPB; e += 256) {
      const int ln = e % LPB, l = b0 + e / LPB, u = u0 + ln;
      if (u >= U) continue;
      const int s = sRun[ln];
      const bool in_run = l > s && l < n - 1;
      if (in_run && COMPRESS) continue;
      // the values of row s stand for the run's; its row is in this tile or was the carry
      const int es = (s - b0) * LPB + ln;
      const double f = !in_run ? sF[e] : s >= b0 ? sF[es] : cF[ln];
      const double p = !in_run ? sP[e] : s >= b0 ? sP[es] : cP[ln];
      const double pm = l == 0 ? 1.0 : (l - 1 > s && l - 1 < n - 1) || l == b0
                                           ? (l - 1 > s && s >= b0 ? sP[es] : cP[ln])
                                           : sP[e - LPB];
      if (l > 0 && (!(fabs(pm) >= fabs(sDL[e])) || pm == 0.0)) raise_error(sc, A3G_ERR_PIVOT, l + 1);
      if (l == n - 1 && p == 0.0) raise_error(sc, A3G_ERR_PIVOT, n);
      const double zh = 1.0 / p;
      put(u, l, CN_FACT, f);
      put(u, l, CN_ZH, zh);
      if (byrow) {
        const double r = fma(-p, zh, 1.0);
        const double zl = r / p;
        put(u, l, CN_ZL, zl);
        put(u, l, CN_ZLL, fma(-p, zl, r) / p);
        tab[CN_ROW * F + (long)u * n + l] = p;
      } else {
        put(u, l, CN_DP, p);
      }
      if (!div_rn_3_covers(p)) sBad[ln] = 1;
    }
    if (__syncthreads_and(tid >= LPB || u0 + tid >= U || sRun[tid] < n) && COMPRESS && b0 + TR < n - 1)
      b0 = (n - 1) / TR * TR - TR;  // every line is in its final run: on to the last row's tile
  }
  if (tid < LPB && u0 + tid < U) {
    double *runs = tab + (byrow ? CN_NF : CN_NFX) * F;
    const int u = u0 + tid;
    runs[u] = (double)min(sRun[tid], n - 2);
    runs[U + u] = (double)(n - 2);
    runs[2 * U + u] = (double)sBad[tid];
  }
}

// The blocks of x, then y, then z.
__global__ void __launch_bounds__(256) k_cn_tables(Layout L, Box box, double imp, Geo3 kap, CnTableJob jx,
                                                   CnTableJob jy, CnTableJob jz, DevScalars *sc) {
  extern __shared__ __align__(16) double ct_smem[];
  int b = blockIdx.x;
  if (b < jx.blocks) {
    if (jx.lpb == 1) cn_table_block<0, 1>(L, box, imp, kap, jx, sc, b, ct_smem);
    else cn_table_block<0, 32>(L, box, imp, kap, jx, sc, b, ct_smem);
  } else if ((b -= jx.blocks) < jy.blocks) {
    if (jy.lpb == 1) cn_table_block<1, 1>(L, box, imp, kap, jy, sc, b, ct_smem);
    else cn_table_block<1, 32>(L, box, imp, kap, jy, sc, b, ct_smem);
  } else {
    b -= jy.blocks;
    if (jz.lpb == 1) cn_table_block<2, 1>(L, box, imp, kap, jz, sc, b, ct_smem);
    else cn_table_block<2, 32>(L, box, imp, kap, jz, sc, b, ct_smem);
  }
}
// Solve of one line (a, b) of grain g from the table.  The eliminated
// right-hand side B' is written to the output line and read back by the back
// substitution, which prefetches PF entries ahead (the loads cannot move
// above the stores to the same line on their own).
template <int DIR>
__device__ __forceinline__ void cn_line(const Layout &L, const Box &box, const LineMap &map,
                                        const double *__restrict__ cin, double *__restrict__ cout,
                                        const CnTab &tab,
                                        const int32_t *__restrict__ aloft, int a, int b, int g) {
  constexpr int PF = 4;
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  const int rmin = (DIR == 0) ? box.imin : (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 0) ? box.imax : (DIR == 1) ? box.jmax : box.kmax;
  const int ncells = rmax - rmin + 1;
  bool active;
  long base, st;
  if (DIR == 0) {
    active = a >= box.jmin && a <= box.jmax && b >= box.kmin && b <= box.kmax;
    base = L.cell(1, a, b); st = 1;
  } else if (DIR == 1) {
    active = a >= box.imin && a <= box.imax && b >= box.kmin && b <= box.kmax;
    base = L.cell(a, 1, b); st = L.P;
  } else {
    active = a >= box.imin && a <= box.imax && b >= box.jmin && b <= box.jmax;
    base = L.cell(a, b, 1); st = L.PY;
  }
  base += (long)g * L.PG;
  const double *q = cin + base;
  double *x = cout + base;
  if (!active || !aloft[g]) {
    for (int c = 1; c <= n; c++) x[(long)(c - 1) * st] = 0.0;
    return;
  }
  for (int c = 1; c < rmin; c++) x[(long)(c - 1) * st] = 0.0;
  for (int c = rmax + 1; c <= n; c++) x[(long)(c - 1) * st] = 0.0;
  const long u = map.u(a, b);
  CnRun R;
  if (DIR == 0) cn_load_run(tab, u, R);
  auto co = [&](int f, int l) {  // the y and z tables are stored in full
    return (DIR == 0) ? cn_coef(tab, u, R, f, l) : tab.at(f, l, u);
  };
  const double *qq = q + (long)(rmin - 1) * st;  // cell rmin
  double *xx = x + (long)(rmin - 1) * st;
  // forward elimination with the right-hand side built on the fly, :813-851
  double qm = qq[0];  // BC_left_t0 = q(rmin)
  double qc = qm;
  double bp = 0.0;
#pragma unroll 4
  for (int l = 0; l < ncells; l++) {
    const double qp = (l + 1 < ncells) ? qq[(long)(l + 1) * st] : qc;  // BC_right_t0 = q(rmax)
    const double B = co(CN_CL, l) * qm + co(CN_CC, l) * qc +
                     co(CN_CR, l) * qp;
    bp = (l == 0) ? B : B - co(CN_FACT, l) * bp;
    xx[(long)l * st] = bp;
    qm = qc;
    qc = qp;
  }
  // back substitution with a PF-deep prefetch of B'
  double ring[PF];
#pragma unroll
  for (int p = 0; p < PF; p++) ring[p] = (ncells - 1 - p >= 0) ? xx[(long)(ncells - 1 - p) * st] : 0.0;
  double xn = 0.0;
  for (int l0 = ncells - 1; l0 >= 0; l0 -= PF) {
#pragma unroll
    for (int p = 0; p < PF; p++) {
      const int l = l0 - p;
      if (l >= 0) {
        const double b2 = ring[p];
        const int lp = l - PF;  // refill this slot for the next round
        ring[p] = (lp >= 0) ? xx[(long)lp * st] : 0.0;
        const double num = (l == ncells - 1) ? b2 : b2 - co(CN_DU, l) * xn;
        const double v = div_rn_rcp(num, co(CN_DP, l), co(CN_ZH, l));
        xx[(long)l * st] = v;
        xn = v;
      }
    }
  }
}

// y and z lines, GC grains of one line per thread: the factor-table row is
// the same for every grain, so its loads are shared, and the GC recurrences
// are independent chains the scheduler interleaves.  Same operations per
// grain as cn_line.
template <int DIR, int GC>
__device__ __forceinline__ void cn_line_gc(const Layout &L, const Box &box, const LineMap &map,
                                           const double *__restrict__ cin, double *__restrict__ cout,
                                           const CnTab &tab,
                                           const int32_t *__restrict__ aloft, int a, int b, int g0) {
  constexpr int PF = 4;
  const int n = (DIR == 1) ? L.ny : L.nz;
  const int rmin = (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 1) ? box.jmax : box.kmax;
  const int ncells = rmax - rmin + 1;
  bool active;
  long base, st;
  if (DIR == 1) {
    active = a >= box.imin && a <= box.imax && b >= box.kmin && b <= box.kmax;
    base = L.cell(a, 1, b); st = L.P;
  } else {
    active = a >= box.imin && a <= box.imax && b >= box.jmin && b <= box.jmax;
    base = L.cell(a, b, 1); st = L.PY;
  }
  const double *q[GC];
  double *x[GC];
  bool on[GC], any = false;
#pragma unroll
  for (int u = 0; u < GC; u++) {
    const int g = g0 + u < L.ns ? g0 + u : L.ns - 1;
    q[u] = cin + base + (long)g * L.PG;
    x[u] = cout + base + (long)g * L.PG;
    on[u] = g0 + u < L.ns && active && aloft[g] != 0;
    any = any || on[u];
    if (g0 + u < L.ns && !on[u])
      for (int c = 1; c <= n; c++) x[u][(long)(c - 1) * st] = 0.0;
    else if (on[u]) {
      for (int c = 1; c < rmin; c++) x[u][(long)(c - 1) * st] = 0.0;
      for (int c = rmax + 1; c <= n; c++) x[u][(long)(c - 1) * st] = 0.0;
    }
  }
  if (!any) return;
  const long line = map.u(a, b);
  auto co = [&](int f, int l) { return tab.at(f, l, line); };
  const long off = (long)(rmin - 1) * st;
  // forward elimination with the right-hand side built on the fly, :813-851
  double qm[GC], qc[GC], bp[GC];
#pragma unroll
  for (int u = 0; u < GC; u++) {
    qm[u] = on[u] ? q[u][off] : 0.0;  // BC_left_t0 = q(rmin)
    qc[u] = qm[u];
    bp[u] = 0.0;
  }
#pragma unroll 4
  for (int l = 0; l < ncells; l++) {
    const double cl = co(CN_CL, l), cc = co(CN_CC, l), cr = co(CN_CR, l), fa = co(CN_FACT, l);
#pragma unroll
    for (int u = 0; u < GC; u++) {
      const double qp = (l + 1 < ncells) ? (on[u] ? q[u][off + (long)(l + 1) * st] : 0.0) : qc[u];
      const double B = cl * qm[u] + cc * qc[u] + cr * qp;
      bp[u] = (l == 0) ? B : B - fa * bp[u];
      if (on[u]) x[u][off + (long)l * st] = bp[u];
      qm[u] = qc[u];
      qc[u] = qp;
    }
  }
  // back substitution with a PF-deep prefetch of B'
  double ring[GC][PF];
#pragma unroll
  for (int u = 0; u < GC; u++)
#pragma unroll
    for (int p = 0; p < PF; p++)
      ring[u][p] = (on[u] && ncells - 1 - p >= 0) ? x[u][off + (long)(ncells - 1 - p) * st] : 0.0;
  double xn[GC];
#pragma unroll
  for (int u = 0; u < GC; u++) xn[u] = 0.0;
  for (int l0 = ncells - 1; l0 >= 0; l0 -= PF) {
#pragma unroll
    for (int p = 0; p < PF; p++) {
      const int l = l0 - p;
      if (l >= 0) {
        const int lp = l - PF;
        const double du = co(CN_DU, l), dp = co(CN_DP, l), rd = co(CN_ZH, l);
#pragma unroll
        for (int u = 0; u < GC; u++) {
          const double b2 = ring[u][p];
          ring[u][p] = (on[u] && lp >= 0) ? x[u][off + (long)lp * st] : 0.0;
          const double num = (l == ncells - 1) ? b2 : b2 - du * xn[u];
          const double v = div_rn_rcp(num, dp, rd);
          if (on[u]) x[u][off + (long)l * st] = v;
          xn[u] = v;
        }
      }
    }
  }
}

template <int DIR, int GC>
__device__ __forceinline__ void cn_solve_gc_thread(const Layout &L, const Box &box, const LineMap &map,
                                                   const double *__restrict__ cin,
                                                   double *__restrict__ cout,
                                                   const CnTab &tab,
                                                   const int32_t *__restrict__ aloft) {
  const int na = L.nx;
  const int nb = (DIR == 2) ? L.ny : L.nz;
  const int ngr = (L.ns + GC - 1) / GC;
  const long nlines = (long)na * nb * ngr;
  const long w = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (w >= nlines) return;
  const int a = (int)(w % na) + 1;
  const long r = w / na;
  const int b = (int)(r % nb) + 1;
  const int gg = (int)(r / nb);
  cn_line_gc<DIR, GC>(L, box, map, cin, cout, tab, aloft, a, b, gg * GC);
}

// z lines: unconstrained registers (64-96, no spills) measured fastest; an
// 8-blocks-per-SM bound slowed the C2 z solve 1.29 -> 1.37 ms on B200.
template <int DIR, int GC>
__global__ void __launch_bounds__(128) k_cn_solve_gc(Layout L, Box box, LineMap map,
                                                     const double *__restrict__ cin,
                                                     double *__restrict__ cout,
                                                     CnTab tab,
                                                     const int32_t *__restrict__ aloft) {
  cn_solve_gc_thread<DIR, GC>(L, box, map, cin, cout, tab, aloft);
}

// y lines: 12 blocks of 128 per SM (at most 40 registers, some spilled to
// L1) hide the strided dependent loads better (C2 1.76 -> 1.62 ms on B200).
template <int GC>
__global__ void __launch_bounds__(128, 12) k_cn_solve_gc_y(Layout L, Box box, LineMap map,
                                                           const double *__restrict__ cin,
                                                           double *__restrict__ cout,
                                                           CnTab tab,
                                                           const int32_t *__restrict__ aloft) {
  cn_solve_gc_thread<1, GC>(L, box, map, cin, cout, tab, aloft);
}

template <int DIR, int GC>
static void launch_cn_solve_gc(a3g_ctx *ctx, const LineMap &map, const CnTab &tab) {
  const Layout &L = ctx->L;
  const long n = (long)map.na * map.nb * ((L.ns + GC - 1) / GC);
  const unsigned grid = (unsigned)((n + 127) / 128);
  if constexpr (DIR == 1)
    k_cn_solve_gc_y<GC><<<grid, 128, 0, ctx->stream>>>(L, ctx->box, map, ctx->c0, ctx->c1, tab, ctx->aloft);
  else
    k_cn_solve_gc<DIR, GC><<<grid, 128, 0, ctx->stream>>>(L, ctx->box, map, ctx->c0, ctx->c1, tab, ctx->aloft);
}

// y and z lines that no tile takes: coefficients that vary along i (terrain),
// where no two lanes share a table row, and columns of more than 256 levels,
// whose 32 share a table by row (ROWS).  A warp holds 32 neighbouring lines of
// one grain and its block the same lines of the other grains, which so find the
// table rows in L1; rows are taken CB_U at a time, all their loads before the
// first of the dependent operations.  Bound by the latency of those loads and
// the memory behind them: a thread per line with a row at a time waited for one
// row after another (201x151x41, 5 grains over terrain: y 324 -> 64 us, z 84 ->
// 69 us; z of 160x160x300, 1 grain: 192 us, 222 over a table by row, 77 here).
constexpr int CB_U = 8, CB_WARPS = 8;

// Lines of 32 neighbouring i: where a thread's line of direction DIR starts.
template <int DIR>
__device__ __forceinline__ bool cb_line(const Layout &L, int *a, int *b, int *g, long *base, long *st) {
  const int nti = (L.nx + 31) >> 5;
  *b = (int)(blockIdx.x / (unsigned)nti) + 1;
  *a = (int)(blockIdx.x % (unsigned)nti) * 32 + (int)(threadIdx.x & 31) + 1;
  *g = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (*a > L.nx || *g >= L.ns) return false;
  *base = (DIR == 1 ? L.cell(*a, 1, *b) : L.cell(*a, *b, 1)) + (long)*g * L.PG;
  *st = DIR == 1 ? L.P : L.PY;
  return true;
}
template <int DIR>
static dim3 cb_grid(const Layout &L, int *threads) {
  const int w = L.ns < CB_WARPS ? L.ns : CB_WARPS;
  *threads = 32 * w;
  return dim3(((L.nx + 31) / 32) * (DIR == 1 ? L.nz : L.ny), (L.ns + w - 1) / w);
}

template <int DIR, bool ROWS>
__global__ void __launch_bounds__(32 * CB_WARPS, 2) k_cn_solve_b(Layout L, Box box, LineMap map,
                                                                 const double *__restrict__ cin,
                                                                 double *__restrict__ cout, CnTab tab,
                                                                 const int32_t *__restrict__ aloft) {
  int a, b, g;
  long base, st;
  if (!cb_line<DIR>(L, &a, &b, &g, &base, &st)) return;
  const int n = (DIR == 1) ? L.ny : L.nz;
  const int rmin = (DIR == 1) ? box.jmin : box.kmin, rmax = (DIR == 1) ? box.jmax : box.kmax;
  const int ncells = rmax - rmin + 1;
  const bool in = a >= box.imin && a <= box.imax && b >= ((DIR == 1) ? box.kmin : box.jmin) &&
                  b <= ((DIR == 1) ? box.kmax : box.jmax) && aloft[g] != 0;
  double *x = cout + base;
  if (!in) {
    for (int c = 1; c <= n; c++) x[(long)(c - 1) * st] = 0.0;
    return;
  }
  for (int c = 1; c < rmin; c++) x[(long)(c - 1) * st] = 0.0;
  for (int c = rmax + 1; c <= n; c++) x[(long)(c - 1) * st] = 0.0;
  const long u = map.u(a, b);
  const double *qq = cin + base + (long)(rmin - 1) * st;
  x += (long)(rmin - 1) * st;
  const double *tp = ROWS ? tab.p + CN_ROW * u * ncells : tab.p + u;
  const double *dpp = tab.p + CN_ROW * tab.F + u * ncells;  // D' of a table by row
  auto co = [&](int f, int l) {
    if (ROWS) return __ldg(f == CN_DP ? dpp + l : tp + (long)CN_ROW * l + f);
    return __ldg(tp + f * tab.F + (long)l * tab.U);
  };
  // forward elimination with the right-hand side built on the fly, :813-851
  double qm = __ldg(qq), qc = qm, bp = 0.0;  // BC_left_t0 = q(rmin)
  int l = 0;
  for (; l + CB_U < ncells; l += CB_U) {
    double q[CB_U], cl[CB_U], cc[CB_U], cr[CB_U], fa[CB_U];
#pragma unroll
    for (int e = 0; e < CB_U; e++) {
      q[e] = __ldg(qq + (long)(l + 1 + e) * st);
      cl[e] = co(CN_CL, l + e);
      cc[e] = co(CN_CC, l + e);
      cr[e] = co(CN_CR, l + e);
      fa[e] = co(CN_FACT, l + e);
    }
#pragma unroll
    for (int e = 0; e < CB_U; e++) {
      const double B = cl[e] * qm + cc[e] * qc + cr[e] * q[e];
      bp = (e == 0 && l == 0) ? B : B - fa[e] * bp;
      x[(long)(l + e) * st] = bp;
      qm = qc;
      qc = q[e];
    }
  }
  for (; l < ncells; l++) {
    const double qp = l + 1 < ncells ? __ldg(qq + (long)(l + 1) * st) : qc;  // BC_right_t0 = q(rmax)
    const double B = co(CN_CL, l) * qm + co(CN_CC, l) * qc + co(CN_CR, l) * qp;
    bp = (l == 0) ? B : B - co(CN_FACT, l) * bp;
    x[(long)l * st] = bp;
    qm = qc;
    qc = qp;
  }
  // back substitution
  double xn = div_rn_rcp(bp, co(CN_DP, ncells - 1), co(CN_ZH, ncells - 1));
  x[(long)(ncells - 1) * st] = xn;
  l = ncells - 2;  // the next row to do
  for (; l >= CB_U - 1; l -= CB_U) {
    double y[CB_U], du[CB_U], dp[CB_U], zh[CB_U];
#pragma unroll
    for (int e = 0; e < CB_U; e++) {
      y[e] = x[(long)(l - e) * st];
      du[e] = co(CN_DU, l - e);
      dp[e] = co(CN_DP, l - e);
      zh[e] = co(CN_ZH, l - e);
    }
#pragma unroll
    for (int e = 0; e < CB_U; e++) {
      xn = div_rn_rcp(y[e] - du[e] * xn, dp[e], zh[e]);
      x[(long)(l - e) * st] = xn;
    }
  }
  for (; l >= 0; l--) {
    xn = div_rn_rcp(x[(long)l * st] - co(CN_DU, l) * xn, co(CN_DP, l), co(CN_ZH, l));
    x[(long)l * st] = xn;
  }
}

// 32 x rows of a grain to a warp, their cells in chunks of 32 through a shared
// tile: row segments come and go coalesced, the lanes work along their own
// rows in between, and the chunk after is on its way (in registers) while one
// is worked on.  A block's warps hold the same rows of several grains.
constexpr int RT_WARPS = 5, RT_S = 33;

struct RowTile {
  double *tile, *own;
  int lane, r0, nr, n, j, k, g;  // first row of the level, rows, cells; this lane's row
  long P;
  __device__ __forceinline__ bool init(const Layout &L, double *t, int cells) {
    lane = threadIdx.x & 31;
    g = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (g >= L.ns) return false;
    const int plane = L.ny * L.nz, p0 = blockIdx.x * 32;
    nr = plane - p0 < 32 ? plane - p0 : 32;
    r0 = g * plane + p0;
    const int pr = lane < nr ? p0 + lane : plane - 1;
    k = pr / L.ny + 1;
    j = pr - (k - 1) * L.ny + 1;
    n = cells;
    P = L.P;
    tile = t;
    own = t + lane * RT_S;
    return true;
  }
  // cell c0 + lane of every row, from src (cell 0 of the level's first row)
  __device__ __forceinline__ void fetch(double (&next)[32], const double *src, int c0) const {
    const double *p = src + (long)r0 * P + c0 + lane;
#pragma unroll
    for (int e = 0; e < 32; e++) next[e] = (e < nr && c0 + lane < n) ? p[(long)e * P] : 0.0;
  }
  __device__ __forceinline__ void fill(const double (&next)[32]) const {
#pragma unroll
    for (int e = 0; e < 32; e++) tile[e * RT_S + lane] = next[e];
    __syncwarp();
  }
  // columns col.. of the tile to the cells c0.. of every row
  __device__ __forceinline__ void drain(double *dst, int c0, int col, int cnt) const {
    __syncwarp();
    double *p = dst + (long)r0 * P + c0 + lane;
    if (lane < cnt) {
#pragma unroll 8
      for (int e = 0; e < nr; e++) p[(long)e * P] = tile[e * RT_S + col + lane];
    }
    __syncwarp();
  }
};
static dim3 rt_grid(const Layout &L, int *threads) {
  const int w = L.ns < RT_WARPS ? L.ns : RT_WARPS;
  *threads = 32 * w;
  return dim3((L.ny * L.nz + 31) / 32, (L.ns + w - 1) / w);
}

// x lines whose coefficients vary along them (terrain): B' goes out and comes
// back, the table rows are taken CB_U at a time.  Bound by the latency of
// those loads; k_cn_solve_xt2, whose fast path needs lines that settle to one
// row, waits for each of them (201x151x41, 5 grains: 298 -> 138 us).  Four
// warps a block (two groups for 5 grains, a second wave) measured 194 us.
__global__ void __launch_bounds__(32 * RT_WARPS, 2) k_cn_solve_xv(Layout L, Box box, LineMap map,
                                                                  const double *__restrict__ cin,
                                                                  double *__restrict__ cout, CnTab tab,
                                                                  const int32_t *__restrict__ aloft) {
  __shared__ double sh[RT_WARPS][32 * RT_S];
  const int n = box.imax - box.imin + 1, nch = (n + 31) >> 5;
  RowTile T;
  if (!T.init(L, sh[threadIdx.x >> 5], n)) return;  // uniform over the warp
  const bool act = T.j >= box.jmin && T.j <= box.jmax && T.k >= box.kmin && T.k <= box.kmax && aloft[T.g] != 0;
  if (n < L.nx)  // cells outside the box
    for (int row = 0; row < T.nr; row++) {
      double *xr = cout + (long)(T.r0 + row) * L.P;
      for (int c = T.lane; c < box.imin - 1; c += 32) xr[c] = 0.0;
      for (int c = box.imax + T.lane; c < L.nx; c += 32) xr[c] = 0.0;
    }
  cin += box.imin - 1;
  cout += box.imin - 1;
  const double *q_own = cin + (long)(T.r0 + (T.lane < T.nr ? T.lane : 0)) * L.P;
  const long u = map.u(T.j, T.k);
  CnRun R;
  cn_load_run(tab, u, R);
  auto co = [&](int f, int l) { return cn_coef(tab, u, R, f, l); };
  double next[32];
  double *const own = T.own;
  // forward elimination with the right-hand side built on the fly, :813-851
  T.fetch(next, cin, 0);
  double qm = 0.0, qc = 0.0, bp = 0.0;
  for (int ch = 0; ch < nch; ch++) {
    const int c0 = 32 * ch, cnt = n - c0 < 32 ? n - c0 : 32;
    T.fill(next);
    if (ch + 1 < nch) {
      own[32] = q_own[c0 + 32];
      T.fetch(next, cin, c0 + 32);
    } else {
      own[cnt] = own[cnt - 1];  // BC_right_t0 = q(rmax)
    }
    if (ch == 0) qm = own[0];  // BC_left_t0 = q(rmin)
    qc = own[0];
    for (int e0 = 0; e0 < cnt; e0 += CB_U) {
      double cl[CB_U], cc[CB_U], cr[CB_U], fa[CB_U];
#pragma unroll
      for (int e = 0; e < CB_U; e++) {
        const int l = c0 + e0 + e < n ? c0 + e0 + e : n - 1;
        cl[e] = co(CN_CL, l);
        cc[e] = co(CN_CC, l);
        cr[e] = co(CN_CR, l);
        fa[e] = co(CN_FACT, l);
      }
#pragma unroll
      for (int e = 0; e < CB_U; e++) {
        if (e0 + e >= cnt) break;
        const double qp = own[e0 + e + 1];
        const double B = cl[e] * qm + cc[e] * qc + cr[e] * qp;
        bp = (e == 0 && c0 + e0 == 0) ? B : B - fa[e] * bp;
        own[e0 + e] = bp;
        qm = qc;
        qc = qp;
      }
    }
    if (ch + 1 < nch) T.drain(cout, c0, 0, cnt);
  }
  // back substitution; the last chunk is still in the tile
  double xn = 0.0;
  __syncwarp();
  for (int ch = nch - 1; ch >= 0; ch--) {
    const int c0 = 32 * ch, cnt = n - c0 < 32 ? n - c0 : 32;
    if (ch != nch - 1) T.fill(next);
    if (ch > 0) T.fetch(next, cout, c0 - 32);
    for (int e0 = cnt - 1; e0 >= 0; e0 -= CB_U) {
      double du[CB_U], dp[CB_U], zh[CB_U];
#pragma unroll
      for (int e = 0; e < CB_U; e++) {
        const int l = c0 + e0 - e > 0 ? c0 + e0 - e : 0;
        du[e] = co(CN_DU, l);
        dp[e] = co(CN_DP, l);
        zh[e] = co(CN_ZH, l);
      }
#pragma unroll
      for (int e = 0; e < CB_U; e++) {
        if (e0 - e < 0) break;
        const double b = own[e0 - e];
        xn = div_rn_rcp((e == 0 && c0 + e0 == n - 1) ? b : b - du[e] * xn, dp[e], zh[e]);
        own[e0 - e] = act ? xn : 0.0;
      }
    }
    T.drain(cout, c0, 0, cnt);
  }
}

// Solve kernel: one thread per line (a, b, grain), lines enumerated with a
// fastest so that a warp holds neighbouring lines (neighbouring i for y and
// z lines: coalesced loads and stores).
template <int DIR>
__global__ void __launch_bounds__(128) k_cn_solve(Layout L, Box box, LineMap map,
                                                  const double *__restrict__ cin,
                                                  double *__restrict__ cout,
                                                  CnTab tab,
                                                  const int32_t *__restrict__ aloft) {
  const int na = (DIR == 0) ? L.ny : L.nx;
  const int nb = (DIR == 2) ? L.ny : L.nz;
  const long nlines = (long)na * nb * L.ns;
  const long w = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (w >= nlines) return;
  const int a = (int)(w % na) + 1;
  const long r = w / na;
  const int b = (int)(r % nb) + 1;
  const int g = (int)(r / nb);
  cn_line<DIR>(L, box, map, cin, cout, tab, aloft, a, b, g);
}

// x lines, warp-tiled.  A warp owns 32 consecutive x rows (row r =
// (g*nz + k-1)*ny + j-1 starts at r*P) and walks them in chunks of 32 cells
// through a shared-memory tile: every global load and store of the
// concentration is a coalesced 256-byte row segment, and each lane then runs
// its own row's recurrence out of the tile.
//   pass 1 (forward): the elimination of B' over the whole row, keeping only
//     B' at the last cell of every chunk (a checkpoint, parked in the output
//     row at that cell);
//   pass 2 (backward, last chunk first): reload the chunk, recompute its B'
//     from the checkpoint of the previous chunk (same operations, same bits),
//     back-substitute, store the chunk.
// Against writing B' out and reading it back this moves one read of the
// input in place of a write and a read of B'.
constexpr int XT_WARPS = 4;
constexpr int XT_S = 35;  // tile row stride in doubles: 34 columns, odd stride

__global__ void __launch_bounds__(128, 5) k_cn_solve_xt(Layout L, Box box, LineMap map,
                                                     const double *__restrict__ cin,
                                                     double *__restrict__ cout,
                                                     CnTab tab,
                                                     const int32_t *__restrict__ aloft) {
  __shared__ double sh[XT_WARPS][32 * XT_S];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double *tile = sh[w];
  const long nrows = (long)L.ny * L.nz * L.ns;
  const long r0 = ((long)blockIdx.x * XT_WARPS + w) * 32;
  if (r0 >= nrows) return;  // uniform over the warp
  const long r = r0 + lane;
  const bool valid = r < nrows;
  const long rc = valid ? r : nrows - 1;
  const int j = (int)(rc % L.ny) + 1;
  const long t1 = rc / L.ny;
  const int k = (int)(t1 % L.nz) + 1;
  const int g = (int)(t1 / L.nz);
  const bool active =
      valid && j >= box.jmin && j <= box.jmax && k >= box.kmin && k <= box.kmax && aloft[g] != 0;
  const unsigned amask = __ballot_sync(0xffffffffu, active);
  const int nvalid = (int)((nrows - r0) < 32 ? (nrows - r0) : 32);
  const int rmin = box.imin, rmax = box.imax;
  const int ncells = rmax - rmin + 1;
  const long P = L.P;
  if (valid) {  // cells outside [rmin, rmax] (FAST_SUBGRID box)
    double *xr = cout + r * P;
    for (int c = 1; c < rmin; c++) xr[c - 1] = 0.0;
    for (int c = rmax + 1; c <= L.nx; c++) xr[c - 1] = 0.0;
  }
  const double *q0 = cin + r0 * P + (rmin - 1);  // row r0, cell rmin
  double *x0 = cout + r0 * P + (rmin - 1);
  const double *qown = q0 + (long)lane * P;
  double *xown = x0 + (long)lane * P;
  const long u = map.u(j, k);
  CnRun R;
  cn_load_run(tab, u, R);
  double *tr = tile + lane * XT_S;  // this lane's row of the tile
  const int nch = (ncells + 31) >> 5;

  // tile columns: 0 = cell l0-1, 1..32 = cells l0..l0+31, 33 = cell l0+32
  auto load_tile = [&](int l0, int cnt) {
#pragma unroll
    for (int h = 0; h < 32; h += 8) {
      double v[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const int row = h + e;
        v[e] = (row < nvalid && lane < cnt) ? q0[(long)row * P + l0 + lane] : 0.0;
      }
#pragma unroll
      for (int e = 0; e < 8; e++) tile[(h + e) * XT_S + 1 + lane] = v[e];
    }
    tr[0] = (valid && l0 > 0) ? qown[l0 - 1] : 0.0;
    tr[33] = (valid && l0 + 32 < ncells) ? qown[l0 + 32] : 0.0;
    __syncwarp();
  };

  // A chunk whose rows all lie inside every lane's constant run (rows
  // lo_w+1 .. ncells-2, lo_w the warp's largest lo) takes its coefficients
  // from registers with no per-row test: the fast path.
  int lo_w = R.lo;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lo_w = max(lo_w, __shfl_xor_sync(0xffffffffu, lo_w, o));
  auto fast_chunk = [&](int l0, int cnt) { return cnt == 32 && l0 > lo_w && l0 + 31 <= ncells - 2; };
  const double fCL = R.v[CN_CL], fCC = R.v[CN_CC], fCR = R.v[CN_CR], fFA = R.v[CN_FACT];
  const double fDU = R.v[CN_DU], fDP = R.v[CN_DP], fRD = R.v[CN_ZH];

  // pass 1: forward elimination, checkpoints only (:813-851 and dgtsv)
  double qm = 0.0, qc = 0.0, bp = 0.0;
  for (int ch = 0; ch < nch; ch++) {
    const int l0 = ch << 5;
    const int cnt = (ncells - l0) < 32 ? (ncells - l0) : 32;
    load_tile(l0, cnt);
    if (ch == 0) {
      qm = tr[1];  // BC_left_t0 = q(rmin)
      qc = qm;
    }
    if (fast_chunk(l0, cnt)) {  // rows l0..l0+31 < ncells-1: qp always from the tile
#pragma unroll 8
      for (int c = 0; c < 32; c++) {
        const double qp = tr[c + 2];
        const double B = fCL * qm + fCC * qc + fCR * qp;
        bp = B - fFA * bp;
        qm = qc;
        qc = qp;
      }
      if (valid && ch + 1 < nch) xown[l0 + 31] = bp;
      __syncwarp();
      continue;
    }
    for (int c = 0; c < cnt; c++) {
      const int l = l0 + c;
      const double qp = (l + 1 < ncells) ? tr[c + 2] : qc;  // BC_right_t0 = q(rmax)
      const double B = cn_coef(tab, u, R, CN_CL, l) * qm + cn_coef(tab, u, R, CN_CC, l) * qc +
                       cn_coef(tab, u, R, CN_CR, l) * qp;
      bp = (l == 0) ? B : B - cn_coef(tab, u, R, CN_FACT, l) * bp;
      qm = qc;
      qc = qp;
    }
    if (valid && ch + 1 < nch) xown[l0 + 31] = bp;  // checkpoint B'(l0+31)
    __syncwarp();
  }

  // pass 2: per chunk, last first: recompute B', back-substitute, store
  double xn = 0.0;
  for (int ch = nch - 1; ch >= 0; ch--) {
    const int l0 = ch << 5;
    const int cnt = (ncells - l0) < 32 ? (ncells - l0) : 32;
    load_tile(l0, cnt);
    double bq = (valid && ch > 0) ? xown[l0 - 1] : 0.0;
    double qm2 = (ch == 0) ? tr[1] : tr[0];
    double qc2 = tr[1];
    if (fast_chunk(l0, cnt)) {
#pragma unroll 8
      for (int c = 0; c < 32; c++) {
        const double qp = tr[c + 2];
        const double B = fCL * qm2 + fCC * qc2 + fCR * qp;
        bq = B - fFA * bq;
        tr[c + 1] = bq;
        qm2 = qc2;
        qc2 = qp;
      }
#pragma unroll 8
      for (int c = 31; c >= 0; c--) {
        const double num = tr[c + 1] - fDU * xn;
        const double v = div_rn_rcp(num, fDP, fRD);
        tr[c + 1] = v;
        xn = v;
      }
    } else {
    for (int c = 0; c < cnt; c++) {
      const int l = l0 + c;
      const double qp = (l + 1 < ncells) ? tr[c + 2] : qc2;
      const double B = cn_coef(tab, u, R, CN_CL, l) * qm2 + cn_coef(tab, u, R, CN_CC, l) * qc2 +
                       cn_coef(tab, u, R, CN_CR, l) * qp;
      bq = (l == 0) ? B : B - cn_coef(tab, u, R, CN_FACT, l) * bq;
      tr[c + 1] = bq;
      qm2 = qc2;
      qc2 = qp;
    }
    for (int c = cnt - 1; c >= 0; c--) {
      const int l = l0 + c;
      const double b2 = tr[c + 1];
      const double num = (l == ncells - 1) ? b2 : b2 - cn_coef(tab, u, R, CN_DU, l) * xn;
      const double v = div_rn_rcp(num, cn_coef(tab, u, R, CN_DP, l), cn_coef(tab, u, R, CN_ZH, l));
      tr[c + 1] = v;
      xn = v;
    }
    }
    __syncwarp();
#pragma unroll 8
    for (int row = 0; row < 32; row++) {
      if (row < nvalid && lane < cnt)
        x0[(long)row * P + l0 + lane] = ((amask >> row) & 1u) ? tile[row * XT_S + 1 + lane] : 0.0;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// The tiled solves through TMA (x, y and z).  Each lane runs one line:
//   forward  B' = (CL*q(l-1) + CC*q(l) + CR*q(l+1)) - FACT*B'(l-1)
//   backward x(l) = (B' - DU*x(l+1)) / D'
// in cn_line's operations (row 0 has FACT = 0 and the last row DU = 0, so that
// the end rows need no tests).  The division is the three dependent
// operations of div_rn_3: a batch of rows runs without a branch, and the rare
// batch with a dividend outside its range (a diffused tail below 2^-900) or a
// pivot it does not cover is done again with the division operator.
// ---------------------------------------------------------------------------
constexpr int ZT_BAR_BYTES = 128;  // barriers ahead of the tiles (keeps tiles 128-byte aligned)

// x lines.  A warp owns 32 consecutive rows (row r = (g*nz + k-1)*ny + j-1 at
// r*P), a row per lane, and walks them in chunks of CX_CH cells that arrive
// and leave by tensor copies in the 128-byte swizzle (the lanes' 16-byte
// accesses of their own rows meet no bank twice), three buffers turning.
// Positions count cells from the even cell at or before the box's first one
// (the 16-byte rule).
//   pass 1 (forward): the elimination over the row, keeping only B' of every
//     chunk's first cell, parked in the output where the chunk will go (the
//     32 lanes' values side by side in its first two rows; the last chunk's
//     stays in a register);
//   pass 2 (backward, last chunk first): the chunk's other B' again from the
//     parked one, read a chunk ahead (same operations, same bits), back
//     substitution in place, and the chunk's store.
// Chunks are loaded 0 .. nch-1, then nch-2 .. 0: the last one of pass 1 is
// still in its buffer for pass 2.  Chunks inside every lane's constant run
// take their coefficients from registers.
//
// Bound by the latency of the two recurrences at 16 warps per SM (registers),
// with 24 B per cell of traffic at 5.3 TB/s.  720x360x60, 10 grains, ash in
// every cell: 1.15 -> 0.70 ms (a cloud in still air, whose tails go by the
// division operator, 1.27 -> 0.82), 317x211x53, 7 grains: 275 -> 180 us, against
// dense tiles that the lanes copied into an odd-stride one and certified
// quotients (96 warp instructions a cell against 55).  Issuing loads two chunks
// ahead instead of one changed nothing; parking the values a sector each per row
// cost 1.33 ms.
constexpr int CXT_WARPS = 2;
constexpr int CXT_BUF = 32 * CX_CH * 8;
constexpr int CXT_SMEM = 1024 + 1024 + CXT_WARPS * 3 * CXT_BUF;  // room to align, barriers, buffers

__global__ void __launch_bounds__(32 * CXT_WARPS, 8) k_cn_solve_xt2(const __grid_constant__ CUtensorMap tin,
                                                                   const __grid_constant__ CUtensorMap tout,
                                                                   Layout L, Box box, RowCover cov, LineMap map,
                                                                   double *__restrict__ cout, CnTab tab,
                                                                   const int32_t *__restrict__ aloft,
                                                                   DevScalars *sc) {
  extern __shared__ unsigned char x2_smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned char *const sm = x2_smem + ((1024u - (smem_u32(x2_smem) & 1023u)) & 1023u);  // the swizzle's period
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm) + 3 * w;
  unsigned char *const bufs = sm + 1024 + w * 3 * CXT_BUF;
  const unsigned tw = blockIdx.x * CXT_WARPS + w;
  const int g = (int)(tw / (unsigned)cov.ntile);
  if (g >= L.ns) return;  // uniform over the warp
  int p0, pend;  // the tile's first row of the plane, the end of its run of rows
  cov.tile((int)(tw - (unsigned)g * (unsigned)cov.ntile), &p0, &pend);
  const int r0 = g * L.ny * L.nz + p0, nval = min(32, pend - p0);  // its first row of the level, its own rows
  const bool valid = lane < nval;
  const int pr = valid ? p0 + lane : pend - 1;
  const int k = pr / L.ny + 1, j = pr - (k - 1) * L.ny + 1;
  const bool active =
      valid && j >= box.jmin && j <= box.jmax && k >= box.kmin && k <= box.kmax && aloft[g] != 0;
  const int rmin = box.imin, rmax = box.imax;
  const int ncells = rmax - rmin + 1;
  const long P = L.P;
  const int xa = (rmin - 1) & ~1, off = (rmin - 1) - xa;  // 0-based cell of position 0; positions before the box
  const int np = off + ncells, nch = (np + CX_CH - 1) / CX_CH;
  const bool any = __any_sync(0xffffffffu, active);
  {  // cells of the cover that no chunk store reaches: zeros
    const int za = any ? xa : cov.x1, zb = any ? xa + nch * CX_CH : cov.x1;
    if (za > cov.x0 - 1 || zb < cov.x1)
      for (int row = 0; row < nval; row++) {
        double *xr = cout + (long)(r0 + row) * P;
        for (int c = cov.x0 - 1 + lane; c < za; c += 32) xr[c] = 0.0;
        for (int c = zb + lane; c < cov.x1; c += 32) xr[c] = 0.0;
      }
  }
  if (!any) return;
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init(&bar[2], 1);
    mbar_init_fence();
  }
  __syncwarp();
  const int nload = 2 * nch - 1;
  auto issue = [&](int p) {  // load p, once its buffer's last store has been read
    if (lane == 0 && p < nload) {
      const int ch = p < nch ? p : 2 * nch - 2 - p;
      bulk_wait_read0();
      mbar_arrive_expect_tx(&bar[p % 3], CXT_BUF);
      tma_load_2d(bufs + (p % 3) * CXT_BUF, &tin, &bar[p % 3], xa + ch * CX_CH, r0);
    }
  };
  issue(0);
  issue(1);
  // this lane's parking place of chunk ch: park[ch*CX_CH]
  double *const park = cout + (long)(r0 + (lane >> 4)) * P + xa + (lane & 15);
  const long u = map.u(j, k);
  CnRun R;
  cn_load_run(tab, u, R);
  int lo_w = R.lo;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lo_w = max(lo_w, __shfl_xor_sync(0xffffffffu, lo_w, o));
  const double fCL = R.v[CN_CL], fCC = R.v[CN_CC], fCR = R.v[CN_CR], fFA = R.v[CN_FACT];
  const double fDU = R.v[CN_DU], fDP = R.v[CN_DP], fZH = R.v[CN_ZH];
  const double rz = fma(-fDP, fZH, 1.0), fZL = rz / fDP, fZLL = fma(-fDP, fZL, rz) / fDP;
  const bool hard = !div_rn_3_covers(fDP);
  auto co = [&](int f, int l) { return cn_coef(tab, u, R, f, l); };
  // this lane's row of a buffer: positions 2e, 2e+1 at pair(e), position e at cell(e)
  const int row_b = lane << 7, row_s = (lane & 7) << 4;
  auto pair = [&](unsigned char *b, int e) { return reinterpret_cast<double2 *>(b + row_b + ((e << 4) ^ row_s)); };
  auto cell = [&](unsigned char *b, int e) { return reinterpret_cast<double *>(pair(b, e >> 1)) + (e & 1); };

  // pass 1
  bool ok = true;
  double qm = 0.0, qc = 0.0, bp = 0.0;
  for (int ch = 0; ch < nch; ch++) {
    issue(ch + 2);
    ok = mbar_wait(&bar[ch % 3], (ch / 3) & 1);
    if (!ok || nch == 1) break;
    unsigned char *const b = bufs + (ch % 3) * CXT_BUF;
    const int l0 = ch * CX_CH - off;  // line row of position e: l0 + e; reading it finishes row l0 + e - 1
    if (l0 - 1 > lo_w && l0 + CX_CH - 2 <= ncells - 2 && ch + 1 < nch) {
      double q[CX_CH];
#pragma unroll
      for (int e = 0; e < CX_CH / 2; e++) {
        const double2 x = *pair(b, e);
        q[2 * e] = x.x;
        q[2 * e + 1] = x.y;
      }
#pragma unroll
      for (int e = 0; e < CX_CH; e++) {
        const double B = fCL * qm + fCC * qc + fCR * q[e];
        bp = B - fFA * bp;
        if (e == 1 && valid) park[ch * CX_CH] = bp;
        qm = qc;
        qc = q[e];
      }
    } else {
      const int cnt = min(np - ch * CX_CH, ch + 1 < nch ? CX_CH : 2);  // of the last chunk: its first row
#pragma unroll 2
      for (int e = 0; e < cnt; e++) {
        const int l = l0 + e;
        if (l < 0) continue;
        const double qv = *cell(b, e);
        if (l == 0) {
          qm = qv;  // BC_left_t0 = q(rmin)
        } else {
          const double B = co(CN_CL, l - 1) * qm + co(CN_CC, l - 1) * qc + co(CN_CR, l - 1) * qv;
          bp = B - co(CN_FACT, l - 1) * bp;
          if (e == 1 && valid && ch + 1 < nch) park[ch * CX_CH] = bp;
          qm = qc;
        }
        qc = qv;
      }
      if (ch + 1 == nch && cnt == 1) {  // the last row is a chunk's first; BC_right_t0 = q(rmax)
        const int l = ncells - 1;
        const double B = co(CN_CL, l) * qm + co(CN_CC, l) * qc + co(CN_CR, l) * qc;
        bp = B - co(CN_FACT, l) * bp;
      }
    }
    __syncwarp();
  }
  fence_proxy_async_all();  // the parked values land before any store of this row's chunks

  // pass 2
  double xn = 0.0, qn = 0.0;  // x and q of the row after the chunk
  double ahead = bp;          // B' of the next chunk's first cell
  for (int ch = nch - 1; ch >= 0 && ok; ch--) {
    const int p = 2 * nch - 2 - ch;
    double bq = ahead;
    ahead = (valid && ch > 1) ? park[(ch - 1) * CX_CH] : 0.0;
    if (ch != nch - 1) {
      ok = mbar_wait(&bar[p % 3], (p / 3) & 1);
      if (!ok) break;
    }
    unsigned char *const b = bufs + (p % 3) * CXT_BUF;
    const int l0 = ch * CX_CH - off;
    if (ch == 0) bq = 0.0;
    if (ch > 0 && l0 > lo_w && l0 + CX_CH - 1 <= ncells - 2) {
      double q[CX_CH + 1], y[CX_CH];
#pragma unroll
      for (int e = 0; e < CX_CH / 2; e++) {
        const double2 x = *pair(b, e);
        q[2 * e] = x.x;
        q[2 * e + 1] = x.y;
      }
      q[CX_CH] = qn;
      qn = q[0];
      y[0] = bq;
#pragma unroll
      for (int e = 1; e < CX_CH; e++) {
        const double B = fCL * q[e - 1] + fCC * q[e] + fCR * q[e + 1];
        y[e] = B - fFA * y[e - 1];
      }
      if (ch != nch - 1) issue(p + 2);  // the store of the chunk before has had the time to be read
      const double xs = xn;
      bool bad = hard;
#pragma unroll
      for (int e = CX_CH - 1; e >= 0; e--) {
        const double num = y[e] - fDU * xn;
        bad = bad || !div_rn_3_takes(num);
        xn = div_rn_3(num, fZH, fZL, fZLL);
        q[e] = xn;
      }
      if (bad) {
#pragma unroll
        for (int e = 0; e < CX_CH; e++) *cell(b, e) = y[e];
        xn = xs;
        for (int e = CX_CH - 1; e >= 0; e--) {
          double *T = cell(b, e);
          xn = ieee_div(*T - fDU * xn, fDP);
          *T = xn;
        }
      } else {
#pragma unroll
        for (int e = 0; e < CX_CH / 2; e++) *pair(b, e) = make_double2(q[2 * e], q[2 * e + 1]);
      }
    } else {
      const int cnt = min(np - ch * CX_CH, CX_CH);
      double pm = 0.0, first = 0.0;
      for (int e = 0; e < CX_CH; e++) {
        const int l = l0 + e;
        double *T = cell(b, e);
        if (l < 0 || e >= cnt) {  // outside the box
          *T = 0.0;
          continue;
        }
        const double qv = *T;
        const double qp = l + 1 < ncells ? (e + 1 < CX_CH ? *cell(b, e + 1) : qn) : qv;  // BC_right_t0 = q(rmax)
        if (e == 0) first = qv;
        if (l == 0) pm = qv;  // BC_left_t0 = q(rmin)
        if (e > 0 || ch == 0) {
          const double B = co(CN_CL, l) * pm + co(CN_CC, l) * qv + co(CN_CR, l) * qp;
          bq = B - co(CN_FACT, l) * bq;
        }
        *T = bq;
        pm = qv;
      }
      qn = first;
      if (ch != nch - 1) issue(p + 2);
#pragma unroll 2
      for (int e = cnt - 1; e >= 0; e--) {
        const int l = l0 + e;
        if (l < 0) break;
        double *T = cell(b, e);
        xn = div_rn_rcp(*T - co(CN_DU, l) * xn, co(CN_DP, l), co(CN_ZH, l));
        *T = xn;
      }
    }
    if (!active) {  // the reference leaves zeros
#pragma unroll
      for (int e = 0; e < CX_CH / 2; e++) *pair(b, e) = make_double2(0.0, 0.0);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (nval == 32) {
      if (lane == 0) {
        tma_store_2d(&tout, b, xa + ch * CX_CH, r0);
        bulk_commit();
      }
    } else {  // the rows past the run's end belong to others
      const int e = lane & 15, x = xa + ch * CX_CH + e;
#pragma unroll 1
      for (int row = lane >> 4; row < nval; row += 2) {
        if (x < L.nx)
          cout[(long)(r0 + row) * P + x] =
              *reinterpret_cast<const double *>(b + (row << 7) + ((((e >> 1) ^ (row & 7)) << 4) | ((e & 1) << 3)));
      }
      __syncwarp();
    }
  }
  if (lane == 0) {
    if (!ok) raise_error(sc, A3G_ERR_TIMEOUT, 5);
    bulk_wait0();
  }
}

// z lines.  A warp owns the 32 z lines of 32 consecutive i at one (j, grain):
// one tensor load brings the whole tile (32 i x nz levels, tile[k][lane]) into
// shared memory, each lane runs its line's elimination and back substitution
// in place, and one tensor store writes the tile back: the level is read once
// and written once.  The table rows of the tile's line (the same for its 32
// lines: the coefficients do not vary along i) come with the first tile that
// needs them by one bulk copy.  Warps are persistent and take contiguous runs
// of tiles (neighbouring i, then j), which share table rows.  Rows go in
// batches of four whose operands are read before the batch's first store, so
// that the reads do not wait on it.
// Bound by the recurrences' latency at the 11 lines per lane that 227 KB of
// shared memory hold for 60 levels.  480x401x50, 6 grains in a box: 148 -> 125
// us; 317x211x53, 7 grains: 133 -> 104 us a solve (44 warp instructions a cell
// against 60).
constexpr int ZT_U = 4;

// doubles of shared memory per warp: the tile and the staged table rows,
// rounded up to 128 bytes so that every warp's tile stays aligned
__host__ __device__ __forceinline__ long zt_warp_doubles(int nz) {
  return (32L * nz + CN_ROW * (long)nz + 15) / 16 * 16;
}

__global__ void __launch_bounds__(64, 8) k_cn_solve_zt(const __grid_constant__ CUtensorMap tin,
                                                    const __grid_constant__ CUtensorMap tout, Layout L,
                                                    Box box, Box cov, LineMap map, CnTab tab,
                                                    const int32_t *__restrict__ aloft, DevScalars *sc,
                                                    int wpb) {
  extern __shared__ __align__(128) unsigned char zt_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nz = L.nz;
  uint64_t *bar = reinterpret_cast<uint64_t *>(zt_smem) + wid;
  double *tile = reinterpret_cast<double *>(zt_smem + ZT_BAR_BYTES) + (long)wid * zt_warp_doubles(nz);
  double *stab = tile + 32L * nz;  // staged rows, CN_ROW doubles each
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_init_fence();
    prefetch_tensormap(&tin);
    prefetch_tensormap(&tout);
  }
  __syncwarp();
  const int it0 = (cov.imin - 1) >> 5, nti = ((cov.imax - 1) >> 5) - it0 + 1, nj = cov.jmax - cov.jmin + 1;
  const long ntiles = (long)nti * nj * L.ns;
  const long nwarps = (long)gridDim.x * wpb;
  const long per = ((unsigned)ntiles + (unsigned)nwarps - 1u) / (unsigned)nwarps;
  const long t0 = ((long)blockIdx.x * wpb + wid) * per;
  const long t1 = t0 + per < ntiles ? t0 + per : ntiles;
  const int rmin = box.kmin, rmax = box.kmax;
  const int ncells = rmax - rmin + 1;
  const uint32_t tile_bytes = 32u * (uint32_t)nz * 8u, tab_bytes = (uint32_t)ncells * CN_ROW * 8u;
  uint32_t phase = 0;
  int staged = -1;            // the line index u whose rows stab holds
  double *xx = tile + lane + (long)(rmin - 1) * 32;  // row l of this lane's line at xx[l*32]
  const double2 *const row2 = reinterpret_cast<const double2 *>(stab);  // FACT,CL  CC,CR  DU,ZH  ZL,ZLL
  for (long t = t0; t < t1; t++) {
    const unsigned r = (unsigned)t / (unsigned)nti, rg = r / (unsigned)nj;
    const int it = it0 + (int)((unsigned)t - r * (unsigned)nti);
    const int j = cov.jmin + (int)(r - rg * (unsigned)nj);
    const int g = (int)rg;
    const int i = (it << 5) + lane + 1;
    const bool act = i <= L.nx && i >= box.imin && i <= box.imax && j >= box.jmin && j <= box.jmax &&
                     aloft[g] != 0;
    const bool any = __any_sync(0xffffffffu, act);
    const int u = map.u(1, j);  // the coefficients do not vary along i (map.da == 0)
    // the previous tile's store must have read the buffer before it is refilled
    if (lane == 0) bulk_wait_read0();
    __syncwarp();
    if (any) {
      if (lane == 0) {
        mbar_arrive_expect_tx(bar, tile_bytes + (u != staged ? tab_bytes : 0u));
        tma_load_4d(tile, &tin, bar, it << 5, j - 1, 0, g);
        if (u != staged) bulk_load(stab, tab.p + (long)CN_ROW * u * ncells, tab_bytes, bar);
      }
      staged = u;
      if (!mbar_wait(bar, phase)) {
        if (lane == 0) {
          raise_error(sc, A3G_ERR_TIMEOUT, 2);
          bulk_wait0();
        }
        return;
      }
      phase ^= 1u;
      __syncwarp();
    }
    if (act) {
      double qm = xx[0], qc = qm, bp = 0.0;  // BC_left_t0 = q(rmin)
      int l = 0;
      for (; l + ZT_U < ncells; l += ZT_U) {
        double q[ZT_U];
        double2 a[ZT_U], b[ZT_U];
#pragma unroll
        for (int e = 0; e < ZT_U; e++) {
          q[e] = xx[(l + 1 + e) * 32];
          a[e] = row2[(l + e) * 4];
          b[e] = row2[(l + e) * 4 + 1];
        }
#pragma unroll
        for (int e = 0; e < ZT_U; e++) {
          const double B = a[e].y * qm + b[e].x * qc + b[e].y * q[e];
          bp = B - a[e].x * bp;
          xx[(l + e) * 32] = bp;
          qm = qc;
          qc = q[e];
        }
      }
      for (; l < ncells; l++) {
        const double qp = l + 1 < ncells ? xx[(l + 1) * 32] : qc;  // BC_right_t0 = q(rmax)
        const double2 a = row2[l * 4], b = row2[l * 4 + 1];
        const double B = a.y * qm + b.x * qc + b.y * qp;
        bp = B - a.x * bp;
        xx[l * 32] = bp;
        qm = qc;
        qc = qp;
      }
      // back substitution
      const bool hard = tab.runs()[2 * tab.U + u] != 0.0;
      double xn = 0.0;
      int top = ncells;  // rows below are to do
      for (; top >= ZT_U; top -= ZT_U) {
        double y[ZT_U], x[ZT_U];
        double2 a[ZT_U], b[ZT_U];
#pragma unroll
        for (int e = 0; e < ZT_U; e++) {
          y[e] = xx[(top - 1 - e) * 32];
          a[e] = row2[(top - 1 - e) * 4 + 2];
          b[e] = row2[(top - 1 - e) * 4 + 3];
        }
        const double xs = xn;
        bool bad = hard;
#pragma unroll
        for (int e = 0; e < ZT_U; e++) {
          const double num = y[e] - a[e].x * xn;
          bad = bad || !div_rn_3_takes(num);
          xn = div_rn_3(num, a[e].y, b[e].x, b[e].y);
          x[e] = xn;
        }
        if (bad) {
          xn = xs;
          for (int e = 0; e < ZT_U; e++) {
            const int m = top - 1 - e;
            xn = ieee_div(xx[m * 32] - row2[m * 4 + 2].x * xn, tab.at(CN_DP, m, u));
            xx[m * 32] = xn;
          }
        } else {
#pragma unroll
          for (int e = 0; e < ZT_U; e++) xx[(top - 1 - e) * 32] = x[e];
        }
      }
      for (int m = top - 1; m >= 0; m--) {
        const double2 a = row2[m * 4 + 2], b = row2[m * 4 + 3];
        const double num = xx[m * 32] - a.x * xn;
        xn = div_rn_3(num, a.y, b.x, b.y);
        if (hard || !div_rn_3_takes(num)) xn = ieee_div(num, tab.at(CN_DP, m, u));
        xx[m * 32] = xn;
      }
      for (int k = 1; k < rmin; k++) tile[(k - 1) * 32 + lane] = 0.0;  // outside the box
      for (int k = rmax + 1; k <= nz; k++) tile[(k - 1) * 32 + lane] = 0.0;
    } else {
      for (int k = 1; k <= nz; k++) tile[(k - 1) * 32 + lane] = 0.0;  // the reference leaves zeros
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_4d(&tout, tile, it << 5, j - 1, 0, g);
      bulk_commit();
    }
  }
  if (lane == 0) bulk_wait0();
}

// y lines.  A warp owns the 32 y lines of 32 consecutive i at one (k, grain)
// and walks them as the x solve walks its rows: chunks of YT_CH cells,
// tile[row][lane], with the chunk's table rows beside them (one bulk copy; the
// same for the warp's 32 lines), three buffers turning; pass 1 parks B' of
// every chunk's first row in the output line, pass 2 solves and stores chunk
// by chunk from the last (the last chunk's B' stays in a register, the others
// are read a chunk ahead).  Warps are persistent and take contiguous runs of
// line groups (neighbouring i, then k), which share table rows.
// Bound as the x solve; 720x360x60, 10 grains, ash in every cell: 0.99 -> 0.88
// ms, 93x131x37, 2 grains: 45 -> 29 us a solve.
constexpr int YT_BUF_D = YT_CH * 32 + YT_CH * CN_ROW;  // doubles of a buffer: the tile, the table rows

__global__ void __launch_bounds__(64, 8) k_cn_solve_yt(const __grid_constant__ CUtensorMap tin,
                                                    const __grid_constant__ CUtensorMap tout, Layout L,
                                                    Box box, Box cov, LineMap map, double *__restrict__ cout, CnTab tab,
                                                    const int32_t *__restrict__ aloft, DevScalars *sc,
                                                    int wpb) {
  extern __shared__ __align__(128) unsigned char yt_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t *bar = reinterpret_cast<uint64_t *>(yt_smem) + 3 * wid;
  double *const bufs = reinterpret_cast<double *>(yt_smem + ZT_BAR_BYTES) + (long)wid * 3 * YT_BUF_D;
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init(&bar[2], 1);
    mbar_init_fence();
    prefetch_tensormap(&tin);
    prefetch_tensormap(&tout);
  }
  __syncwarp();
  const int it0 = (cov.imin - 1) >> 5, nti = ((cov.imax - 1) >> 5) - it0 + 1, nk = cov.kmax - cov.kmin + 1;
  const long ngroups = (long)nti * nk * L.ns;
  const long nwarps = (long)gridDim.x * wpb;
  const long per = ((unsigned)ngroups + (unsigned)nwarps - 1u) / (unsigned)nwarps;
  const long t0 = ((long)blockIdx.x * wpb + wid) * per;
  const long t1 = t0 + per < ngroups ? t0 + per : ngroups;
  const int rmin = box.jmin, rmax = box.jmax;
  const int ncells = rmax - rmin + 1;
  const int nch = (ncells + YT_CH - 1) / YT_CH, nload = 2 * nch - 1;
  const int cnt_last = ncells - (nch - 1) * YT_CH;
  uint32_t s0 = 0;  // loads of the groups before: load p of this one is the warp's load s0 + p
  for (long t = t0; t < t1; t++) {
    const unsigned r = (unsigned)t / (unsigned)nti, rg = r / (unsigned)nk;
    const int it = it0 + (int)((unsigned)t - r * (unsigned)nti);
    const int k = cov.kmin + (int)(r - rg * (unsigned)nk);
    const int g = (int)rg;
    const int i = (it << 5) + lane + 1;
    const bool act = i <= L.nx && i >= box.imin && i <= box.imax && k >= box.kmin && k <= box.kmax &&
                     aloft[g] != 0;
    const bool any = __any_sync(0xffffffffu, act);
    double *xg = cout + (long)g * L.PG + (long)(k - 1) * L.PY + (i - 1);  // cell (i, 1, k) of this lane
    if (!any) {  // the reference leaves zeros
      if (i <= L.nx)
        for (int j = cov.jmin; j <= cov.jmax; j++) xg[(long)(j - 1) * L.P] = 0.0;
      continue;
    }
    if (i <= L.nx) {  // cells that no chunk store covers: outside [rmin, rmin + nch*YT_CH)
      for (int j = cov.jmin; j < rmin; j++) xg[(long)(j - 1) * L.P] = 0.0;
      for (int j = rmin + nch * YT_CH; j <= cov.jmax; j++) xg[(long)(j - 1) * L.P] = 0.0;
    }
    xg += (long)(rmin - 1) * L.P;  // row 0
    const long u = map.u(1, k);    // the coefficients do not vary along i (map.da == 0)
    auto buf = [&](int p) { return bufs + ((s0 + (uint32_t)p) % 3u) * YT_BUF_D; };
    auto issue = [&](int p) {  // load p, once its buffer's last store has been read
      if (lane == 0 && p < nload) {
        const int ch = p < nch ? p : 2 * nch - 2 - p;
        const uint32_t tb = (uint32_t)(ch + 1 < nch ? YT_CH : cnt_last) * CN_ROW * 8u;
        uint64_t *b = &bar[(s0 + (uint32_t)p) % 3u];
        bulk_wait_read0();
        mbar_arrive_expect_tx(b, YT_CH * 32u * 8u + tb);
        tma_load_4d(buf(p), &tin, b, it << 5, rmin - 1 + ch * YT_CH, k - 1, g);
        bulk_load(buf(p) + YT_CH * 32, tab.p + CN_ROW * (u * ncells + (long)ch * YT_CH), tb, b);
      }
    };
    auto wait = [&](int p) {
      const uint32_t s = s0 + (uint32_t)p;
      return mbar_wait(&bar[s % 3u], (s / 3u) & 1u);
    };
    issue(0);
    issue(1);
    // pass 1: forward elimination, B' of the chunks' first rows only
    bool ok = true;
    double qm = 0.0, qc = 0.0, bp = 0.0;
    double2 ca = make_double2(0.0, 0.0), cb = ca;  // FACT,CL and CC,CR of the chunk before's last row
    for (int ch = 0; ch < nch; ch++) {
      issue(ch + 2);
      ok = wait(ch);
      if (!ok || nch == 1) break;
      const double *T = buf(ch) + lane;
      const double2 *row2 = reinterpret_cast<const double2 *>(buf(ch) + YT_CH * 32);
      auto row = [&](double2 a, double2 b, double qp) {  // the next row of the elimination
        const double B = a.y * qm + b.x * qc + b.y * qp;
        bp = B - a.x * bp;
        qm = qc;
        qc = qp;
      };
      if (ch == 0) {
        qm = T[0];  // BC_left_t0 = q(rmin)
        qc = qm;
      } else {
        row(ca, cb, T[0]);
      }
      if (ch + 1 < nch) {
        double q[YT_CH];
#pragma unroll
        for (int e = 1; e < YT_CH; e++) q[e] = T[e * 32];
#pragma unroll
        for (int e = 1; e < YT_CH; e++) {
          row(row2[(e - 1) * 4], row2[(e - 1) * 4 + 1], q[e]);
          if (e == 1 && act) xg[(long)(ch * YT_CH) * L.P] = bp;
        }
        ca = row2[(YT_CH - 1) * 4];
        cb = row2[(YT_CH - 1) * 4 + 1];
      } else {  // of the last chunk: its first row; BC_right_t0 = q(rmax)
        row(row2[0], row2[1], cnt_last > 1 ? T[32] : qc);
      }
      __syncwarp();
    }
    fence_proxy_async_all();  // the parked values land before any store of this line's chunks
    // pass 2
    const bool hard = tab.runs()[2 * tab.U + u] != 0.0;
    double xn = 0.0, qn = 0.0;  // x and q of the row after the chunk
    double ahead = bp;          // B' of the next chunk's first row
    for (int ch = nch - 1; ch >= 0 && ok; ch--) {
      const int p = 2 * nch - 2 - ch;
      double b0 = ahead;
      ahead = (act && ch > 1) ? xg[(long)((ch - 1) * YT_CH) * L.P] : 0.0;
      if (ch != nch - 1) {
        ok = wait(p);
        if (!ok) break;
      }
      double *T = buf(p) + lane;
      const double2 *row2 = reinterpret_cast<const double2 *>(buf(p) + YT_CH * 32);
      const int cnt = ch + 1 < nch ? YT_CH : cnt_last;
      const double q0 = T[0];
      if (ch == 0) {
        const double q1 = ncells > 1 ? T[32] : q0;
        b0 = row2[0].y * q0 + row2[1].x * q0 + row2[1].y * q1;  // FACT = 0
      }
      if (cnt == YT_CH) {  // lanes outside the box run along: their tile is cleared below
        double q[YT_CH + 1], y[YT_CH];
#pragma unroll
        for (int e = 0; e < YT_CH; e++) q[e] = T[e * 32];
        q[YT_CH] = ch + 1 < nch ? qn : q[YT_CH - 1];  // BC_right_t0 = q(rmax)
        y[0] = b0;
#pragma unroll
        for (int e = 1; e < YT_CH; e++) {
          const double2 a = row2[e * 4], b = row2[e * 4 + 1];
          const double B = a.y * q[e - 1] + b.x * q[e] + b.y * q[e + 1];
          y[e] = B - a.x * y[e - 1];
        }
        if (ch != nch - 1) issue(p + 2);  // the store of the chunk before has had the time to be read
        const double xs = xn;
        bool bad = hard;
#pragma unroll
        for (int e = YT_CH - 1; e >= 0; e--) {
          const double2 a = row2[e * 4 + 2], b = row2[e * 4 + 3];
          const double num = y[e] - a.x * xn;
          bad = bad || !div_rn_3_takes(num);
          xn = div_rn_3(num, a.y, b.x, b.y);
          T[e * 32] = xn;
        }
        if (bad && act) {
#pragma unroll
          for (int e = 0; e < YT_CH; e++) T[e * 32] = y[e];
          xn = xs;
          for (int e = YT_CH - 1; e >= 0; e--) {
            xn = ieee_div(T[e * 32] - row2[e * 4 + 2].x * xn, tab.at(CN_DP, ch * YT_CH + e, u));
            T[e * 32] = xn;
          }
        }
      } else if (act) {
        double pm = q0, bq = b0;
        T[0] = b0;
#pragma unroll 2
        for (int e = 1; e < cnt; e++) {
          const double qv = T[e * 32], qp = e + 1 < cnt ? T[(e + 1) * 32] : qv;  // BC_right_t0 = q(rmax)
          const double2 a = row2[e * 4], b = row2[e * 4 + 1];
          const double B = a.y * pm + b.x * qv + b.y * qp;
          bq = B - a.x * bq;
          T[e * 32] = bq;
          pm = qv;
        }
#pragma unroll 2
        for (int e = cnt - 1; e >= 0; e--) {
          const double2 a = row2[e * 4 + 2], b = row2[e * 4 + 3];
          const double num = T[e * 32] - a.x * xn;
          xn = div_rn_3(num, a.y, b.x, b.y);
          if (hard || !div_rn_3_takes(num)) xn = ieee_div(num, tab.at(CN_DP, ch * YT_CH + e, u));
          T[e * 32] = xn;
        }
        for (int e = cnt; e < YT_CH; e++) T[e * 32] = 0.0;  // beyond rmax
      }
      qn = q0;
      if (!act) {
        for (int e = 0; e < YT_CH; e++) T[e * 32] = 0.0;  // the reference leaves zeros
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_4d(&tout, buf(p), it << 5, rmin - 1 + ch * YT_CH, k - 1, g);
        bulk_commit();
      }
    }
    if (!ok) {
      if (lane == 0) {
        raise_error(sc, A3G_ERR_TIMEOUT, 1);
        bulk_wait0();
      }
      return;
    }
    s0 += (uint32_t)nload;
  }
  if (lane == 0) bulk_wait0();
}

// ---------------------------------------------------------------------------
// TMA tensor maps over the concentration levels
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

// Looked up once per process; the initialisation of a function-local static
// is thread-safe, and contexts may make their first launches from several
// host threads at once (concurrent ensemble members).
static EncodeTiledFn encode_tiled_fn() {
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeTiledFn>(p);
    cudaGetLastError();
    return nullptr;
  }();
  return fn;
}

// A level as a 4-D tensor (i, j, k, grain) of doubles with the device
// layout's pitches (a wind array: the same with one grain); the box is one
// tile of the given kind (TmapKind).
bool tensor_map(a3g_ctx *ctx, const double *p, int kind, CUtensorMap *out) {
  for (const TmapEntry &e : ctx->tmaps)
    if (e.p == p && e.kind == kind) {
      *out = e.map;
      return true;
    }
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return false;
  const Layout &L = ctx->L;
  const bool wind = kind == TM_ADV_VY || kind == TM_ADV_VZ || kind == TM_ADV_VX;
  const cuuint64_t dims[4] = {(cuuint64_t)L.nx, (cuuint64_t)L.ny, (cuuint64_t)L.nz,
                              (cuuint64_t)(wind ? 1 : L.ns)};
  const cuuint64_t strides[3] = {(cuuint64_t)L.P * 8, (cuuint64_t)L.PY * 8, (cuuint64_t)L.PG * 8};
  cuuint32_t box[4] = {32, 1, 1, 1};
  cuuint32_t rank = 4;
  // the rows of a level form a 2-D array: row r = (g*nz + k-1)*ny + j-1 at r*P
  const cuuint64_t rdims[2] = {(cuuint64_t)L.nx, (cuuint64_t)L.ny * L.nz * (kind == TM_VROWS ? 1 : L.ns)};
  CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_NONE;
  if (kind == TM_XROWS) {
    rank = 2;
    box[0] = CX_CH;
    box[1] = 32;
    swizzle = CU_TENSOR_MAP_SWIZZLE_128B;
  } else if (kind == TM_QROWS || kind == TM_VROWS) {
    rank = 2;
    box[0] = 8;
    box[1] = 32;
    swizzle = CU_TENSOR_MAP_SWIZZLE_64B;
  } else if (kind == TM_COLUMN) {
    if (L.nz > 256) return false;
    box[2] = (cuuint32_t)L.nz;
  } else if (kind == TM_YCHUNK) {
    box[1] = YT_CH;
  } else if (kind == TM_ADV_QY || kind == TM_ADV_VY) {
    box[1] = ACH;

  } else if (kind == TM_ADV_QZ || kind == TM_ADV_VZ) {
    box[2] = ACH;
  } else if (kind == TM_ADV_QX1 || kind == TM_ADV_VX) {
  } else if (kind == TM_ADV_QX2) {
    if (L.ns < 2) return false;
    box[3] = 2;
  } else {
    return false;
  }
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  TmapEntry e;
  e.p = p;
  e.kind = kind;
  if (enc(&e.map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, rank, const_cast<double *>(p), rank == 2 ? rdims : dims,
          strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  // a step uses about 17 (two levels alternating under each tile shape, and
  // the wind arrays); the adjoint's stage levels add more
  if (ctx->tmaps.size() >= 64) ctx->tmaps.erase(ctx->tmaps.begin());
  ctx->tmaps.push_back(e);
  *out = e.map;
  return true;
}

// Opts a tiled kernel in to the largest dynamic shared memory; `per_sm`: its
// resident blocks per SM.
template <typename K>
static bool tile_kernel_setup(a3g_ctx *ctx, K kernel, int threads, size_t smem, int *per_sm, int *nsm) {
  int optin = 0;
  // the opt-in maximum, so that contexts of any extent can share the attribute
  return cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) == cudaSuccess &&
         (size_t)optin >= smem &&
         cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) == cudaSuccess &&
         cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                              cudaSharedmemCarveoutMaxShared) == cudaSuccess &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, threads, smem) == cudaSuccess &&
         cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, ctx->device) == cudaSuccess && *per_sm >= 1;
}

// Launches the z solve through column tiles; false when the shape is outside
// what the tiles cover (the caller takes the per-thread kernel).
static bool launch_cn_solve_zt(a3g_ctx *ctx, const LineMap &map, const CnTab &tab) {
  const Layout &L = ctx->L;
  if (L.nz > 256 || map.da) return false;
  CUtensorMap tin, tout;
  if (!tensor_map(ctx, ctx->c0, TM_COLUMN, &tin) || !tensor_map(ctx, ctx->c1, TM_COLUMN, &tout)) return false;
  const int wpb = L.nz <= 128 ? 2 : 1;
  const size_t smem = ZT_BAR_BYTES + (size_t)wpb * zt_warp_doubles(L.nz) * sizeof(double);
  if (ctx->tma_grid[0] == 0) {
    int per_sm = 0, nsm = 0;
    if (!tile_kernel_setup(ctx, k_cn_solve_zt, 32 * wpb, smem, &per_sm, &nsm)) return false;
    ctx->tma_grid[0] = per_sm * nsm;
  }
  const Box cov = cover_box(ctx);
  const long ntiles = (long)((cov.imax - 1) / 32 - (cov.imin - 1) / 32 + 1) * (cov.jmax - cov.jmin + 1) * L.ns;
  const long need = (ntiles + wpb - 1) / wpb;
  const int grid = (int)(need < ctx->tma_grid[0] ? need : ctx->tma_grid[0]);
  k_cn_solve_zt<<<grid, 32 * wpb, smem, ctx->stream>>>(tin, tout, L, ctx->box, cov, map, tab, ctx->aloft, ctx->sc,
                                                       wpb);
  return true;
}

// Launches the y solve through chunk tiles; false when the maps cannot be
// made (the caller takes the per-thread kernel).
static bool launch_cn_solve_yt(a3g_ctx *ctx, const LineMap &map, const CnTab &tab) {
  const Layout &L = ctx->L;
  if (map.da) return false;
  CUtensorMap tin, tout;
  if (!tensor_map(ctx, ctx->c0, TM_YCHUNK, &tin) || !tensor_map(ctx, ctx->c1, TM_YCHUNK, &tout)) return false;
  const int wpb = 2;
  const size_t smem = ZT_BAR_BYTES + (size_t)wpb * 3 * YT_BUF_D * sizeof(double);
  if (ctx->tma_grid[1] == 0) {
    int per_sm = 0, nsm = 0;
    if (!tile_kernel_setup(ctx, k_cn_solve_yt, 32 * wpb, smem, &per_sm, &nsm)) return false;
    ctx->tma_grid[1] = per_sm * nsm;
  }
  const Box cov = cover_box(ctx);
  const long ngroups = (long)((cov.imax - 1) / 32 - (cov.imin - 1) / 32 + 1) * (cov.kmax - cov.kmin + 1) * L.ns;
  const long need = (ngroups + wpb - 1) / wpb;
  const int grid = (int)(need < ctx->tma_grid[1] ? need : ctx->tma_grid[1]);
  k_cn_solve_yt<<<grid, 32 * wpb, smem, ctx->stream>>>(tin, tout, L, ctx->box, cov, map, ctx->c1, tab, ctx->aloft,
                                                       ctx->sc, wpb);
  return true;
}

// Launches the x solve through TMA tiles; false when the maps cannot be made.
static bool launch_cn_solve_xt2(a3g_ctx *ctx, const LineMap &map, const CnTab &tab) {
  const Layout &L = ctx->L;
  CUtensorMap tin, tout;
  if (!tensor_map(ctx, ctx->c0, TM_XROWS, &tin) || !tensor_map(ctx, ctx->c1, TM_XROWS, &tout)) return false;
  if (ctx->tma_grid[2] == 0) {
    int per_sm = 0, nsm = 0;
    if (!tile_kernel_setup(ctx, k_cn_solve_xt2, 32 * CXT_WARPS, CXT_SMEM, &per_sm, &nsm)) return false;
    ctx->tma_grid[2] = per_sm * nsm;
  }
  const RowCover cov = row_cover(L, cover_box(ctx));
  const long nwarps = (long)cov.ntile * L.ns;
  k_cn_solve_xt2<<<(unsigned)((nwarps + CXT_WARPS - 1) / CXT_WARPS), 32 * CXT_WARPS, CXT_SMEM, ctx->stream>>>(
      tin, tout, L, ctx->box, cov, map, ctx->c1, tab, ctx->aloft, ctx->sc);
  return true;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// Brings the explicit sweeps' table up to date; false where something varies
// along i and k_diff / k_adj_diff have to run.
static bool diff_table(a3g_ctx *ctx) {
  if (ctx->snx.si || ctx->sny.si || ctx->snz.si || ctx->kappa.si || ctx->kx.si || ctx->ky.si || ctx->kz.si) return false;
  const Layout &L = ctx->L;
  const int n = (L.ny + 1) * (L.nz + 1);
  if (!ctx->diff_tab) {
    if (cudaMalloc((void **)&ctx->diff_tab, sizeof(DiffRow) * (size_t)n) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    ctx->bytes += sizeof(DiffRow) * (size_t)n;
  }
  if (!ctx->diff_valid) {
    k_diff_table<<<(n + 127) / 128, 128, 0, ctx->stream>>>(L, ctx->snx, ctx->sny, ctx->snz, ctx->kappa, ctx->kx,
                                                         ctx->ky, ctx->kz, static_cast<DiffRow *>(ctx->diff_tab));
    ctx->launches++;
    ctx->diff_valid = cudaPeekAtLastError() == cudaSuccess;  // the caller's check reports a refused launch
  }
  return ctx->diff_valid;
}

// segments of a marched line of n cells that leave at least 8 cells each and
// give the chip about `per_sm` warps an SM: 24 for the fused horizontal sweeps
// (48 warps: 360x161x40, 5 grains, 50 -> 60 us), 128 for the vertical one, whose
// whole columns wait on each load in turn (24 warps: 317x211x53, 3 grains, 72 us
// and 82 for the transpose, where a thread a cell took 72 and 75; 51 and 57 with
// 128; 317x211x53, 7 grains, 120 and 136 against 135 and 134; 101 and 113).
static int diff_segments(int n, long warps, long per_sm) {
  const long want = (148L * per_sm + warps - 1) / warps, most = n / 8 > 1 ? n / 8 : 1;
  return (int)(want < 1 ? 1 : want < most ? want : most);
}

// The horizontal sweeps in one pass, x first or y first; diff_table holds.
template <bool ADJ>
static void run_diff_xy(a3g_ctx *ctx, bool xfirst, const Box &box, const Box &cov, const double *cin, double *cout) {
  const Layout &L = ctx->L;
  const int n = cov.jmax - cov.jmin + 1;
  const long lines = (long)((cov.imax - cov.imin + 30) / 30) * (cov.kmax - cov.kmin + 1) * L.ns;
  const int want = diff_segments(n, lines, 24), seg = (n + want - 1) / want;
  const int nseg = (n + seg - 1) / seg;
  const unsigned blocks = (unsigned)((lines * nseg + 3) / 4);
  const DiffRow *tab = static_cast<const DiffRow *>(ctx->diff_tab);
#define A3G_DXY(X_, P_) \
  k_diff_xy<X_, ADJ, P_><<<blocks, 128, 0, ctx->stream>>>(L, box, cov, nseg, seg, cin, cout, tab, ctx->aloft, ctx->sc)
  if (ctx->grid.periodic) {
    if (xfirst) A3G_DXY(true, true); else A3G_DXY(false, true);
  } else {
    if (xfirst) A3G_DXY(true, false); else A3G_DXY(false, false);
  }
#undef A3G_DXY
}

// A march needs columns enough: on small grids a thread a cell (k_diff,
// k_adj_diff) is sooner done (50x50x23, 1 grain: 5.1 us, the march 8.2, its
// transpose 4.7, 8.2; 60x80x30, 2 grains: 6.2, 6.5 and 6.2, 7.9; but 100x100x40,
// 1 grain: 10.3, 6.2 and 10.3, 7.8).
template <bool ADJ>
static bool run_diff_z(a3g_ctx *ctx, const Box &box, const Box &cov, const double *cin, double *cout) {
  const Layout &L = ctx->L;
  if ((long)L.nx * L.ny * L.nz < 250000 || !diff_table(ctx)) return false;
  const int n = cov.kmax - cov.kmin + 1;
  const long lines = (long)((cov.imax - cov.imin + 32) / 32) * (cov.jmax - cov.jmin + 1) * L.ns;
  const int want = diff_segments(n, lines, 128), seg = (n + want - 1) / want;
  const int nseg = (n + seg - 1) / seg;
  k_diff_z<ADJ><<<(unsigned)((lines * nseg + 3) / 4), 128, 0, ctx->stream>>>(
      L, box, cov, nseg, seg, cin, cout, static_cast<const DiffRow *>(ctx->diff_tab), ctx->aloft, ctx->sc);
  return true;
}

template <int DIR>
static int launch_diff_dir(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  tbegin(ctx, A3G_K_DIFF_X + DIR);
  if (DIR == 2 && run_diff_z<false>(ctx, ctx->box, cover_box(ctx), ctx->c0, ctx->c1)) {
    // marched
  } else {
    const Geo3 &sig = (DIR == 0) ? ctx->snx : (DIR == 1) ? ctx->sny : ctx->snz;
    const Geo3 &kk = (DIR == 0) ? ctx->kx : (DIR == 1) ? ctx->ky : ctx->kz;
    dim3 grid((L.nx + 31) / 32, (L.ny + 7) / 8, L.nz);
    k_diff<DIR><<<grid, dim3(32, 8), 0, ctx->stream>>>(L, ctx->box, ctx->grid.periodic, ctx->c0,
                                                       ctx->c1, sig, ctx->kappa, kk, ctx->aloft,
                                                       ctx->sc);
  }
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  sweep_done(ctx);
  return A3G_OK;
}

// DiffuseHorz, explicit: both sweeps, x first or y first.  One timed launch
// (A3G_K_DIFF_X) where they are fused, one each where they are not.
int launch_diff_horz(a3g_ctx *ctx, bool xfirst) {
  if (!diff_table(ctx)) {
    int rc = xfirst ? launch_diff_dir<0>(ctx) : launch_diff_dir<1>(ctx);
    if (!rc) rc = xfirst ? launch_diff_dir<1>(ctx) : launch_diff_dir<0>(ctx);
    return rc;
  }
  tbegin(ctx, A3G_K_DIFF_X);
  run_diff_xy<false>(ctx, xfirst, ctx->box, cover_box(ctx), ctx->c0, ctx->c1);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  sweep_done(ctx);
  return A3G_OK;
}

int launch_diff_z(a3g_ctx *ctx) { return launch_diff_dir<2>(ctx); }

static inline bool varies(const Geo3 &g, int idx) {  // idx 0:i 1:j 2:k
  return (idx == 0 ? g.si : idx == 1 ? g.sj : g.sk) != 0;
}

template <int DIR>
static LineMap line_map(const a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  const Geo3 &sig = (DIR == 0) ? ctx->snx : (DIR == 1) ? ctx->sny : ctx->snz;
  const Geo3 &kk = (DIR == 0) ? ctx->kx : (DIR == 1) ? ctx->ky : ctx->kz;
  const int ia = (DIR == 0) ? 1 : 0, ib = (DIR == 2) ? 1 : 2;
  auto any = [&](int i) { return varies(ctx->kappa, i) || varies(sig, i) || varies(kk, i); };
  LineMap map;
  map.na = (DIR == 0) ? L.ny : L.nx;
  map.nb = (DIR == 2) ? L.ny : L.nz;
  map.da = any(ia);
  map.db = any(ib);
  map.ds = any(DIR);
  map.U = (map.da ? map.na : 1) * (map.db ? map.nb : 1);
  return map;
}

// the y and z tables are stored by row unless their lines differ along i
static bool cn_byrow(int dir, const LineMap &map) { return dir != 0 && !map.da; }

size_t cn_table_doubles(const a3g_ctx *ctx, int dir) {
  const LineMap map = dir == 0 ? line_map<0>(ctx) : dir == 1 ? line_map<1>(ctx) : line_map<2>(ctx);
  const size_t n = (dir == 0) ? ctx->L.nx : (dir == 1) ? ctx->L.ny : ctx->L.nz;
  return ((cn_byrow(dir, map) ? CN_NF : CN_NFX) * n + 3) * (size_t)map.U;
}

static inline bool same_box(const Box &a, const Box &b) {
  return a.imin == b.imin && a.imax == b.imax && a.jmin == b.jmin && a.jmax == b.jmax && a.kmin == b.kmin &&
         a.kmax == b.kmax;
}

static inline int box_cells(const Box &b, int dir) {
  return dir == 0 ? b.imax - b.imin + 1 : dir == 1 ? b.jmax - b.jmin + 1 : b.kmax - b.kmin + 1;
}

// What direction DIR needs of the next k_cn_tables; no blocks where the host
// knows that nothing has changed since the last build.
template <int DIR>
static CnTableJob cn_table_job(a3g_ctx *ctx) {
  CnTableJob j{};
  const bool may = ctx->cn_valid[DIR] && same_box(ctx->cn_box[DIR], ctx->box);
  if (!ctx->cn_tab[DIR] || box_cells(ctx->box, DIR) <= 1 || (may && ctx->cn_stamp[DIR] == ctx->dt_stamp)) return j;
  double *const st = ctx->cn_state + 2 * DIR;
  j.map = line_map<DIR>(ctx);
  j.sig = (DIR == 0) ? ctx->snx : (DIR == 1) ? ctx->sny : ctx->snz;
  j.kk = (DIR == 0) ? ctx->kx : (DIR == 1) ? ctx->ky : ctx->kz;
  j.st_old = st + ctx->cn_slot[DIR];
  j.st_new = st + (ctx->cn_slot[DIR] ^ 1);
  j.tab = ctx->cn_tab[DIR];
  j.may = may ? 1 : 0;
  j.byrow = cn_byrow(DIR, j.map) ? 1 : 0;
  // many lines: 32 share a block's serial warp; few: a block each, more of its rows at once (the three
  // tables of 20, 20 and 400 lines 16 us a block each, 19 with 32; of 624, 672 and 728 lines 50 and 25;
  // of 1224, 1360 and 1440 lines 102 and 30)
  j.lpb = j.map.U >= 512 ? 32 : 1;
  j.blocks = (j.map.U + j.lpb - 1) / j.lpb;
  return j;
}

// The factor table of direction DIR for the step's dt: built by k_cn_tables,
// or kept from the previous build when nothing it depends on has changed.
// No launch at all while the host knows that dt has not been set since.  A
// build takes the other directions' stale tables along: each is one serial
// chain per line, and the three run side by side (a step's tables on
// 93x131x37: 38 us in three launches, 26 in one; 317x211x53: 35, 26;
// 201x151x41 over terrain: 176, 96).
// `timed`: the launch has a bracket of its own (the caller has none open).
template <int DIR>
static int cn_table(a3g_ctx *ctx, const LineMap &map, bool timed, CnTab *out) {
  const Box &box = ctx->box;
  const int n = box_cells(box, DIR);
  *out = CnTab{ctx->cn_tab[DIR], (long)n * map.U, map.U, n, cn_byrow(DIR, map)};
  if (ctx->cn_valid[DIR] && same_box(ctx->cn_box[DIR], box) && ctx->cn_stamp[DIR] == ctx->dt_stamp) return A3G_OK;
  const CnTableJob jx = cn_table_job<0>(ctx), jy = cn_table_job<1>(ctx), jz = cn_table_job<2>(ctx);
  const bool wide = jx.lpb > 1 || jy.lpb > 1 || jz.lpb > 1;
  if (timed) tbegin(ctx, A3G_K_CN_TABLE);
  k_cn_tables<<<jx.blocks + jy.blocks + jz.blocks, 256, 5 * (wide ? 1024 : 256) * sizeof(double), ctx->stream>>>(
      ctx->L, box, ctx->prm.imp_fac, ctx->kappa, jx, jy, jz, ctx->sc);
  if (timed) tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  const int built[3] = {jx.blocks, jy.blocks, jz.blocks};
  for (int d = 0; d < 3; d++)
    if (built[d]) {
      ctx->cn_slot[d] ^= 1;
      ctx->cn_stamp[d] = ctx->dt_stamp;
      ctx->cn_valid[d] = true;
      ctx->cn_box[d] = box;
    }
  return A3G_OK;
}

template <int DIR>
static int launch_cn_dir(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  const Box &box = ctx->box;
  const int rmin = (DIR == 0) ? box.imin : (DIR == 1) ? box.jmin : box.kmin;
  const int rmax = (DIR == 0) ? box.imax : (DIR == 1) ? box.jmax : box.kmax;
  if (rmax - rmin + 1 <= 1) {
    // :770 skips the solve and the copy-back; ts1 stays zero.
    ctx->ts1_zeroed = true;
    return A3G_OK;
  }
  const LineMap map = line_map<DIR>(ctx);
  CnTab tab;
  int rc = cn_table<DIR>(ctx, map, true, &tab);
  if (rc) return rc;
  const long nlines = (long)map.na * map.nb * L.ns;
  tbegin(ctx, A3G_K_CN_SOLVE_X + DIR);
  if (DIR == 0 && ctx->tune_cn_x == 2 && map.ds) {
    int threads;
    const dim3 grid = rt_grid(L, &threads);
    k_cn_solve_xv<<<grid, threads, 0, ctx->stream>>>(L, box, map, ctx->c0, ctx->c1, tab, ctx->aloft);
  } else if (DIR == 0 && ctx->tune_cn_x == 2 && launch_cn_solve_xt2(ctx, map, tab)) {
    // tiles through TMA
  } else if (DIR == 0 && ctx->tune_cn_x == 0) {
    const long nwarps = (nlines + 31) / 32;
    k_cn_solve_xt<<<(unsigned)((nwarps + XT_WARPS - 1) / XT_WARPS), 32 * XT_WARPS, 0, ctx->stream>>>(
        L, box, map, ctx->c0, ctx->c1, tab, ctx->aloft);
  } else if (DIR == 2 && ctx->tune_cn_yz == 3 && launch_cn_solve_zt(ctx, map, tab)) {
    // column tiles through TMA
  } else if (DIR == 1 && ctx->tune_cn_yz == 3 && launch_cn_solve_yt(ctx, map, tab)) {
    // chunk tiles through TMA
  } else if (DIR != 0 && ctx->tune_cn_yz == 3) {
    constexpr int D = DIR == 0 ? 1 : DIR;
    int threads;
    const dim3 grid = cb_grid<D>(L, &threads);
    if (tab.byrow) k_cn_solve_b<D, true><<<grid, threads, 0, ctx->stream>>>(L, box, map, ctx->c0, ctx->c1, tab, ctx->aloft);
    else k_cn_solve_b<D, false><<<grid, threads, 0, ctx->stream>>>(L, box, map, ctx->c0, ctx->c1, tab, ctx->aloft);
  } else if (DIR != 0 && ctx->tune_cn_yz == 1 && L.ns >= 2) {
    launch_cn_solve_gc<DIR == 0 ? 1 : DIR, 2>(ctx, map, tab);
  } else if (DIR != 0 && ctx->tune_cn_yz == 2 && L.ns >= 2) {
    launch_cn_solve_gc<DIR == 0 ? 1 : DIR, 4>(ctx, map, tab);
  } else {
    k_cn_solve<DIR><<<(unsigned)((nlines + 127) / 128), 128, 0, ctx->stream>>>(
        L, box, map, ctx->c0, ctx->c1, tab, ctx->aloft);
  }
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  sweep_done(ctx);
  ctx->ts1_zeroed = false;
  return A3G_OK;
}

int launch_diffcn_x(a3g_ctx *ctx) { return launch_cn_dir<0>(ctx); }
int launch_diffcn_y(a3g_ctx *ctx) { return launch_cn_dir<1>(ctx); }
int launch_diffcn_z(a3g_ctx *ctx) { return launch_cn_dir<2>(ctx); }

// ===========================================================================
// Discrete adjoint of the diffusion sweeps (no counterpart in the reference).
// Both sweeps are linear; full box only.
// ===========================================================================
// Explicit: out(l) = q(l) + cR(l)(q(l+1)-q(l)) - cL(l)(q(l)-q(l-1)) with the
// Neumann ghosts (periodic in x); the transpose gathers, per cell m,
//   lam_q(m) = lam(m)(1 - cR(m) - cL(m)) + cR(m-1)lam(m-1) + cL(m+1)lam(m+1)
// and folds the ghost terms back: cL(1)lam(1) into cell 1 and cR(n)lam(n)
// into cell n (Neumann), or into cells n and 1 (periodic).
template <int DIR>
__global__ void __launch_bounds__(256) k_adj_diff(Layout L, int periodic, const double *__restrict__ lin,
                                                  double *__restrict__ lout, Geo3 sig, Geo3 kap, Geo3 kk,
                                                  const int32_t *__restrict__ aloft,
                                                  const DevScalars *__restrict__ sc) {
  const int i = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > L.nx || j > L.ny) return;
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  const int l = (DIR == 0) ? i : (DIR == 1) ? j : k;
  const long st = (DIR == 0) ? 1 : (DIR == 1) ? L.P : L.PY;
  const long cell = L.cell(i, j, k);
  auto G = [&](const Geo3 &a, int m) {
    return (DIR == 0) ? a.at(m, j, k) : (DIR == 1) ? a.at(i, m, k) : a.at(i, j, m);
  };
  const double dt = sc->dt;
  auto cR = [&](int m) {
    const double dsR = 2.0 * G(sig, m + 1) / (G(kap, m) + G(kap, m + 1));
    return dt * (0.5 * (G(kk, m) + G(kk, m + 1)) * dsR) * (G(sig, m + 1) / G(kap, m));
  };
  auto cL = [&](int m) {
    const double dsL = 2.0 * G(sig, m) / (G(kap, m - 1) + G(kap, m));
    return dt * (0.5 * (G(kk, m - 1) + G(kk, m)) * dsL) * (G(sig, m) / G(kap, m));
  };
  const bool per = DIR == 0 && periodic;
  const double cRl = cR(l), cLl = cL(l);
  const double cRm = (l > 1) ? cR(l - 1) : 0.0, cLp = (l < n) ? cL(l + 1) : 0.0;
  const double cRn = (l == 1 && per) ? cR(n) : 0.0, cL1 = (l == n && per) ? cL(1) : 0.0;
  for (int g = 0; g < L.ns; g++) {
    const long a = (long)g * L.PG + cell;
    if (!aloft[g]) { lout[a] = 0.0; continue; }
    const double lm = lin[a];
    double v = lm - cRl * lm - cLl * lm;
    if (l > 1) v = v + cRm * lin[a - st];
    if (l < n) v = v + cLp * lin[a + st];
    if (!per) {
      if (l == 1) v = v + cLl * lm;
      if (l == n) v = v + cRl * lm;
    } else {
      if (l == 1) v = v + cRn * lin[a + (long)(n - 1) * st];
      if (l == n) v = v + cL1 * lin[a - (long)(n - 1) * st];
    }
    lout[a] = v;
  }
}

// Crank-Nicolson: out = M^-1 N q.  With dgtsv's factors M = L U (L unit
// lower with multipliers fact(r), U upper with D'(r), DU(r)), the adjoint
// solves U^T z = lam (forward), L^T y = z (backward), then applies N^T:
//   lam_q(r) = CC(r)y(r) + CR(r-1)y(r-1) + CL(r+1)y(r+1)
// plus CL(0)y(0) in row 0 and CR(n-1)y(n-1) in the last row (the Neumann
// columns of N).  One thread per line; z is parked in the output line.
// y and z lines: 32 neighbouring lines of a grain to a warp, rows CB_U at a
// time with all loads before the first dependent operation (k_cn_solve_b's
// layout).  ROWS: the table is by row, and divisions by the pivots take three
// operations; a table by field (geometry that varies along i) has not the
// values for that, and its rows are divided one by one.  Latency of the loads
// and of the chain of quotients bound it (121x104x45, 5 grains: y 47 us with
// div_rn_rcp, 33 now; z 43 -> 21).
template <int DIR, bool ROWS>
__global__ void __launch_bounds__(32 * CB_WARPS, 2) k_adj_cn(Layout L, LineMap map, const double *__restrict__ lin,
                                                             double *__restrict__ lout, CnTab tab,
                                                             const int32_t *__restrict__ aloft) {
  int a, b, g;
  long base, st;
  if (!cb_line<DIR>(L, &a, &b, &g, &base, &st)) return;
  const int n = (DIR == 1) ? L.ny : L.nz;
  const double *li = lin + base;
  double *lo = lout + base;
  if (!aloft[g]) {
    for (int r = 0; r < n; r++) lo[(long)r * st] = 0.0;
    return;
  }
  const long u = map.u(a, b);
  const double2 *const row2 = reinterpret_cast<const double2 *>(tab.p + CN_ROW * u * n);  // FACT,CL CC,CR DU,ZH ZL,ZLL
  auto two = [&](int r, int c) {  // fields 2c, 2c+1 of row r
    return ROWS ? __ldg(row2 + 4 * r + c) : make_double2(tab.at(2 * c, r, u), tab.at(2 * c + 1, r, u));
  };
  const bool hard = !ROWS || __ldg(tab.runs() + 2 * tab.U + u) != 0.0;
  // U^T z = lam
  double zp = 0.0, du = 0.0;  // z and DU of the row before
  for (int r0 = 0; r0 < n; r0 += CB_U) {
    double x[CB_U], z[CB_U];
    double2 c[CB_U], d[CB_U];
#pragma unroll
    for (int e = 0; e < CB_U; e++) {
      const int r = r0 + e < n ? r0 + e : n - 1;
      x[e] = __ldg(li + (long)r * st);
      c[e] = two(r, 2);
      d[e] = ROWS ? two(r, 3) : make_double2(0.0, 0.0);
    }
    const double zs = zp, dus = du;
    bool bad = hard;
#pragma unroll
    for (int e = 0; e < CB_U; e++) {
      const double num = (e == 0 && r0 == 0) ? x[e] : x[e] - du * zp;
      bad = bad || !div_rn_3_takes(num);
      zp = div_rn_3(num, c[e].y, d[e].x, d[e].y);
      du = c[e].x;
      z[e] = zp;
    }
    if (bad) {
      zp = zs;
      du = dus;
      for (int e = 0; e < CB_U && r0 + e < n; e++) {
        const double v = __ldg(li + (long)(r0 + e) * st);
        zp = ieee_div(r0 + e == 0 ? v : v - du * zp, tab.at(CN_DP, r0 + e, u));
        du = two(r0 + e, 2).x;
        lo[(long)(r0 + e) * st] = zp;
      }
    } else {
#pragma unroll
      for (int e = 0; e < CB_U; e++)
        if (r0 + e < n) lo[(long)(r0 + e) * st] = z[e];
    }
  }
  // L^T y = z, with lam_q(q) emitted as soon as y(q-1) is known
  double y1 = lo[(long)(n - 1) * st], y2 = 0.0;  // y(q), y(q+1)
  double2 f1 = two(n - 1, 0), g1 = two(n - 1, 1);  // rows q
  double cl2 = 0.0;                                                            // CL(q+1)
  {
    const double2 f0 = two(n - 2, 0), g0 = two(n - 2, 1);
    const double y0 = lo[(long)(n - 2) * st] - f1.x * y1;
    double v = g1.x * y1;
    v = v + g0.y * y0;
    v = v + g1.y * y1;
    lo[(long)(n - 1) * st] = v;
    cl2 = f1.y;
    y2 = y1;
    y1 = y0;
    f1 = f0;
    g1 = g0;
  }
  auto row = [&](int q, double z, double2 f0, double2 g0) {  // row q from row q-1
    const double y0 = z - f1.x * y1;
    double v = g1.x * y1;
    v = v + g0.y * y0;
    v = v + cl2 * y2;
    lo[(long)q * st] = v;
    cl2 = f1.y;
    y2 = y1;
    y1 = y0;
    f1 = f0;
    g1 = g0;
  };
  int q = n - 2;
  for (; q >= CB_U; q -= CB_U) {
    double z[CB_U];
    double2 f[CB_U], c[CB_U];
#pragma unroll
    for (int e = 0; e < CB_U; e++) {
      z[e] = lo[(long)(q - e - 1) * st];
      f[e] = two(q - e - 1, 0);
      c[e] = two(q - e - 1, 1);
    }
#pragma unroll
    for (int e = 0; e < CB_U; e++) row(q - e, z[e], f[e], c[e]);
  }
  for (; q >= 1; q--) row(q, lo[(long)(q - 1) * st], two(q - 1, 0), two(q - 1, 1));
  double v = g1.x * y1;
  v = v + cl2 * y2;
  v = v + f1.y * y1;
  lo[0] = v;
}

// x lines, through RowTile: upwards for U^T z = lam, then downwards for the
// rest.  lam_q(q) needs y(q-1), so a chunk's results are its cells shifted by
// one, and the line's first cell comes last.  121x104x45, 5 grains, x and y
// together: 190 -> 89 us, a lane per line at the row pitch before.
__global__ void __launch_bounds__(32 * RT_WARPS, 2) k_adj_cn_x(Layout L, LineMap map, const double *__restrict__ lin,
                                                               double *__restrict__ lout, CnTab tab,
                                                               const int32_t *__restrict__ aloft) {
  __shared__ double sh[RT_WARPS][32 * RT_S];
  RowTile T;
  if (!T.init(L, sh[threadIdx.x >> 5], L.nx)) return;  // uniform over the warp
  const bool act = aloft[T.g] != 0;
  const int n = L.nx, nch = (n + 31) >> 5;
  const long u = map.u(T.j, T.k);
  CnRun R;
  cn_load_run(tab, u, R);
  auto co = [&](int f, int l) { return cn_coef(tab, u, R, f, l); };
  double next[32];
  double *const own = T.own;
  T.fetch(next, lin, 0);
  double zp = 0.0;
  for (int ch = 0; ch < nch; ch++) {
    const int c0 = 32 * ch, cnt = n - c0 < 32 ? n - c0 : 32;
    T.fill(next);
    if (ch + 1 < nch) T.fetch(next, lin, c0 + 32);
    for (int e0 = 0; e0 < cnt; e0 += CB_U) {
      double du[CB_U], dp[CB_U], zh[CB_U];
#pragma unroll
      for (int e = 0; e < CB_U; e++) {
        const int r = c0 + e0 + e < n ? c0 + e0 + e : n - 1;
        du[e] = co(CN_DU, r > 0 ? r - 1 : 0);
        dp[e] = co(CN_DP, r);
        zh[e] = co(CN_ZH, r);
      }
#pragma unroll
      for (int e = 0; e < CB_U; e++) {
        if (e0 + e >= cnt) break;
        const double x = own[e0 + e];
        zp = div_rn_rcp((e == 0 && c0 + e0 == 0) ? x : x - du[e] * zp, dp[e], zh[e]);
        own[e0 + e] = act ? zp : 0.0;
      }
    }
    if (ch + 1 < nch) T.drain(lout, c0, 0, cnt);
  }
  // downwards; the last chunk is still in the tile
  double y2 = 0.0, y1 = 0.0;
  __syncwarp();
  for (int ch = nch - 1; ch >= 0; ch--) {
    const int c0 = 32 * ch, cnt = n - c0 < 32 ? n - c0 : 32;
    if (ch != nch - 1) T.fill(next);
    if (ch > 0) T.fetch(next, lout, c0 - 32);
    for (int e0 = cnt - 1; e0 >= 0; e0 -= CB_U) {
      double fa[CB_U], cc[CB_U], cr[CB_U], cl[CB_U];
#pragma unroll
      for (int e = 0; e < CB_U; e++) {
        const int r = c0 + e0 - e > 0 ? c0 + e0 - e : 0;  // y(r) is next, q = r + 1
        const int q = r + 1 < n ? r + 1 : n - 1;
        fa[e] = co(CN_FACT, q);
        cc[e] = co(CN_CC, q);
        cr[e] = co(CN_CR, r);
        cl[e] = co(CN_CL, q + 1 < n ? q + 1 : n - 1);
      }
#pragma unroll
      for (int e = 0; e < CB_U; e++) {
        if (e0 - e < 0) break;
        const int q = c0 + e0 - e + 1;
        double y0 = own[e0 - e];
        if (q < n) {
          y0 = y0 - fa[e] * y1;
          double v = cc[e] * y1;
          v = v + cr[e] * y0;
          v = v + (q < n - 1 ? cl[e] * y2 : co(CN_CR, n - 1) * y1);
          own[e0 - e + 1] = act ? v : 0.0;
        }
        y2 = y1;
        y1 = y0;
      }
    }
    T.drain(lout, c0 + 1, 1, c0 + cnt < n ? cnt : cnt - 1);
  }
  if (T.lane < T.nr) {
    double v = co(CN_CC, 0) * y1;
    v = v + co(CN_CL, 1) * y2;
    v = v + co(CN_CL, 0) * y1;
    lout[(long)(T.r0 + T.lane) * L.P] = act ? v : 0.0;
  }
}

template <int DIR>
static int launch_adj_diff_dir(a3g_ctx *ctx, const double *lin, double *lout) {
  const Layout &L = ctx->L;
  const Geo3 &sig = (DIR == 0) ? ctx->snx : (DIR == 1) ? ctx->sny : ctx->snz;
  const Geo3 &kk = (DIR == 0) ? ctx->kx : (DIR == 1) ? ctx->ky : ctx->kz;
  dim3 grid((L.nx + 31) / 32, (L.ny + 7) / 8, L.nz);
  const Box full{1, L.nx, 1, L.ny, 1, L.nz};
  tbegin(ctx, A3G_K_ADJOINT);
  if (!(DIR == 2 && run_diff_z<true>(ctx, full, full, lin, lout)))
    k_adj_diff<DIR><<<grid, dim3(32, 8), 0, ctx->stream>>>(L, ctx->grid.periodic, lin, lout, sig, ctx->kappa,
                                                         kk, ctx->aloft, ctx->sc);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// lam_out <- (D_h)^T lam_in of the explicit horizontal sweeps in one pass, the
// x transpose first or the y transpose first; *done false where they have to
// be launched one by one (launch_adj_diffuse).
int launch_adj_diff_horz(a3g_ctx *ctx, bool xfirst, const double *lin, double *lout, bool *done) {
  *done = diff_table(ctx);
  if (!*done) return A3G_OK;
  const Box full{1, ctx->L.nx, 1, ctx->L.ny, 1, ctx->L.nz};
  tbegin(ctx, A3G_K_ADJOINT);
  run_diff_xy<true>(ctx, xfirst, full, full, lin, lout);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

template <int DIR>
static int launch_adj_cn_dir(a3g_ctx *ctx, const double *lin, double *lout) {
  const Layout &L = ctx->L;
  const int n = (DIR == 0) ? L.nx : (DIR == 1) ? L.ny : L.nz;
  if (n <= 1) {  // the forward sweep leaves ts0 unchanged (:770)
    A3G_CUDA(cudaMemcpyAsync(lout, lin, sizeof(double) * L.PG * L.ns, cudaMemcpyDeviceToDevice,
                             ctx->stream));
    return A3G_OK;
  }
  const LineMap map = line_map<DIR>(ctx);
  CnTab tab;
  tbegin(ctx, A3G_K_ADJOINT);
  int rc = cn_table<DIR>(ctx, map, false, &tab);
  if (rc) return rc;
  if (DIR == 0) {
    int threads;
    const dim3 grid = rt_grid(L, &threads);
    k_adj_cn_x<<<grid, threads, 0, ctx->stream>>>(L, map, lin, lout, tab, ctx->aloft);
  } else {
    int threads;
    const dim3 grid = cb_grid<DIR == 0 ? 1 : DIR>(L, &threads);
    if (tab.byrow)
      k_adj_cn<DIR == 0 ? 1 : DIR, true><<<grid, threads, 0, ctx->stream>>>(L, map, lin, lout, tab, ctx->aloft);
    else
      k_adj_cn<DIR == 0 ? 1 : DIR, false><<<grid, threads, 0, ctx->stream>>>(L, map, lin, lout, tab, ctx->aloft);
  }
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// lam_out <- D^T lam_in for the diffusion sweep along dir (explicit or CN
// as the context is configured).  Full box.
int launch_adj_diffuse(a3g_ctx *ctx, int dir, const double *lin, double *lout) {
  if (ctx->prm.use_cn) {
    if (dir == 0) return launch_adj_cn_dir<0>(ctx, lin, lout);
    if (dir == 1) return launch_adj_cn_dir<1>(ctx, lin, lout);
    return launch_adj_cn_dir<2>(ctx, lin, lout);
  }
  if (dir == 0) return launch_adj_diff_dir<0>(ctx, lin, lout);
  if (dir == 1) return launch_adj_diff_dir<1>(ctx, lin, lout);
  return launch_adj_diff_dir<2>(ctx, lin, lout);
}

}  // namespace a3g
