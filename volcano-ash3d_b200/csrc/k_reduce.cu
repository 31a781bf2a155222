// k_reduce.cu -- reductions and small per-step kernels.
//
//  * CFL maxima and the dt arithmetic of Adjust_DT (src/Adjust_dt.f90:136-332):
//    maxima are exact and order independent, so the result is bit-identical
//    to the CPU loop (NaNs are skipped as the reference's `if (tmp.gt.max)`
//    skips them; a met step's are combined with atomicMax on the IEEE bit
//    patterns of non-negative doubles).
//  * mass totals (src/Output_Vars.f90:1255-1459): per-grain sums of c*kappa,
//    eight cells of a row added pairwise in double, their sums accumulated in
//    double-double (TwoSum) and combined in a fixed order, so the result is
//    deterministic and within a few ulp of the exact sum.
//  * subgrid plane occupancy for get_minmax_index (src/Calc_Mesh.f90:432-542).
//  * met-step interpolation (src/MesoInterpolater.f90:207-223) and the vent
//    column source insertion (src/Ash3d.F90:428-431).
#include "a3g_internal.cuh"
#include "exact_div.cuh"

#include <cstring>

namespace a3g {

__device__ __forceinline__ void atomic_max_pos(double *addr, double v) {
  if (!(v == v)) return;  // NaN: ignored like the reference's comparisons
  atomicMax(reinterpret_cast<unsigned long long *>(addr),
            (unsigned long long)__double_as_longlong(v));
}
__device__ __forceinline__ void atomic_min_pos(double *addr, double v) {
  if (!(v == v)) return;
  atomicMin(reinterpret_cast<unsigned long long *>(addr),
            (unsigned long long)__double_as_longlong(v));
}

__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmx(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// What Adjust_DT's last block does with the maxima (k_dt_finalize's arguments).
struct DtArgs {
  int latlon, use_diffusion, use_cn, n_gs_aloft;
  double dx, dy, cfl, dt_min, dt_max, imp_dt_fac, eps_small, time, next_write_time, simtime;
  int diff_fresh, meso;
};

// dt arithmetic, src/Adjust_dt.f90:176-179 and :288-332.
// meso (FAST_DT, Adjust_DT(mesostep=.true.)): bit 1 first copies
// dt_meso_next to dt_meso_last (the toggle of src/MesoInterpolater.f90:187),
// bit 0 stores the dt formed here as dt_meso_next (src/Adjust_dt.f90:335-337).
__device__ void dt_finalize(const DtArgs &a, DevScalars *sc) {
  if (a.meso & 2) sc->dt_meso_last = sc->dt_meso_next;
  double vx_dx = sc->vmax[0], vy_dy = sc->vmax[1], vz_dz = sc->vmax[2];
  if (!a.latlon) {
    vx_dx = vx_dx / a.dx;
    vy_dy = vy_dy / a.dy;
  }
  if (a.n_gs_aloft == 0) vz_dz = 0.0;
  const double time_advect = 1.0 / fmx(fmx(vx_dx, vy_dy), vz_dz);
  double td;
  if (a.use_diffusion) {
    if (a.diff_fresh) {
      td = sc->time_diffuse;  // min(DT_MAX, min_cells tmp4)
      td = a.use_cn ? td * a.imp_dt_fac : td * 0.5;
      sc->time_diffuse = td;
      sc->have_diffuse = 1;
    } else {
      td = sc->time_diffuse;
    }
  } else {
    td = a.dt_max;
  }
  const double dt_tmp = fmn(time_advect, td);
  double dt;
  if (dt_tmp < a.dt_min) dt = a.dt_min;
  else if (dt_tmp > a.dt_max) dt = a.dt_max;
  else dt = fmn(1.0, a.cfl) * dt_tmp;
  const long long fac = (long long)(dt / a.dt_min);
  dt = a.dt_min * (double)fac;
  if ((a.next_write_time - a.time) > a.eps_small && (a.next_write_time - a.time) < dt) dt = a.next_write_time - a.time;
  if (a.time + dt > a.simtime) dt = a.simtime - a.time;
  sc->dt = dt;
  if (a.meso & 1) sc->dt_meso_next = dt;
}

// The last block of a grid to come here (true in every thread of that block):
// what the others wrote before is visible to it.  The counter is left at zero.
__device__ bool last_block(unsigned *counter, unsigned nblocks) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(counter, 1u) == nblocks - 1;
    if (last) {
      *counter = 0u;
      __threadfence();
    }
  }
  __syncthreads();
  return last;
}

// CFL maxima: vmax[0] |vx| (projected) or max |vx|*minsig/kappa (lon/lat);
// vmax[1] the same for y; vmax[2] the vertical (|vz| + max_g |vf|)/dz_k
// (src/Adjust_dt.f90:136-173); then, with `finish`, the step's dt and (dtv not
// null, a small kappa table) dt/kappa, by the last block.  A warp takes a row:
// where the row's geometry and settling speeds are constant along i, the
// products and quotients are formed once, from the row's largest winds --
// rounding is monotone, so the maximum is the same.  Bound by the winds' 24 B a
// cell; with per-warp atomics on three words, a memset before and the dt in a
// kernel of its own it took 26 us on 93x131x37 (2 of them the dt kernel), now 14.
__global__ void __launch_bounds__(256) k_cfl(Layout L, int latlon, const double *__restrict__ vx,
                                             const double *__restrict__ vy,
                                             const double *__restrict__ vz, Geo4 vf, Geo3 snx,
                                             Geo3 sny, Geo3 kap, const double *__restrict__ dz_vec,
                                             double *__restrict__ part, unsigned *__restrict__ counter, int finish,
                                             DtArgs args, double *__restrict__ dtv, int dtv_len, DevScalars *sc) {
  __shared__ double sh[3][8];
  const int nrow = L.ny * L.nz, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool vf_const = vf.si == 0 && vf.sj == 0 && vf.sk == 0;  // per-grain settling speeds
  const bool row_const = vf_const && (!latlon || (snx.si == 0 && sny.si == 0 && kap.si == 0));
  double vf0 = 0.0;
  if (vf_const)
    for (int g = 0; g < L.ns; g++) {
      const double a = fabs(vf.at(1, 1, 1, g));
      if (g == 0 || a > vf0) vf0 = a;
    }
  double m0 = 0.0, m1 = 0.0, m2 = 0.0;
  auto cell = [&](int i, int j, int k, double ax, double ay, double az, double vfm) {
    double t1 = ax, t2 = ay;
    if (latlon) {
      const double kp = kap.at(i, j, k);
      t1 = ax * fmn(snx.at(i, j, k), snx.at(i + 1, j, k)) / kp;
      t2 = ay * fmn(sny.at(i, j, k), sny.at(i, j + 1, k)) / kp;
    }
    const double t3 = (az + vfm) / dz_vec[k + 1];
    if (t1 > m0) m0 = t1;
    if (t2 > m1) m1 = t2;
    if (t3 > m2) m2 = t3;
  };
  for (int r = blockIdx.x * 8 + w; r < nrow; r += gridDim.x * 8) {
    const int j = r % L.ny + 1, k = r / L.ny + 1;
    const long rb = (long)r * L.P;
    double ax = -INFINITY, ay = -INFINITY, az = -INFINITY;  // of no wind: a row that is all NaN sets no limit
#pragma unroll 4
    for (int i = lane; i < L.nx; i += 32) {
      const double x = fabs(vx[rb + i]), y = fabs(vy[rb + i]), z = fabs(vz[rb + i]);
      if (row_const) {
        if (x > ax) ax = x;
        if (y > ay) ay = y;
        if (z > az) az = z;
      } else {
        double vfm = vf0;
        if (!vf_const) {
          vfm = 0.0;
          for (int g = 0; g < L.ns; g++) {
            const double a = fabs(vf.at(i + 1, j, k, g));
            if (g == 0 || a > vfm) vfm = a;
          }
        }
        cell(i + 1, j, k, x, y, z, vfm);
      }
    }
    if (row_const) cell(1, j, k, ax, ay, az, vf0);
  }
  auto block_max = [&]() {  // the block's maxima, in thread 0
    m0 = warp_max(m0);
    m1 = warp_max(m1);
    m2 = warp_max(m2);
    if (lane == 0) {
      sh[0][w] = m0;
      sh[1][w] = m1;
      sh[2][w] = m2;
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int q = 1; q < 8; q++) {
        m0 = fmx(m0, sh[0][q]);
        m1 = fmx(m1, sh[1][q]);
        m2 = fmx(m2, sh[2][q]);
      }
  };
  block_max();
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x] = m0;
    part[3 * blockIdx.x + 1] = m1;
    part[3 * blockIdx.x + 2] = m2;
  }
  if (!last_block(counter, gridDim.x)) return;
  m0 = m1 = m2 = 0.0;
  for (int q = threadIdx.x; q < (int)gridDim.x; q += 256) {
    m0 = fmx(m0, __ldcg(part + 3 * q));
    m1 = fmx(m1, __ldcg(part + 3 * q + 1));
    m2 = fmx(m2, __ldcg(part + 3 * q + 2));
  }
  block_max();
  if (threadIdx.x == 0) {
    sc->vmax[0] = m0;
    sc->vmax[1] = m1;
    sc->vmax[2] = m2;
    sc->vmax[3] = 0.0;
    if (finish) dt_finalize(args, sc);
  }
  if (finish && dtv) {
    __syncthreads();
    const double dt = sc->dt;
    for (int t = threadIdx.x; t < dtv_len; t += 256) dtv[t] = dt / kap.p[t];
  }
}

// Diffusion time limit, src/Adjust_dt.f90:191-235 (min over cells of
// sum_d (kappa/minsig_d)^2 / k_d, starting from DT_MAX).
__global__ void __launch_bounds__(256) k_diff_limit(Layout L, Geo3 snx, Geo3 sny, Geo3 snz,
                                                    Geo3 kap, Geo3 kx, Geo3 ky, Geo3 kz,
                                                    DevScalars *sc) {
  const long ncell = (long)L.nx * L.ny * L.nz;
  double m = 1.0e300;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < ncell; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)(t % L.nx) + 1;
    const long r = t / L.nx;
    const int j = (int)(r % L.ny) + 1;
    const int k = (int)(r / L.ny) + 1;
    const double kp = kap.at(i, j, k);
    const double r1 = kp / fmn(snx.at(i, j, k), snx.at(i + 1, j, k));
    const double t1 = (r1 * r1) / kx.at(i, j, k);
    const double r2 = kp / fmn(sny.at(i, j, k), sny.at(i, j + 1, k));
    const double t2 = (r2 * r2) / ky.at(i, j, k);
    const double r3 = kp / fmn(snz.at(i, j, k), snz.at(i, j, k + 1));
    const double t3 = (r3 * r3) / kz.at(i, j, k);
    const double t4 = t1 + t2 + t3;
    if (t4 < m) m = t4;
  }
  m = warp_min(m);
  if ((threadIdx.x & 31) == 0) atomic_min_pos(&sc->time_diffuse, m);
}

__global__ void k_dt_finalize(DtArgs args, DevScalars *sc) { dt_finalize(args, sc); }

// Adjust_DT(mesostep=.true.), the FAST_DT branch of src/Adjust_dt.f90:96-135:
// the maxima over the FP32 met step `vx,vy,vz` (m/s, [k][j][i] without
// padding), widened and scaled as the reference writes them:
//   projected: real(max|vx_sp|)*3.6 (divided by dx in k_dt_finalize);
//   lon/lat:   real(|vx_sp|)*3.6*minsig/kappa per cell;
//   vertical:  real(|vz_sp| + max_g|vf_sp|)*3.6/dz_k, the sum in FP32.
// real(.)*3.6 is monotone, so the projected maximum of the scaled cells is the
// scaled maximum.  vfm: max_g |vf_meso_next_step_sp| per cell, or null for
// the single value vfm0.
__global__ void __launch_bounds__(256) k_cfl_meso(Layout L, int latlon, const float *__restrict__ vx,
                                                  const float *__restrict__ vy, const float *__restrict__ vz,
                                                  const float *__restrict__ vfm, float vfm0, Geo3 snx, Geo3 sny,
                                                  Geo3 kap, const double *__restrict__ dz_vec, DevScalars *sc) {
  const int nrow = L.ny * L.nz;
  double m0 = 0.0, m1 = 0.0, m2 = 0.0;
  for (int r = blockIdx.x; r < nrow; r += gridDim.x) {
    const int j = r % L.ny + 1, k = r / L.ny + 1;
    const double rdz = dz_vec[k + 1];
    const long rb = (long)r * L.nx;
    for (int i = threadIdx.x + 1; i <= L.nx; i += blockDim.x) {
      const long c = rb + (i - 1);
      const double ax = (double)fabsf(vx[c]) * 3.6, ay = (double)fabsf(vy[c]) * 3.6;
      double t1, t2;
      if (latlon) {
        const double kp = kap.at(i, j, k);
        t1 = ax * fmn(snx.at(i, j, k), snx.at(i + 1, j, k)) / kp;
        t2 = ay * fmn(sny.at(i, j, k), sny.at(i, j + 1, k)) / kp;
      } else {
        t1 = ax;
        t2 = ay;
      }
      const float s = __fadd_rn(fabsf(vz[c]), vfm ? vfm[c] : vfm0);
      const double t3 = (double)s * 3.6 / rdz;
      if (t1 > m0) m0 = t1;
      if (t2 > m1) m1 = t2;
      if (t3 > m2) m2 = t3;
    }
  }
  m0 = warp_max(m0);
  m1 = warp_max(m1);
  m2 = warp_max(m2);
  if ((threadIdx.x & 31) == 0) {
    atomic_max_pos(&sc->vmax[0], m0);
    atomic_max_pos(&sc->vmax[1], m1);
    atomic_max_pos(&sc->vmax[2], m2);
  }
}

// The FAST_DT step dt of src/MesoInterpolater.f90:250-258: interpolated
// between the met steps' dt (no DT_MIN rounding), then clipped to the next
// write time and the end of the simulation.
// Every thread forms it, thread 0 stores it, and (dtv not null) all write dt/kappa.
__global__ void k_fast_dt(double frac, double eps_small, double time, double next_write_time, double simtime,
                          const double *__restrict__ kap, double *__restrict__ dtv, int dtv_len, DevScalars *sc) {
  const double last = sc->dt_meso_last, next = sc->dt_meso_next;
  double dt = last + (next - last) * frac;
  if ((next_write_time - time) > eps_small && (next_write_time - time) < dt) dt = next_write_time - time;
  if (time + dt > simtime) dt = simtime - time;
  if (threadIdx.x == 0) sc->dt = dt;
  if (dtv)
    for (int t = threadIdx.x; t < dtv_len; t += blockDim.x) dtv[t] = dt / kap[t];
}

// dt/kappa's buffer for a kernel that forms dt and, where kappa's table is
// small (a projected grid's; one block forms it within a microsecond or two),
// dt/kappa with it; null where k_dtv is left to do it.
double *dtv_target(const a3g_ctx *ctx) {
  return ctx->have_geometry && ctx->kappa_len <= 2048 ? ctx->dtv_buf : nullptr;
}

// After such a kernel's launch, and only if it was not refused: dt is another,
// and dt/kappa (dtv, from dtv_target) is of that dt.
void dt_formed(a3g_ctx *ctx, const double *dtv) {
  ctx->dt_stamp++;
  if (!dtv) return;
  ctx->dtv_valid = true;
  ctx->dtv_stamp = ctx->dt_stamp;
}

int launch_cfl_maxima_meso(a3g_ctx *ctx, int slot) {
  const long n = ctx->met_n;
  return launch_cfl_maxima_meso_ptr(ctx, ctx->met + (size_t)3 * n * (slot == 0 ? ctx->met_last : ctx->met_next));
}

// the maxima over a met step (vx, vy, vz of nx*ny*nz FP32 each) at m
int launch_cfl_maxima_meso_ptr(a3g_ctx *ctx, const float *m) {
  const Layout &L = ctx->L;
  A3G_CUDA(cudaMemsetAsync(ctx->sc->vmax, 0, sizeof(ctx->sc->vmax), ctx->stream));
  const long n = (long)L.nx * L.ny * L.nz;
  const long ncell = (long)L.nx * L.ny * L.nz;
  int blocks = (int)((ncell + 255) / 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  tbegin(ctx, A3G_K_CFL);
  k_cfl_meso<<<blocks, 256, 0, ctx->stream>>>(L, ctx->grid.latlon, m, m + n, m + 2 * n, ctx->vfm_sp,
                                              ctx->vfm_sp_const, ctx->snx, ctx->sny, ctx->kappa, ctx->dz_vec,
                                              ctx->sc);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_fast_dt(a3g_ctx *ctx, double frac, double time, double next_write_time, double simtime) {
  tbegin(ctx, A3G_K_OTHER);
  double *const dtv = dtv_target(ctx);
  k_fast_dt<<<1, 256, 0, ctx->stream>>>(frac, ctx->prm.eps_small, time, next_write_time, simtime, ctx->kappa.p, dtv,
                                        (int)ctx->kappa_len, ctx->sc);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  dt_formed(ctx, dtv);
  return A3G_OK;
}

static DtArgs dt_args(const a3g_ctx *ctx, int n_gs_aloft, double time, double next_write_time, double simtime,
                      int fresh, int meso) {
  return DtArgs{ctx->grid.latlon,  ctx->prm.use_diffusion, ctx->prm.use_cn,  n_gs_aloft,       ctx->grid.dx,
                ctx->grid.dy,      ctx->prm.cfl,           ctx->prm.dt_min,  ctx->prm.dt_max,  ctx->prm.imp_dt_fac,
                ctx->prm.eps_small, time,                  next_write_time,  simtime,          fresh,
                meso};
}

// blocks of k_cfl: two rows a warp at least, and a few blocks per SM
static int cfl_blocks(const Layout &L) {
  const int n = (L.ny * L.nz + 15) / 16;
  return n < CFL_BLOCKS ? n : CFL_BLOCKS;
}

static int run_cfl(a3g_ctx *ctx, int finish, const DtArgs &args, double *dtv) {
  const Layout &L = ctx->L;
  tbegin(ctx, A3G_K_CFL);
  k_cfl<<<cfl_blocks(L), 256, 0, ctx->stream>>>(L, ctx->grid.latlon, ctx->vx, ctx->vy, ctx->vz, ctx->vf, ctx->snx,
                                               ctx->sny, ctx->kappa, ctx->dz_vec, ctx->cfl_part,
                                               ctx->block_count + 1, finish, args, dtv, (int)ctx->kappa_len, ctx->sc);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_cfl_maxima(a3g_ctx *ctx) { return run_cfl(ctx, 0, dt_args(ctx, 0, 0.0, 0.0, 0.0, 0, 0), nullptr); }

// The diffusion time limit, formed the first time a dt needs it; *fresh is 1
// when it was formed now.
static int diffusion_limit(a3g_ctx *ctx, int *fresh) {
  const Layout &L = ctx->L;
  *fresh = 0;
  if (!ctx->prm.use_diffusion || ctx->h_sc->have_diffuse) return A3G_OK;
  const long ncell = (long)L.nx * L.ny * L.nz;
  int blocks = (int)((ncell + 255) / 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  const double init = ctx->prm.dt_max;
  A3G_CUDA(cudaMemcpyAsync(&ctx->sc->time_diffuse, &init, sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  tbegin(ctx, A3G_K_CFL);
  k_diff_limit<<<blocks, 256, 0, ctx->stream>>>(L, ctx->snx, ctx->sny, ctx->snz, ctx->kappa, ctx->kx, ctx->ky,
                                                ctx->kz, ctx->sc);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  *fresh = 1;
  ctx->h_sc->have_diffuse = 1;  // host mirror; the device flag is set by dt_finalize
  return A3G_OK;
}

// dt from maxima already in sc->vmax (local, or set from an all-reduce).
int launch_dt_from_maxima(a3g_ctx *ctx, int n_gs_aloft, double time, double next_write_time,
                          double simtime, int meso) {
  int fresh;
  int rc = diffusion_limit(ctx, &fresh);
  if (rc) return rc;
  tbegin(ctx, A3G_K_OTHER);
  k_dt_finalize<<<1, 1, 0, ctx->stream>>>(dt_args(ctx, n_gs_aloft, time, next_write_time, simtime, fresh, meso),
                                          ctx->sc);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_cfl(a3g_ctx *ctx, double time, double next_write_time, double simtime) {
  int fresh;
  int rc = diffusion_limit(ctx, &fresh);
  if (rc) return rc;
  double *const dtv = dtv_target(ctx);
  rc = run_cfl(ctx, 1, dt_args(ctx, ctx->n_gs_aloft, time, next_write_time, simtime, fresh, 0), dtv);
  if (!rc) dt_formed(ctx, dtv);
  return rc;
}

// ---------------------------------------------------------------------------
// mass totals
// ---------------------------------------------------------------------------
struct DD {
  double hi, lo;
};
__device__ __forceinline__ DD dd_add(DD a, double b) {  // TwoSum accumulate
  const double s = a.hi + b;
  const double bb = s - a.hi;
  const double err = (a.hi - (s - bb)) + (b - bb);
  DD r;
  r.hi = s;
  r.lo = a.lo + err;
  return r;
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {
  DD r = dd_add(a, b.hi);
  r.lo = r.lo + b.lo;
  return r;
}
__device__ __forceinline__ DD dd_shfl(DD v, int o) {
  DD r;
  r.hi = __shfl_xor_sync(0xffffffffu, v.hi, o);
  r.lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
  return r;
}

// Jobs: 0 aloft (c*kappa over the interior), 1 deposit (xy1*kappa(:,:,0)),
// 2 yz1*kappa(0,:,:), 3 yz2*kappa(nx+1,:,:), 4 xz1*kappa(:,0,:),
// 5 xz2*kappa(:,ny+1,:), 6 xy2*kappa(:,:,nz+1).
constexpr int NJOBS = 7;

// nb blocks a grain for the airborne mass, fxy and fs for a face; the last block of
// the grid to finish combines the partial sums in a fixed order and writes the
// ns*NJOBS results to `out` (pinned host memory).
// Airborne mass: a warp takes a row, a lane eight cells of it at a time (four
// 16-byte loads in flight), added pairwise in double, times kappa -- once when
// it does not vary along i -- and carried in double-double: a relative error of
// three roundings per term, far inside the 1e-13 the totals keep (against sums in
// extended precision on six grids, projected and lon/lat, 0.25 to 0.43 x 2^-53 on
// average and 0.93 at most, as with every cell in double-double).
// Bound by the read of the level where that is large: 720x360x60, 10 grains,
// 339 -> 215 us; and by latency where it is small, in which every face took 296
// blocks and the combination a kernel and a copy of their own: 93x131x37, 2
// grains, 28 us and the copy -> 10.5 us.
__global__ void __launch_bounds__(256) k_totals(Layout L, const double *__restrict__ c,
                                                Geo3 kap, const double *__restrict__ yz1,
                                                const double *__restrict__ yz2,
                                                const double *__restrict__ xz1,
                                                const double *__restrict__ xz2,
                                                const double *__restrict__ xy1,
                                                const double *__restrict__ xy2, Box nz, int nb, int fxy, int fs,
                                                double *__restrict__ part, unsigned *__restrict__ counter,
                                                double *__restrict__ out) {
  const int g = blockIdx.y, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ double sh[2][8];
  DD acc = {0.0, 0.0};
  if ((int)blockIdx.x < nb) {
    // rows of the cells that can be nonzero, from the even cell at or before the first one
    const int nj = nz.jmax - nz.jmin + 1, nrow = nj * (nz.kmax - nz.kmin + 1);
    const int ib = (nz.imin - 1) & ~1, n = nz.imax - ib;
    const bool row_const = kap.si == 0;
    for (int r = blockIdx.x * 8 + w; r < nrow; r += nb * 8) {
      const int j = r % nj + nz.jmin, k = r / nj + nz.kmin;
      const double *row = c + (long)g * L.PG + L.cell(1, j, k) + ib;
      const double kr = row_const ? kap.at(1, j, k) : 0.0;
      for (int i0 = 2 * lane; i0 < n; i0 += 256) {
        double2 x[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
          x[q] = i0 + 64 * q < n ? __ldg(reinterpret_cast<const double2 *>(row + i0 + 64 * q)) : make_double2(0.0, 0.0);
        double v[8];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          v[2 * q] = x[q].x;
          v[2 * q + 1] = i0 + 64 * q + 1 < n ? x[q].y : 0.0;
        }
        if (!row_const) {
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const int i = i0 + 64 * (q >> 1) + (q & 1);
            if (i < n) v[q] = v[q] * kap.at(ib + i + 1, j, k);
          }
        }
        const double s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        acc = dd_add(acc, row_const ? s * kr : s);
      }
    }
  } else {
    // the xy faces' blocks first, fxy each, then the others', fs each
    const int x = (int)blockIdx.x - nb;
    const bool xy = x < 2 * fxy;
    const int job = xy ? (x < fxy ? 1 : 6) : (x - 2 * fxy) / fs + 2;
    const int fb = xy ? fxy : fs, b = xy ? x % fxy : (x - 2 * fxy) % fs;
    const bool yz = job == 2 || job == 3;
    const unsigned len = yz ? L.ny : L.nx, n = len * (xy ? L.ny : L.nz);
    const double *face = (job == 1 ? xy1 : job == 2 ? yz1 : job == 3 ? yz2 : job == 4 ? xz1 : job == 5 ? xz2 : xy2) +
                         (long)g * n;
    for (unsigned t = b * 256u + threadIdx.x; t < n; t += fb * 256u) {
      const int row = (int)(t / len) + 1, at = (int)(t - (row - 1) * len) + 1;
      const double v = face[t] * (xy ? kap.at(at, row, job == 1 ? 0 : L.nz + 1)
                                  : yz ? kap.at(job == 2 ? 0 : L.nx + 1, at, row)
                                       : kap.at(at, job == 4 ? 0 : L.ny + 1, row));
      acc = dd_add(acc, v);
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc = dd_add(acc, dd_shfl(acc, o));
  if (lane == 0) { sh[0][w] = acc.hi; sh[1][w] = acc.lo; }
  __syncthreads();
  const int nx = gridDim.x;
  if (threadIdx.x == 0) {
    DD s = {0.0, 0.0};
    for (int q = 0; q < 8; q++) s = dd_add(s, DD{sh[0][q], sh[1][q]});
    const long o = ((long)g * nx + blockIdx.x) * 2;
    part[o] = s.hi;
    part[o + 1] = s.lo;
  }
  if (!last_block(counter, gridDim.x * gridDim.y)) return;
  // a warp per (g, job): lanes take every 32nd partial, then a fixed shuffle tree (the same order on every run)
  for (int t = w; t < L.ns * NJOBS; t += 8) {
    const int gg = t / NJOBS, job = t % NJOBS;
    const int b0 = job == 0 ? 0 : job == 1 ? nb : job == 6 ? nb + fxy : nb + 2 * fxy + (job - 2) * fs;
    const int b1 = b0 + (job == 0 ? nb : job == 1 || job == 6 ? fxy : fs);
    DD s = {0.0, 0.0};
    for (int b = b0 + lane; b < b1; b += 32) {
      const double *p = part + ((long)gg * nx + b) * 2;
      s = dd_add(s, DD{__ldcg(p), __ldcg(p + 1)});
    }
    for (int o = 16; o > 0; o >>= 1) s = dd_add(s, dd_shfl(s, o));
    if (lane == 0) out[t] = s.hi + s.lo;
  }
}

// The totals' sums, written to h_dst (ns*NJOBS doubles of pinned memory) by the
// time the stream gets past this launch.
int launch_totals_partials(a3g_ctx *ctx, double *h_dst) {
  const Layout &L = ctx->L;
  Box nz = state_box(ctx);
  if (empty(nz)) nz = Box{1, 1, 1, 1, 1, 1};
  const int rows = (nz.jmax - nz.jmin + 1) * (nz.kmax - nz.kmin + 1);
  // four rows a warp at least, eight blocks per SM at most; 1024 face cells a block (4096 made the faces
  // the last to finish on 93x131x37: 17 us a launch, 10.5 now), from 16 blocks a face on 4096, and 64 at most
  // (16 at most were too few for 1000x1000x4, 1 grain: 77 us, 296 blocks 34, these 28)
  int nb = (rows + 31) / 32;
  const int most = 148 * 8 / L.ns > 1 ? 148 * 8 / L.ns : 1;
  if (nb > most) nb = most;
  auto face_blocks = [](long cells) {
    const long some = cells / 1024 + 1, many = cells / 4096 > 16 ? cells / 4096 : 16, n = some < many ? some : many;
    return (int)(n < 64 ? n : 64);
  };
  const int fxy = face_blocks((long)L.nx * L.ny), fs = face_blocks((long)(L.nx > L.ny ? L.nx : L.ny) * L.nz);
  tbegin(ctx, A3G_K_TOTALS);
  k_totals<<<dim3(nb + 2 * fxy + 4 * fs, L.ns), 256, 0, ctx->stream>>>(
      L, ctx->c0, ctx->kappa, ctx->out_yz1, ctx->out_yz2, ctx->out_xz1, ctx->out_xz2, ctx->out_xy1, ctx->out_xy2, nz, nb,
      fxy, fs, ctx->red_buf, ctx->block_count, h_dst);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// volumes in the reference's order, src/Output_Vars.f90:1285-1290,1395-1401,1440-1456
void totals_volumes(a3g_ctx *ctx, const double *h_src, double *out4, double *mass_aloft) {
  const int ns = ctx->L.ns;
  const double rho = ctx->prm.magma_density, km3 = 1.0e9;
  double aloft = 0.0, depv = 0.0, outv = 0.0;
  for (int g = 0; g < ns; g++) {
    const double *r = h_src + (size_t)g * NJOBS;
    if (mass_aloft) mass_aloft[g] = r[0];
    aloft = aloft + r[0] / rho / km3;
  }
  for (int g = 0; g < ns; g++) depv = depv + h_src[(size_t)g * NJOBS + 1] / rho / km3;
  for (int g = 0; g < ns; g++) {
    const double *r = h_src + (size_t)g * NJOBS;
    outv = outv + (r[2] + r[3] + r[4] + r[5] + r[6]) / rho / km3;
  }
  out4[0] = aloft;
  out4[1] = depv;
  out4[2] = outv;
  out4[3] = aloft + depv + outv;
}

// ---------------------------------------------------------------------------
// subgrid plane occupancy: flags[i] (i=1..nx), flags[nx+1+j], flags[nx+ny+2+k]
// set when some grain has c >= thresh in that plane.
// ---------------------------------------------------------------------------
// 2^lw lanes take a row of the box outside which the level is zero (a warp one
// row of 65 columns and more, several shorter ones), four cells a lane of four
// grains in flight, and a warp whose lanes have all met the threshold goes on
// to its next rows; blockIdx.y shares the grains out where the rows alone
// leave the chip idle.  A block marks planes in shared memory and hands on at
// its end what is not set yet: a cloud's warps otherwise all read and write
// the same few global words.  us a launch by events, for a thread a cell, a warp
// a row whatever its length with the global words, and now -- ash in every cell:
// 60x500x20, 1 grain, 28, 30, 13; 3x400x40, 2 grains, 13, 27, 10; 317x211x53, 7
// grains, 64, 60, 35; 480x401x50, 6 grains, 108, 129, 68; in the last of 60
// grains on 25x25x10: 18, 15, 8; no ash on 500x60x20, 1 grain: 9, 8, 10.
constexpr int PF_SMEM = 32 * 1024;  // larger extents mark the global words themselves
__global__ void __launch_bounds__(256) k_plane_flags(Layout L, Box nz, int lw, int per_y, const double *__restrict__ c,
                                                     double thresh, int32_t *__restrict__ flags) {
  extern __shared__ uint8_t pf_seen[];
  constexpr int U = 4;
  const int lane = threadIdx.x & 31, sub = lane & ((1 << lw) - 1), nf = L.nx + L.ny + L.nz + 3;
  const bool local = nf <= PF_SMEM;
  if (local)
    for (int t = threadIdx.x; t < nf; t += 256) pf_seen[t] = 0;
  __syncthreads();
  auto mark = [&](int at) {
    if (local) pf_seen[at] = 1;
    else if (!__ldcg(flags + at)) flags[at] = 1;
  };
  const int ga = blockIdx.y * per_y, gb = min(L.ns, ga + per_y);
  const int nj = nz.jmax - nz.jmin + 1, nrow = nj * (nz.kmax - nz.kmin + 1), rows = 32 >> lw;  // rows of a warp
  for (int r0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * rows; r0 < nrow; r0 += gridDim.x * 8 * rows) {
    const int r = min(r0 + (lane >> lw), nrow - 1);  // past the last row: that row again
    const int j = r % nj + nz.jmin, k = r / nj + nz.kmin;
    const double *row = c + L.cell(1, j, k);
    bool any = false;
    for (int i0 = nz.imin; i0 <= nz.imax; i0 += U << lw) {
      int at[U];  // past the row's end: its last cell again
      bool hit[U];
#pragma unroll
      for (int q = 0; q < U; q++) {
        at[q] = min(i0 + sub + (q << lw), nz.imax);
        hit[q] = false;
      }
      for (int g0 = ga; g0 < gb; g0 += 4) {
        double v[4][U];
#pragma unroll
        for (int g = 0; g < 4; g++)
#pragma unroll
          for (int q = 0; q < U; q++) v[g][q] = g0 + g < gb ? __ldg(row + (long)(g0 + g) * L.PG + at[q] - 1) : nan("");
        bool all = true;
#pragma unroll
        for (int q = 0; q < U; q++) {
#pragma unroll
          for (int g = 0; g < 4; g++) hit[q] |= v[g][q] >= thresh;
          all = all && hit[q];
        }
        if (__all_sync(0xffffffffu, all)) break;
      }
#pragma unroll
      for (int q = 0; q < U; q++)
        if (hit[q]) {
          any = true;
          mark(at[q]);
        }
    }
    const unsigned mine = __ballot_sync(0xffffffffu, any) >> (lane - sub) & (0xffffffffu >> (32 - (1 << lw)));
    if (mine && sub == 0) {
      mark(L.nx + 1 + j);
      mark(L.nx + L.ny + 2 + k);
    }
  }
  if (!local) return;
  __syncthreads();
  for (int t = threadIdx.x; t < nf; t += 256)
    if (pf_seen[t] && !__ldcg(flags + t)) flags[t] = 1;
}

int launch_plane_flags(a3g_ctx *ctx) {
  const Layout &L = ctx->L;
  const size_t nf = (size_t)L.nx + L.ny + L.nz + 3;
  A3G_CUDA(cudaMemsetAsync(ctx->plane_flags, 0, nf * sizeof(int32_t), ctx->stream));
  // a threshold of zero or less is met by the zeros outside the state's box too
  Box nz = ctx->prm.cloudcon_grid_thresh > 0.0 ? state_box(ctx) : full_box_of(L);
  if (empty(nz)) nz = Box{1, 1, 1, 1, 1, 1};
  int lw = 0;
  while (lw < 5 && (4 << lw) < nz.imax - nz.imin + 1) lw++;
  const int per = 8 * (32 >> lw);  // rows of a block
  const int rows = ((nz.jmax - nz.jmin + 1) * (nz.kmax - nz.kmin + 1) + per - 1) / per;
  // grains in one block, or in fours where that leaves less than four blocks an SM
  int ny = 148 * 4 / rows, most = (L.ns + 3) / 4;
  ny = ny < 1 ? 1 : ny < most ? ny : most;
  const int per_y = ((L.ns + ny - 1) / ny + 3) / 4 * 4;
  const dim3 grid(rows < 148 * 8 ? rows : 148 * 8, (L.ns + per_y - 1) / per_y);
  tbegin(ctx, A3G_K_OTHER);
  k_plane_flags<<<grid, 256, nf <= (size_t)PF_SMEM ? nf : 0, ctx->stream>>>(
      L, nz, lw, per_y, ctx->c0, ctx->prm.cloudcon_grid_thresh, ctx->plane_flags);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  A3G_CUDA(cudaMemcpyAsync(ctx->h_plane_flags, ctx->plane_flags, nf * sizeof(int32_t),
                           cudaMemcpyDeviceToHost, ctx->stream));
  A3G_CUDA(cudaStreamSynchronize(ctx->stream));
  return A3G_OK;
}

// ---------------------------------------------------------------------------
// winds and source
// ---------------------------------------------------------------------------
// 2^lw lanes take up to 4 * 2^lw cells of a row of one of the three winds, four
// cells a lane in flight (no division per cell); bound by the 48 B a cell.  us
// for a thread a cell, for a warp taking whole rows of all three winds, and here:
// 720x360x60, 136, 141, 134; 480x401x50, 85, 90, 81; 400x3x40, 4.2, 8.2, 4.2;
// 1000x20x10, 4.7, 13.4, 4.2.
__global__ void __launch_bounds__(256) k_interp_winds(Layout L, int lw, const float *__restrict__ last,
                                                      const float *__restrict__ next, long n, double frac,
                                                      double *__restrict__ vx, double *__restrict__ vy,
                                                      double *__restrict__ vz) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31, sub = lane & ((1 << lw) - 1), rows = 32 >> lw, nrow = L.ny * L.nz;
  const int d = blockIdx.z, i0 = blockIdx.y * (U << lw) + sub;
  const float *const a0 = last + d * n, *const b0 = next + d * n;
  double *const v0 = d == 0 ? vx : d == 1 ? vy : vz;
  for (int r = (blockIdx.x * 8 + (threadIdx.x >> 5)) * rows + (lane >> lw); r < nrow; r += gridDim.x * 8 * rows) {
    const float *a = a0 + (long)r * L.nx, *b = b0 + (long)r * L.nx;
    double *v = v0 + (long)r * L.P;
    float x[U], y[U];
#pragma unroll
    for (int q = 0; q < U; q++) {
      const bool in = i0 + (q << lw) < L.nx;
      x[q] = in ? a[i0 + (q << lw)] : 0.0f;
      y[q] = in ? b[i0 + (q << lw)] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < U; q++)
      if (i0 + (q << lw) < L.nx) v[i0 + (q << lw)] = ((double)x[q] + (double)(y[q] - x[q]) * frac) * 3.6;
  }
}

// the winds between the met steps `last` and `next` (3 FP32 arrays each)
int launch_interp_pair(a3g_ctx *ctx, const float *last, const float *next, double frac) {
  const Layout &L = ctx->L;
  int lw = 0;
  while (lw < 5 && (4 << lw) < L.nx) lw++;
  const int per = 8 * (32 >> lw), chunks = (L.nx + (4 << lw) - 1) / (4 << lw);  // rows of a block, turns of a row
  const int rows = (L.ny * L.nz + per - 1) / per, most = 148 * 16 / (3 * chunks) + 1;
  tbegin(ctx, A3G_K_WINDS);
  k_interp_winds<<<dim3(rows < most ? rows : most, chunks, 3), 256, 0, ctx->stream>>>(
      L, lw, last, next, (long)L.nx * L.ny * L.nz, frac, ctx->vx, ctx->vy, ctx->vz);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_interp_winds(a3g_ctx *ctx, double frac) {
  const long n = ctx->met_n;
  return launch_interp_pair(ctx, ctx->met + (size_t)3 * n * ctx->met_last, ctx->met + (size_t)3 * n * ctx->met_next,
                            frac);
}

// Calc_Vmod_Topo (src/Topography.f90:2138-2166) on the interior, fused with
// the sum the z sweep needs: vzh = vz + vh, vh = f(k)*(vx*dhdx + vy*dhdy)
// with f = -1.0 (ZScaling_ID 1) or s_cc(k)/Ztop - 1.0 (2), precomputed on the
// host in those operations.  The ghost levels keep plain vz (vh is zero
// there in the reference: vx_pd and vy_pd are never written at ghost k).
__global__ void __launch_bounds__(256) k_vmod_topo(Layout L, const double *__restrict__ topo,
                                                   const double *__restrict__ vx,
                                                   const double *__restrict__ vy,
                                                   const double *__restrict__ vz,
                                                   double *__restrict__ vzh) {
  const long n = (long)L.nx * L.ny * L.nz;
  const long n2 = (long)(L.nx + 4) * (L.ny + 4);
  const double *dhdx = topo, *dhdy = topo + n2, *fac = topo + 4 * n2;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)(t % L.nx) + 1;
    const long r = t / L.nx;
    const int j = (int)(r % L.ny) + 1;
    const int k = (int)(r / L.ny) + 1;
    const long c = L.cell(i, j, k);
    const long m = (long)(i + 1) + (long)(L.nx + 4) * (j + 1);
    const double vh = fac[k - 1] * (vx[c] * dhdx[m] + vy[c] * dhdy[m]);
    vzh[c] = vz[c] + vh;
  }
}

int launch_vmod_topo(a3g_ctx *ctx) {
  const long n = (long)ctx->L.nx * ctx->L.ny * ctx->L.nz;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  tbegin(ctx, A3G_K_WINDS);
  k_vmod_topo<<<blocks, 256, 0, ctx->stream>>>(ctx->L, ctx->topo_buf, ctx->vx, ctx->vy, ctx->vz, ctx->vzh);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// umbrella_winds' radial winds added to the interpolated winds over the
// cloud's bounding box and the levels ibase..itop
// (src/MesoInterpolater.f90:237-241): vx += uvx, vy += uvy.
__global__ void __launch_bounds__(256) k_umbrella_winds(Layout L, int i0, int ni, int j0, int nj, int kb,
                                                        int nk, const double *__restrict__ uv,
                                                        double *__restrict__ vx, double *__restrict__ vy) {
  const long n = (long)ni * nj * nk;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const int a = (int)(t % ni);
    const long r = t / ni;
    const int b = (int)(r % nj);
    const int k = kb + (int)(r / nj);
    const long c = L.cell(i0 + a, j0 + b, k);
    const long m = a + (long)ni * b;
    vx[c] = vx[c] + uv[m];
    vy[c] = vy[c] + uv[(long)ni * nj + m];
  }
}

int launch_umbrella_winds(a3g_ctx *ctx, int i0, int ni, int j0, int nj, const double *uv) {
  const int nk = ctx->umb_itop - ctx->umb_ibase + 1;
  const long n = (long)ni * nj * nk;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  tbegin(ctx, A3G_K_WINDS);
  k_umbrella_winds<<<blocks, 256, 0, ctx->stream>>>(ctx->L, i0, ni, j0, nj, ctx->umb_ibase, nk, uv, ctx->vx,
                                                    ctx->vy);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// Umbrella source insertion (src/Ash3d.F90:446-458): on ibase..itop the 3x3
// patch around the vent is first set to its volume-weighted average
// (AvgCon_Umbrella, src/Source_Umbrella.f90:539-560, i outer, j inner), then
// every patch cell of levels 1..nz gains dt*SourceNodeFlux_Umbrella.  One
// thread per (level, grain).
__global__ void k_source_umbrella(Layout L, int ivent, int jvent, int ibase, int itop,
                                  const double *__restrict__ sten, const double *__restrict__ flux, double dt,
                                  double *__restrict__ c) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;  // (k-1) + nz*g
  if (t >= L.nz * L.ns) return;
  const int k = t % L.nz + 1, g = t / L.nz;
  double v[3][3];
  long a[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      a[i][j] = (long)g * L.PG + L.cell(ivent - 1 + i, jvent - 1 + j, k);
      v[i][j] = c[a[i][j]];
    }
  if (k >= ibase && k <= itop) {
    double avg = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) avg = avg + v[i][j] * sten[i + 3 * j + 9 * (k - 1)];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) v[i][j] = avg;
  }
  const long f0 = 9 * ((long)(k - 1) + (long)(L.nz + 1) * g);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) c[a[i][j]] = v[i][j] + dt * flux[f0 + i + 3 * j];
}

int launch_source_umbrella(a3g_ctx *ctx, double dt) {
  touch(ctx, ctx->umb_ivent - 1, ctx->umb_ivent + 1, ctx->umb_jvent - 1, ctx->umb_jvent + 1);
  const int n = ctx->L.nz * ctx->L.ns;
  const double *sten = ctx->umb_buf;
  const double *flux = ctx->umb_buf + 9 * (size_t)ctx->L.nz;
  tbegin(ctx, A3G_K_OTHER);
  k_source_umbrella<<<(n + 127) / 128, 128, 0, ctx->stream>>>(ctx->L, ctx->umb_ivent, ctx->umb_jvent,
                                                              ctx->umb_ibase, ctx->umb_itop, sten, flux, dt,
                                                              ctx->c0);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// Scheduled source on the device: CheckEruptivePulses (src/Source.f90:613-685)
// and TephraSourceNodes (:708-783) with the step's dt from the device
// scalars, then the vent-column insertion of src/Ash3d.F90:428-431.  One
// block; thread 0 runs the pulse bookkeeping (ieruption/jeruption persist in
// state), the block inserts the (level, grain) fluxes.
constexpr int SRC_MAX_PULSES = 64;

__global__ void k_source_sched(Layout L, int ivent, int jvent, int np, const double *__restrict__ sched,
                               int32_t *__restrict__ state, const DevScalars *__restrict__ sc, Geo3 kap,
                               double time, double *__restrict__ c) {
  __shared__ double frac[SRC_MAX_PULSES + 1];
  __shared__ int ie_s, je_s, in_s;
  const double *t0 = sched, *t1 = sched + np, *mfr = sched + 2 * np, *col = sched + 3 * np;
  const double *bin = col + (size_t)np * (L.nz + 1);
  const double dt = sc->dt;
  if (threadIdx.x == 0) {
    const double tstart = time, tend = time + dt;
    const int ie = state[0];
    int je = state[1];
    int in = 0;
    for (int i = 1; i <= np; i++) frac[i] = 0.0;
    for (int i = ie; i <= np; i++) {
      bool pc = false;
      if (tstart >= t0[i - 1] && tstart < t1[i - 1]) {
        pc = true;
        je = i;
      } else if (tend > t0[i - 1] && tend <= t1[i - 1]) {
        je = i;  // :646-651: the loop exits before this pulse's fraction is formed
        break;
      } else if (tstart < t0[i - 1] && tend > t1[i - 1]) {
        pc = true;
        je = i;
      }
      if (pc) {
        in = 1;
        frac[i] = (fmin(tend, t1[i - 1]) - fmax(tstart, t0[i - 1])) / dt;
      }
    }
    ie_s = ie;
    je_s = je;
    in_s = in;
  }
  __syncthreads();
  const int ie = ie_s, je = je_s;
  if (in_s) {
    for (int t = threadIdx.x; t < L.nz * L.ns; t += blockDim.x) {
      const int k = t % L.nz + 1, g = t / L.nz;
      double tfr = 0.0;
      for (int i = ie; i <= je; i++)
        tfr = tfr + mfr[i - 1] * frac[i] * col[(ie - 1) + (size_t)np * (k - 1)];
      const double kv = kap.p[(long)(ivent + 1) * kap.si + (long)(jvent + 1) * kap.sj + (long)(k + 1) * kap.sk];
      const double flux = bin[g] * tfr / kv;
      const long a = (long)g * L.PG + L.cell(ivent, jvent, k);
      c[a] = c[a] + dt * flux;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    state[1] = je;
    if (in_s) state[0] = je;  // :776, only when TephraSourceNodes ran
  }
}

int launch_source_sched(a3g_ctx *ctx, double time) {
  touch(ctx, ctx->src_iv, ctx->src_iv, ctx->src_jv, ctx->src_jv);
  tbegin(ctx, A3G_K_OTHER);
  k_source_sched<<<1, 256, 0, ctx->stream>>>(ctx->L, ctx->src_iv, ctx->src_jv, ctx->src_np, ctx->src_sched,
                                             ctx->src_state, ctx->sc, ctx->kappa, time, ctx->c0);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

__global__ void k_source(Layout L, int ivent, int jvent, const double *__restrict__ flux, double dt,
                         double *__restrict__ c) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;  // (k-1) + nz*g
  if (t >= L.nz * L.ns) return;
  const int k = t % L.nz + 1, g = t / L.nz;
  const long a = (long)g * L.PG + L.cell(ivent, jvent, k);
  c[a] = c[a] + dt * flux[(long)(k - 1) + (long)(L.nz + 1) * g];
}

// the vent-column insertion with the step's dt read from the device scalars
__global__ void k_source_devdt(Layout L, int ivent, int jvent, const double *__restrict__ flux,
                               const DevScalars *__restrict__ sc, double *__restrict__ c) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;  // (k-1) + nz*g
  if (t >= L.nz * L.ns) return;
  const int k = t % L.nz + 1, g = t / L.nz;
  const long a = (long)g * L.PG + L.cell(ivent, jvent, k);
  c[a] = c[a] + sc->dt * flux[(long)(k - 1) + (long)(L.nz + 1) * g];
}

int launch_source_devdt(a3g_ctx *ctx, int ivent, int jvent) {
  touch(ctx, ivent, ivent, jvent, jvent);
  const int n = ctx->L.nz * ctx->L.ns;
  tbegin(ctx, A3G_K_OTHER);
  k_source_devdt<<<(n + 127) / 128, 128, 0, ctx->stream>>>(ctx->L, ivent, jvent, ctx->src_buf, ctx->sc, ctx->c0);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_source(a3g_ctx *ctx, int ivent, int jvent, double dt) {
  touch(ctx, ivent, ivent, jvent, jvent);
  const int n = ctx->L.nz * ctx->L.ns;
  tbegin(ctx, A3G_K_OTHER);
  k_source<<<(n + 127) / 128, 128, 0, ctx->stream>>>(ctx->L, ivent, jvent, ctx->src_buf, dt, ctx->c0);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// ---------------------------------------------------------------------------
// observation operators for the adjoint (no counterpart in the reference's
// transport path; the column load is Gen_Output_Vars' CloudLoad)
// ---------------------------------------------------------------------------
// CloudLoad(i,j) = sum_k sum_g c(i,j,k,g) * dz(k) / 1e3 (tonnes/km^2), in the
// order of src/Output_Vars.f90:1061-1069, without the cloud mask.
// Sums over the grains, in order, of the levels 0 .. cnt-1 of a column from p
// on: OV_K levels side by side and four grains, so that loads are in flight
// whatever the number of grains.  One level at a time with the grains' loads
// unrolled by eight left 1 to 7 grains, and the rest of a count that is no
// multiple of eight, waiting for one load after another.  us a launch by
// events for that (the compiler's own unrolling before it) and now: column
// load, 140x120x40, 4 grains, 41 (25), 19; 12: 61 (39), 30; 60: 512 (291), 250;
// products, 480x361x50, 1 grain, 78 (120 in two passes), 70; 4: 208 (149), 79; 8:
// 122 (208), 123.  Eight levels, two to eight grains or sixteen levels at a time
// were slower from four grains up (480x361x50, 4: 95 .. 107).
constexpr int OV_K = 4;
__device__ __forceinline__ void level_sums(const Layout &L, const double *__restrict__ p, int cnt, double (&t)[OV_K]) {
#pragma unroll
  for (int e = 0; e < OV_K; e++) t[e] = 0.0;
  if (cnt >= OV_K) {
#pragma unroll 4
    for (int g = 0; g < L.ns; g++, p += L.PG)
#pragma unroll
      for (int e = 0; e < OV_K; e++) t[e] = t[e] + __ldg(p + e * L.PY);
  } else {
    for (int g = 0; g < L.ns; g++, p += L.PG)
#pragma unroll
      for (int e = 0; e < OV_K; e++)
        if (e < cnt) t[e] = t[e] + __ldg(p + e * L.PY);
  }
}

__global__ void k_cloud_load(Layout L, const double *__restrict__ c, const double *__restrict__ dz_vec,
                             double *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y + 1;
  if (i > L.nx) return;
  double load = 0.0;
  for (int k0 = 1; k0 <= L.nz; k0 += OV_K) {
    double s[OV_K];
    level_sums(L, c + L.cell(i, j, k0), L.nz - k0 + 1, s);
#pragma unroll
    for (int e = 0; e < OV_K; e++)
      if (k0 + e <= L.nz) load = load + s[e] * dz_vec[k0 + e + 1] / 1.0e3;
  }
  out[(long)(j - 1) * L.nx + (i - 1)] = load;
}

// lam(i,j,k,g) += w(i,j) * dz(k) / 1e3: the transpose of the column load.
__global__ void k_adj_cloud_load(Layout L, const double *__restrict__ w, const double *__restrict__ dz_vec,
                                 double *__restrict__ lam) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y + 1;
  const int kg = blockIdx.z;
  if (i > L.nx) return;
  const int k = kg % L.nz + 1, g = kg / L.nz;
  const long a = (long)g * L.PG + L.cell(i, j, k);
  lam[a] = lam[a] + w[(long)(j - 1) * L.nx + (i - 1)] * dz_vec[k + 1] / 1.0e3;
}

// lam at the vent column, (nz+1) x ns with k fastest (row nz+1, the ghost
// that Set_BC(1) zeroes, is 0): the adjoint of the source insertion.
__global__ void k_vent_column(Layout L, int ivent, int jvent, const double *__restrict__ lam,
                              double *__restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (L.nz + 1) * L.ns) return;
  const int k = t % (L.nz + 1) + 1, g = t / (L.nz + 1);
  out[t] = (k <= L.nz) ? lam[(long)g * L.PG + L.cell(ivent, jvent, k)] : 0.0;
}

int launch_cloud_load(a3g_ctx *ctx, const double *c, double *out) {
  const Layout &L = ctx->L;
  tbegin(ctx, A3G_K_ADJOINT);
  k_cloud_load<<<dim3((L.nx + 127) / 128, L.ny), 128, 0, ctx->stream>>>(L, c, ctx->dz_vec, out);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_adj_cloud_load(a3g_ctx *ctx, const double *w, double *lam) {
  const Layout &L = ctx->L;
  tbegin(ctx, A3G_K_ADJOINT);
  k_adj_cloud_load<<<dim3((L.nx + 127) / 128, L.ny, L.nz * L.ns), 128, 0, ctx->stream>>>(L, w, ctx->dz_vec,
                                                                                        lam);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// grad(k, g) += dt * lam(ivent, jvent, k, g) / kappa(ivent, jvent, k) for
// k = 1..nz: the source-gradient gather of one reverse step, on the device
// (the same operations as the host's dt*col/kappa added to grad).
__global__ void k_vent_accumulate(Layout L, int ivent, int jvent, const double *__restrict__ lam, Geo3 kap,
                                  double dt, double *__restrict__ dst) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;  // (k-1) + nz*g
  if (t >= L.nz * L.ns) return;
  const int k = t % L.nz + 1, g = t / L.nz;
  const double kv = kap.p[(long)(ivent + 1) * kap.si + (long)(jvent + 1) * kap.sj + (long)(k + 1) * kap.sk];
  dst[t] = dst[t] + dt * lam[(long)g * L.PG + L.cell(ivent, jvent, k)] / kv;
}

int launch_vent_accumulate(a3g_ctx *ctx, int ivent, int jvent, double dt, double *dst) {
  const int n = ctx->L.nz * ctx->L.ns;
  tbegin(ctx, A3G_K_ADJOINT);
  k_vent_accumulate<<<(n + 127) / 128, 128, 0, ctx->stream>>>(ctx->L, ivent, jvent, ctx->lam0, ctx->kappa, dt,
                                                              dst);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_vent_column(a3g_ctx *ctx, int ivent, int jvent, const double *lam, double *out) {
  const int n = (ctx->L.nz + 1) * ctx->L.ns;
  k_vent_column<<<(n + 127) / 128, 128, 0, ctx->stream>>>(ctx->L, ivent, jvent, lam, out);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// ---------------------------------------------------------------------------
// output products of Gen_Output_Vars, one thread per column (i,j), in the
// reference's order: ConcentrationCalculator (src/Output_Vars.f90:1026-1123),
// AshThicknessCalculator (:855-895), the arrival-time marks (:1226-1236).
// ---------------------------------------------------------------------------
// One pass up the column (the lowest level at or below CLOUDCON_THRESH is the
// last one the reference's downward loop meets); bound by the 8 B a cell and
// grain.  cls: the cell's area classes, j fastest: bit 0 deposit, 1 cloud, 2..
// CloudLoadArea's five thresholds.
__global__ void __launch_bounds__(128) k_output_vars(
    Layout L, Box box, const double *__restrict__ c, const double *__restrict__ dz_vec,
    const double *__restrict__ zcc, const double *__restrict__ dep, double cloudcon, double cloudload_th,
    double depo_th, double density, double time, double *__restrict__ load, double *__restrict__ maxh,
    double *__restrict__ minh, double *__restrict__ maxc, int32_t *__restrict__ mcl, double *__restrict__ dthick,
    int32_t *__restrict__ mdep, uint8_t *__restrict__ cls, double *__restrict__ carr, double *__restrict__ darr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y + 1;
  if (i > L.nx) return;
  const long o = (long)(j - 1) * L.nx + (i - 1);
  const long plane = (long)L.nx * L.ny;
  // deposit thickness (mm) from DepositGranularity
  double sg = 0.0;
#pragma unroll 4
  for (int g = 0; g < L.ns; g++) sg = sg + dep[(long)g * plane + o];
  const double th = sg * dz_vec[2] / 1.0e6 / density * 1.0e3;
  const bool md = th > depo_th;
  dthick[o] = th;
  mdep[o] = md;
  double ld = 0.0, mh = 0.0, nh = 100.0, mx = 0.0;
  bool mc = false;
  unsigned bits = md ? 1u : 0u;
  if (L.ns > 0 && i >= box.imin && i <= box.imax && j >= box.jmin && j <= box.jmax) {
    bool low = false;
    for (int k0 = 1; k0 <= L.nz; k0 += OV_K) {
      double s[OV_K];
      level_sums(L, c + L.cell(i, j, k0), L.nz - k0 + 1, s);
#pragma unroll
      for (int e = 0; e < OV_K; e++) {
        const int k = k0 + e;
        if (k > L.nz) break;
        const double t = s[e];
        ld = ld + t * dz_vec[k + 1] / 1.0e3;
        if (t >= cloudcon) mh = zcc[k - 1] + 0.5 * dz_vec[k + 1];
        if (!low && t <= cloudcon) {
          low = true;
          nh = zcc[k - 1] - 0.5 * dz_vec[k + 1];
        }
        mx = (k == 1) ? t : fmx(mx, t);
      }
    }
    mc = ld >= cloudload_th;
    if (mc) {
      if (nh < 0.0 && mh > 0.0) nh = 0.0;
      nh = fmn(mh, nh);
      mx = mx * 1.0e6 / 1.0e9;
    } else {
      ld = 0.0; mx = 0.0; mh = 0.0; nh = 0.0;
    }
    bits |= mc ? 2u : 0u;
    bits |= (ld > 0.24 ? 4u : 0u) | (ld > 1.0 ? 8u : 0u) | (ld > 2.0 ? 16u : 0u) | (ld > 4.0 ? 32u : 0u) |
            (ld > 6.0 ? 64u : 0u);
  }
  load[o] = ld;
  maxh[o] = mh;
  minh[o] = nh;
  maxc[o] = mx;
  mcl[o] = mc;
  cls[(long)(i - 1) * L.ny + (j - 1)] = (uint8_t)bits;
  if (md && darr[o] < 0.0) darr[o] = time;
  if (mc && carr[o] < 0.0) carr[o] = time;
}

// Calc_vprofile (src/Output_Vars.f90:1308-1360): per profile point the
// column total (Fortran SUM order: k fastest, then the grains) against
// CLOUDCON_THRESH, and per level the sum over the grains in mg/m3.  One block
// per point; thread 0 forms the total.
__global__ void k_vprofiles(Layout L, const int32_t *__restrict__ pts, double thresh,
                            const double *__restrict__ c, double *__restrict__ out,
                            int32_t *__restrict__ written) {
  const int p = blockIdx.x;
  const int i = pts[2 * p], j = pts[2 * p + 1];
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int g = 0; g < L.ns; g++)
      for (int k = 1; k <= L.nz; k++) total = total + c[(long)g * L.PG + L.cell(i, j, k)];
    written[p] = !(total < thresh);
  }
  for (int k = 1 + threadIdx.x; k <= L.nz; k += blockDim.x) {
    double sum = 0.0;
    for (int g = 0; g < L.ns; g++) sum = sum + c[(long)g * L.PG + L.cell(i, j, k)];
    out[(long)(k - 1) + (long)L.nz * p] = sum * 1.0e6 / 1.0e9;  // KG_2_MG / KM3_2_M3
  }
}

int launch_vprofiles(a3g_ctx *ctx, int npts, const int32_t *pts, double *out, int32_t *written) {
  tbegin(ctx, A3G_K_OTHER);
  k_vprofiles<<<npts, 64, 0, ctx->stream>>>(ctx->L, pts, ctx->ov_cloudcon, ctx->c0, out, written);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_output_vars(a3g_ctx *ctx, double time, double *load, double *maxh, double *minh, double *maxc,
                       int32_t *mcl, double *dthick, int32_t *mdep, uint8_t *cls, double *carr, double *darr) {
  const Layout &L = ctx->L;
  tbegin(ctx, A3G_K_OTHER);
  k_output_vars<<<dim3((L.nx + 127) / 128, L.ny), 128, 0, ctx->stream>>>(
      L, ctx->box, ctx->c0, ctx->dz_vec, ctx->ov_zcc, ctx->out_xy1, ctx->ov_cloudcon, ctx->ov_cloudload,
      ctx->ov_depo, ctx->ov_density, time, load, maxh, minh, maxc, mcl, dthick, mdep, cls, carr, darr);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// ---------------------------------------------------------------------------
// NetCDF output arrays and restart (src/write_NETCDF.f90): FP32 (op = 4,
// src/Ash3d_VariableModules.f90:31) arrays with x fastest, the layout the
// writer passes to nf90_put_var.
// ---------------------------------------------------------------------------
// ashcon(i,j,k,g) = real(concen_pd(i,j,k,g,ts1), kind=op) (:3296-3298), and
// NC_RestartFile_LoadConcen (:3701-3707): concen_pd(i,j,k,g) = real(ashcon, ip).
// A warp takes whole rows (the level's pitch P, the array's nx), eight cells a
// lane in flight; bound by the 12 B a cell.  720x360x60, 10 grains: 601 -> 292
// us out and 590 -> 331 us in against a block per 256 cells.
constexpr int NC_U = 8;
__global__ void __launch_bounds__(256) k_pack_ashcon(Layout L, const double *__restrict__ c,
                                                     float *__restrict__ ashcon) {
  const int lane = threadIdx.x & 31;
  const long nrow = (long)L.ny * L.nz * L.ns;
  for (long r = blockIdx.x * 8L + (threadIdx.x >> 5); r < nrow; r += gridDim.x * 8L) {
    const double *src = c + r * L.P;
    float *dst = ashcon + r * L.nx;
    for (int i0 = lane; i0 < L.nx; i0 += 32 * NC_U) {
      double v[NC_U];
#pragma unroll
      for (int q = 0; q < NC_U; q++) v[q] = i0 + 32 * q < L.nx ? src[i0 + 32 * q] : 0.0;
#pragma unroll
      for (int q = 0; q < NC_U; q++)
        if (i0 + 32 * q < L.nx) dst[i0 + 32 * q] = __double2float_rn(v[q]);
    }
  }
}

__global__ void __launch_bounds__(256) k_unpack_ashcon(Layout L, const float *__restrict__ ashcon,
                                                       double *__restrict__ c) {
  const int lane = threadIdx.x & 31;
  const long nrow = (long)L.ny * L.nz * L.ns;
  for (long r = blockIdx.x * 8L + (threadIdx.x >> 5); r < nrow; r += gridDim.x * 8L) {
    const float *src = ashcon + r * L.nx;
    double *dst = c + r * L.P;
    for (int i0 = lane; i0 < L.nx; i0 += 32 * NC_U) {
      float v[NC_U];
#pragma unroll
      for (int q = 0; q < NC_U; q++) v[q] = i0 + 32 * q < L.nx ? src[i0 + 32 * q] : 0.0f;
#pragma unroll
      for (int q = 0; q < NC_U; q++)
        if (i0 + 32 * q < L.nx) dst[i0 + 32 * q] = (double)v[q];
    }
  }
}

// depocon(i,j,g) = real(DepositGranularity*dz_vec_pd(0)/KM2_2_M2, kind=op),
// then 0 where depocon <= EPS_SMALL, the FP32 value compared in FP64
// (:3320-3330).  DepositGranularity is outflow_xy1 ([g][j][i]).
__global__ void k_pack_depocon(Layout L, const double *__restrict__ xy1, const double *__restrict__ dz_vec,
                               float *__restrict__ depocon) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= L.nx) return;
  for (int g = blockIdx.z; g < L.ns; g += gridDim.z) {
    const long a = ((long)g * L.ny + j) * L.nx + i;
    float d = __double2float_rn(xy1[a] * dz_vec[1] / 1.0e6);  // dz_vec[1] = dz_vec_pd(0)
    if ((double)d <= 1.0e-6) d = 0.0f;
    depocon[a] = d;
  }
}

// outflow_xy1_pd(i,j,g) = DepositGranularity(i,j,g) = real(depocon(i,j,g), ip)
__global__ void k_unpack_depocon(Layout L, const float *__restrict__ depocon, double *__restrict__ xy1) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= L.nx) return;
  for (int g = blockIdx.z; g < L.ns; g += gridDim.z) {
    const long a = ((long)g * L.ny + j) * L.nx + i;
    xy1[a] = (double)depocon[a];
  }
}

static dim3 netcdf_grid(const Layout &L, int planes) {
  return dim3((L.nx + 255) / 256, L.ny, planes < 65535 ? planes : 65535);
}

static unsigned row_blocks(const Layout &L) {  // eight rows a block, eight blocks per SM
  const long n = ((long)L.ny * L.nz * L.ns + 7) / 8;
  return (unsigned)(n < 148 * 8 ? n : 148 * 8);
}

int launch_netcdf_pack(a3g_ctx *ctx, float *ashcon, float *depocon) {
  const Layout &L = ctx->L;
  tbegin(ctx, A3G_K_OTHER);
  if (ashcon) k_pack_ashcon<<<row_blocks(L), 256, 0, ctx->stream>>>(L, ctx->c0, ashcon);
  if (depocon)
    k_pack_depocon<<<netcdf_grid(L, L.ns), 256, 0, ctx->stream>>>(L, ctx->out_xy1, ctx->dz_vec, depocon);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

int launch_netcdf_unpack(a3g_ctx *ctx, const float *ashcon, const float *depocon) {
  const Layout &L = ctx->L;
  tbegin(ctx, A3G_K_OTHER);
  if (ashcon) k_unpack_ashcon<<<row_blocks(L), 256, 0, ctx->stream>>>(L, ashcon, ctx->c0);
  if (depocon) k_unpack_depocon<<<netcdf_grid(L, L.ns), 256, 0, ctx->stream>>>(L, depocon, ctx->out_xy1);
  tend(ctx);
  A3G_LAUNCH_CHECK(ctx);
  return A3G_OK;
}

// ---------------------------------------------------------------------------
// self-test of exact_div.cuh against the IEEE division operator
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t x) {  // splitmix64 finaliser
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  return x ^ (x >> 31);
}

__device__ double test_operand(uint64_t h) {
  const int kind = (int)(h & 15);
  const double sgn = (h & 16) ? -1.0 : 1.0;
  const uint64_t m = (h >> 12) & 0x000fffffffffffffULL;
  int e;
  if (kind < 8) e = (int)((h >> 5) & 63) - 32;          // moderate magnitudes
  else if (kind < 12) e = (int)((h >> 5) & 1023) - 512;  // wide range (fallbacks)
  else if (kind < 13) e = (int)((h >> 5) & 15) - 8;
  else if (kind < 14) e = -830 - (int)((h >> 5) & 255);  // tiny, down to subnormal (below)
  else e = (int)((h >> 5) & 7) - 4;
  double v = __longlong_as_double(
      (long long)(((uint64_t)(1023 + (kind == 13 ? e + 300 : e)) << 52) | (kind == 14 ? 0 : m)));
  if (kind == 13) v = v * 0x1p-300;  // exact while normal, rounded below 2^-1022
  if (kind == 15) v = (double)((h >> 20) & 255) - 128.0;  // small integers, zeros, exact ratios
  return sgn * v;
}

__global__ void k_selftest_div(uint64_t n, uint64_t seed, unsigned long long *bad) {
  unsigned long long local = 0;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x) {
    const double a = test_operand(mix64(seed ^ (2 * t)));
    const double b = test_operand(mix64(seed ^ (2 * t + 1)));
    if (b == 0.0) continue;
    const double q1 = div_rn(a, b), q2 = a / b;
    const double y = 1.0 / b;
    const double q3 = div_rn_rcp(a, b, y);
    const bool same1 = __double_as_longlong(q1) == __double_as_longlong(q2) || (q1 != q1 && q2 != q2);
    const bool same3 = __double_as_longlong(q3) == __double_as_longlong(q2) || (q3 != q3 && q2 != q2);
    local += (same1 ? 0 : 1) + (same3 ? 0 : 1);
  }
  if (local) atomicAdd(bad, local);
}

// A mantissa in [1, 2): any, just below 2, a few ulps from 1 or 2, or short (exact quotients).
__device__ double test_mantissa(uint64_t h) {
  uint64_t m = (h >> 8) & 0x000fffffffffffffULL;
  const int fam = (int)(h & 3);
  if (fam == 1) m |= 0x000fffff00000000ULL & ~((h >> 62) << 32);
  if (fam == 2) m = (h & 4) ? (h >> 60) : 0x000fffffffffffffULL - (h >> 60);
  if (fam == 3) m &= 0x000ffff000000000ULL;
  return __longlong_as_double((long long)(0x3ff0000000000000ULL | m));
}

// counts: wrong quotients of quot_rn and of div_rn_3 (a zero's sign aside),
// then the operands either leaves to the division operator
__global__ void k_selftest_quotients(uint64_t n, uint64_t seed, unsigned long long *counts) {
  unsigned long long c[4] = {0, 0, 0, 0};
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t h = mix64(seed ^ (3 * t + 2));
    const double ma = test_mantissa(mix64(seed ^ (3 * t))), mb = test_mantissa(mix64(seed ^ (3 * t + 1)));
    // the limiter's ratio: |b| in 2^-210 .. 2^210, |a| from 2|b| down 40 (one in four: 700) binades
    double b = ldexp(mb, (int)(h % 420) - 210), q;
    double a = ldexp(ma, ilogb(b) - (int)((h >> 12) % ((h >> 10 & 3) ? 40 : 700)));
    if (h & (1ull << 40)) a = -a;
    if (h & (1ull << 41)) b = -b;
    if (fabs(a) < 2.0 * fabs(b)) {
      if (quot_rn(a, b, &q)) c[0] += __double_as_longlong(q) != __double_as_longlong(a / b);
      else c[2]++;
    }
    // the back substitution's: a pivot in 1 .. 2^8, a dividend down to the subnormals
    b = ldexp(mb, (int)(h >> 24 & 7));
    a = ldexp(ma, (h >> 30 & 3) ? (int)((h >> 44) % 200) - 100 : -(int)((h >> 44) % 1090));
    if (h & (1ull << 42)) a = -a;
    if (div_rn_3_covers(b) && div_rn_3_takes(a)) {
      const double zh = 1.0 / b, r = fma(-b, zh, 1.0), zl = r / b, zll = fma(-b, zl, r) / b;
      const double v = div_rn_3(a, zh, zl, zll), want = a / b;
      c[1] += __double_as_longlong(v) != __double_as_longlong(want) && !(v == 0.0 && want == 0.0);
    } else {
      c[3]++;
    }
  }
  for (int q = 0; q < 4; q++)
    if (c[q]) atomicAdd(counts + q, c[q]);
}

// The largest |1 - b*rcp_approx(b)| over every leading 20-bit mantissa, the
// lower word zero, all ones or any, at the ends and the middle of quot_rn's
// exponents.
__global__ void k_selftest_estimate(uint64_t seed, unsigned long long *worst) {
  double m = 0.0;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < 9u << 20; t += gridDim.x * blockDim.x) {
    const uint64_t lead = t & 0xfffffu, kind = t >> 20;
    const uint64_t low = kind % 3 == 0 ? 0 : kind % 3 == 1 ? 0xffffffffu : mix64(seed ^ t) & 0xffffffffu;
    const uint64_t e = kind < 3 ? 1023 - 200 : kind < 6 ? 1023 : 1023 + 200;
    const double b = __longlong_as_double((long long)(e << 52 | lead << 32 | low));
    m = fmax(m, fabs(fma(-b, rcp_approx(b), 1.0)));
  }
  atomicMax(worst, (unsigned long long)__double_as_longlong(m));
}

}  // namespace a3g

extern "C" int a3g_selftest_quotients(int device, uint64_t n, uint64_t seed, uint64_t *counts, double *estimate) {
  if (!counts || !estimate) { a3g::set_error("null counts or estimate"); return A3G_ERR_ARG; }
  A3G_CUDA(cudaSetDevice(device));
  unsigned long long *d = nullptr, h[5];
  A3G_CUDA(cudaMalloc((void **)&d, sizeof(h)));
  cudaError_t e = cudaMemset(d, 0, sizeof(h));
  if (e == cudaSuccess) {
    a3g::k_selftest_quotients<<<148 * 8, 256>>>(n, seed, d);
    a3g::k_selftest_estimate<<<148 * 8, 256>>>(seed, d + 4);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return a3g::cuda_fail(e, "a3g_selftest_quotients");
  for (int q = 0; q < 4; q++) counts[q] = h[q];
  std::memcpy(estimate, &h[4], sizeof(double));
  return A3G_OK;
}

extern "C" int a3g_selftest_div(int device, uint64_t n, uint64_t seed, uint64_t *mismatches) {
  if (!mismatches) { a3g::set_error("null mismatches"); return A3G_ERR_ARG; }
  A3G_CUDA(cudaSetDevice(device));
  unsigned long long *d = nullptr;
  A3G_CUDA(cudaMalloc((void **)&d, sizeof(*d)));
  cudaError_t e = cudaMemset(d, 0, sizeof(*d));
  if (e == cudaSuccess) {
    a3g::k_selftest_div<<<148 * 8, 256>>>(n, seed, d);
    e = cudaGetLastError();
  }
  unsigned long long h = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return a3g::cuda_fail(e, "a3g_selftest_div");
  *mismatches = h;
  return A3G_OK;
}
