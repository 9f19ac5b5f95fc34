// FP64 kernels: compiled with --fmad=false, so that fused multiply-adds are
// those the sources write (mad) and no others.
#define GPUMHD_LAUNCH_IMPL
#include "gpumhd_launch.cuh"

namespace gpumhd {

template struct Launch<double>;
GPUMHD_CONVERSIONS(double)

// The values derive_one reads.
struct DeriveIn {
  double dt, dt_prev, dt_tvd, inv_va2max, vsqr_diff, v_lim, e_lim;
};

// derive_one for both precisions by one warp, one derived value per lane, from
// lane 0's inputs: the step control is a single dependent chain between two
// kernels of every step, latency-bound (the derived values' ~40 FP64 divisions
// and the reloads of Dyn between its stores).  Same expressions and types as
// derive_one, so the same bits.
__device__ __forceinline__ void derive_lanes(const Consts& c, Dyn* dyn, DeriveIn d) {
  constexpr int NQ = sizeof(DynR<double>) / sizeof(double);  // fields in declaration order
  static_assert(NQ == 25 && sizeof(DynR<float>) == NQ * sizeof(float), "one lane per derived value");
  auto lane0 = [](double& x) { x = __shfl_sync(0xffffffffu, x, 0); };
  lane0(d.dt); lane0(d.dt_prev); lane0(d.dt_tvd); lane0(d.inv_va2max); lane0(d.vsqr_diff); lane0(d.v_lim); lane0(d.e_lim);
  const int l = threadIdx.x;
  if (l >= NQ) return;
  // num / den, or num alone
  double num = 0.0, den = 1.0;
  if (l == 0) num = d.dt_tvd;
  else if (l < 4) { num = 0.975 * c.dx[l - 1]; den = d.dt_tvd; }
  else if (l < 7) num = 0.5 * c.idx[l - 4];
  else if (l == 7) num = d.inv_va2max;
  else if (l == 8) num = d.vsqr_diff;
  else if (l == 9) num = d.v_lim > 0.0 ? d.v_lim : c.tchk_vmax;
  else if (l == 10) num = d.e_lim > 0.0 ? d.e_lim : c.tchk_eps_max;
  else if (l == 11) num = d.v_lim * 0.95;
  else if (l == 12) num = d.e_lim * 0.95;
  else if (l == 13) num = 0.0;
  else if (l < 18) { num = d.dt; den = (double)(18 - l); }  // wdt[st] = dt / (5 - st) at lane 13 + st
  else if (l == 18) { num = c.rt_cfl; den = d.dt; }
  else {  // Spitzer relaxation caps: speed, diffusivity, hyperdiffusion; [0] the previous dt, [1] this one
    const int kind = (l - 19) >> 1;
    const double dth = ((l - 19) & 1) ? d.dt : d.dt_prev;
    num = kind == 0 ? c.spt_cfl_dx : (kind == 1 ? 0.25 : 0.02);
    den = dth;
    if (!(dth > 0.0)) {
      num = kind == 0 ? 0.0 : num * 0.0;
      den = kind == 0 ? 1.0 : c.spt_cfl_dx;
    }
  }
  const double v = num / den;
  reinterpret_cast<float*>(&dyn->rf)[l] = (float)v;
  reinterpret_cast<double*>(&dyn->rd)[l] = v;
}

__device__ __forceinline__ bool step_begin(const Consts& c, Dyn* dyn, double* dt_hist, int dt_hist_cap, DeriveIn& o);

__global__ void k_step_begin(Consts c, Dyn* dyn, double* dt_hist, int dt_hist_cap, cudaGraphConditionalHandle tvd2,
                             int use_cond) {
  int ok = 0;
  DeriveIn d{};
  if (threadIdx.x == 0) {
    ok = step_begin(c, dyn, dt_hist, dt_hist_cap, d) ? 1 : 0;
    if (use_cond) {  // the captured step's second TVD half pass runs only when this step takes it
      const bool take = ok && d.dt_tvd != d.dt;  // a half pass: dt_tvd = 0.5 * dt
      if (take) dyn->cond_launches += 3ULL;
      cudaGraphSetConditional(tvd2, take ? 1u : 0u);
    }
  }
  if (__shfl_sync(0xffffffffu, ok, 0)) derive_lanes(c, dyn, d);
}

// Adjust_Valf_Max with adaptive limits (src/Adjust_Valf_Max.C:92-144) from the
// maxima and near-limit counts the previous pass reduced over the step's
// stage-1 state: the first call takes v_lim and e_lim from the maxima, later
// calls scale them by 1.04 / 1.01 / 0.99 from the counts; va_max follows the
// velocity and sound-speed maxima and decays by at most 1 % per call.  The
// function statics of the reference (ini_flag, va_max_old) live in Dyn.
// Where the reference squares with pow(x, 2.0), this squares with one
// multiplication: the correctly rounded square, which glibc's pow misses by
// one ulp for about 0.1 % of arguments.
__device__ __forceinline__ void step_limits(const Consts& c, Dyn* dyn) {
  const double g0 = __longlong_as_double((long long)dyn->stat_max_bits[0]);
  const double g1 = sqrt(__longlong_as_double((long long)dyn->stat_max_bits[1]));
  const double g2 = __longlong_as_double((long long)dyn->stat_max_bits[2]);
  const double n0 = (double)dyn->stat_cnt[0], n1 = (double)dyn->stat_cnt[1];
  const double cs_fac = 2.0, vv_fac = 3.0, eps_decay = 0.99, mf = c.max_fill;
  double v_lim = dyn->v_lim, e_lim = dyn->e_lim;
  if (dyn->va_ini_flag) {
    v_lim = fmin(g0, c.tchk_vmax);
    e_lim = fmin(g2, c.tchk_eps_max);
    dyn->va_max_old = 0.0;
    dyn->va_ini_flag = 0;
  } else {
    if (n0 >= 4 * mf) v_lim *= 1.04;
    else if (n0 >= mf) v_lim *= 1.01;
    else if (n0 < 0.5 * mf) v_lim *= 0.99;
    if (n1 >= 4 * mf) e_lim *= 1.04;
    else if (n1 >= mf) e_lim *= 1.01;
    else if (n1 < 0.5 * mf) e_lim *= 0.99;
  }
  double va_max = fmax(c.va_max, c.va_adjust * vv_fac * g0);
  va_max = fmax(va_max, c.va_adjust * cs_fac * g1);
  va_max = fmax(va_max, dyn->va_max_old * eps_decay);
  v_lim = fmax(v_lim, c.va_max / vv_fac);
  v_lim = fmin(v_lim, c.tchk_vmax);
  const double ef = c.va_max / cs_fac;
  e_lim = fmax(e_lim, ef * ef);
  e_lim = fmin(e_lim, c.tchk_eps_max);
  dyn->v_lim = v_lim;
  dyn->e_lim = e_lim;
  dyn->inv_va2max = 1.0 / (va_max * va_max);
  dyn->va_max_old = va_max;
  // TVDlimit's velocity cap (src/tvdlimit_SR.C:194-197); with vmax_lim >= 1
  // it does not depend on v_lim and keeps the host's value
  if (c.vmax_lim < 1.0) {
    const double vl = c.vmax_lim * v_lim;
    dyn->vsqr_diff = vl * vl;
  }
  dyn->cmax_bits = 0ULL;  // the CFL pass that follows uses the new inv_va2max
}

// What derive_one reads, from Dyn (lane 0).
__device__ __forceinline__ DeriveIn derive_in(const Dyn* dyn) {
  DeriveIn d{};
  if (threadIdx.x == 0)
    d = DeriveIn{dyn->dt, dyn->dt_prev, dyn->dt_tvd, dyn->inv_va2max, dyn->vsqr_diff, dyn->v_lim, dyn->e_lim};
  return d;
}

__global__ void k_step_limits(Consts c, Dyn* dyn) {
  if (dyn->err) return;
  if (threadIdx.x == 0) step_limits(c, dyn);
  derive_lanes(c, dyn, derive_in(dyn));
}

// Thread 0's part: reads Dyn first, stores at the end; false after an error
// (nothing derived then).
__device__ __forceinline__ bool step_begin(const Consts& c, Dyn* dyn, double* dt_hist, int dt_hist_cap, DeriveIn& o) {
  const int err = dyn->err, done = dyn->steps_done;
  const unsigned long long cmax_bits = dyn->cmax_bits;
  const double dt_old = dyn->dt, time = dyn->time;
  o.inv_va2max = dyn->inv_va2max;
  o.vsqr_diff = dyn->vsqr_diff;
  o.v_lim = dyn->v_lim;
  o.e_lim = dyn->e_lim;
  if (err) return false;
  // Adjust_Valf_Max (src/Adjust_Valf_Max.C:136-142): without va_adjust the
  // limits are the run constants; with it k_step_limits has set them.
  if (!(c.va_adjust > 0.0)) {
    o.v_lim = c.tchk_vmax;
    o.e_lim = c.tchk_eps_max;
    dyn->v_lim = o.v_lim;
    dyn->e_lim = o.e_lim;
  }
  o.dt_prev = dt_old;  // Run.dt as MHD_Residual sees it at stage 1
  dyn->dt_prev = dt_old;
  const double cmax = __longlong_as_double((long long)cmax_bits);
  double dt_mhd = c.dxmin / cmax;
  if (c.has_eta) dt_mhd = smin(dt_mhd, c.dt_res);  // resistive limit (src/mhdres_SR.C:815-819)
  dyn->dt_mhd = dt_mhd;
  // Sync_timestep (src/solver.C:487-548) on one rank
  double r0 = c.dt_rad, r1 = dt_mhd;
  if (bad_pos(r0)) { dyn->err = ERR_BAD_DT_RAD; return false; }
  if (bad_pos(r1)) { dyn->err = ERR_BAD_DT_MHD; return false; }
  const double dt_min_rt = c.rt_tstep * c.CFL * r1;
  if (r0 < dt_min_rt) r0 = smax(r0, dt_min_rt);
  const double dt_min = smin(r0, r1);
  double dt = smin(r0, c.CFL * r1);
  if (c.outcad > 0) {
    const double num = time / c.outcad;
    const int ce = cvt_x86(num);
    const double rem = (num == (double)ce) ? 0.0 : (ce + 1) * c.outcad - time;
    if (rem > 0.0) dt = smin(dt, rem);
  }
  o.dt = c.autostep ? dt : dt_old;
  if (c.autostep) dyn->dt = dt;
  const double cfl = o.dt / dt_min;
  dyn->cfl = cfl;
  if (cfl >= 2.) { dyn->err = ERR_CFL; return false; }
  // TVD branch (src/solver.C:325-339)
  const int two_half = (cfl <= c.CFL_tvd) ? 0 : 1;
  o.dt_tvd = two_half ? 0.5 * o.dt : o.dt;
  dyn->two_half = two_half;
  dyn->dt_tvd = o.dt_tvd;
  if (dt_hist && done >= 0 && done < dt_hist_cap) dt_hist[done] = o.dt;
  dyn->steps_done = done + 1;
  dyn->time = time + o.dt;
  // the last TVD pass of this step accumulates the next step's values
  dyn->cmax_bits = 0ULL;
  dyn->stat_max_bits[0] = dyn->stat_max_bits[1] = dyn->stat_max_bits[2] = 0ULL;
  dyn->stat_cnt[0] = dyn->stat_cnt[1] = 0ULL;
  return true;
}

}  // namespace gpumhd

namespace gpumhd {

// Loop control of the ensemble's while-graph: one tick per step.
__global__ void k_loop_tick(int* counter, cudaGraphConditionalHandle h) {
  if (threadIdx.x == 0) {
    const int left = --(*counter);
    cudaGraphSetConditional(h, left > 0 ? 1u : 0u);
  }
}

__global__ void k_set_counter(int* counter, int n) {
  if (threadIdx.x == 0) *counter = n;
}

__global__ void k_fused_reinit(Consts c, Dyn* dyn, double inv_va2max, double v_lim, double e_lim, double vsqr_diff) {
  if (threadIdx.x == 0) {
    if (!(c.va_adjust > 0.0)) {  // adaptive limits keep their history (the reference's function statics)
      dyn->va_ini_flag = 0;
      dyn->inv_va2max = inv_va2max;
      dyn->v_lim = v_lim;
      dyn->e_lim = e_lim;
      dyn->vsqr_diff = vsqr_diff;
    }
    dyn->err = 0;
    dyn->cmax_bits = 0ULL;
    dyn->stat_max_bits[0] = dyn->stat_max_bits[1] = dyn->stat_max_bits[2] = 0ULL;
    dyn->stat_cnt[0] = dyn->stat_cnt[1] = 0ULL;
  }
  derive_lanes(c, dyn, derive_in(dyn));
}

__global__ void k_divb_begin(Dyn* dyn) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (dyn->err) return;
  dyn->divb_iters = dyn->divb_next;
  dyn->divb_err_bits[0] = 0ULL;
  dyn->divb_err_bits[1] = 0ULL;
}

// Clean_divB: error ratio and the next call's iteration count (src/clean_divB.C:335-354).
__global__ void k_divb_end(Consts c, Dyn* dyn) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (dyn->err) return;
  const int n = dyn->divb_iters;
  const double e0 = __longlong_as_double((long long)dyn->divb_err_bits[0]) * c.divb_err_unit;
  const double e1 = __longlong_as_double((long long)dyn->divb_err_bits[1]) * c.divb_err_unit;
  const double err = e1 / e0;
  int next = n;
  if (err > c.divb_err) next += 1;
  else next -= 1;
  next = min(next, c.divb_itmax);
  next = max(1, next);
  dyn->divb_next = next;
  dyn->divb_last = n;
  dyn->divb_err0 = e0;
  dyn->divb_err1 = e1;
}


__global__ void k_bc_setup(Consts c, Dyn* dyn, const double* __restrict__ part, int nb) {
  if (dyn->err) return;
  __shared__ double sh[BND_NQ][BND_SETUP_THREADS];
  const int tid = threadIdx.x;
  double t[BND_NQ];
  for (int q = 0; q < BND_NQ; q++) t[q] = 0.0;
  for (int k = tid; k < nb; k += BND_SETUP_THREADS)
    for (int q = 0; q < BND_NQ; q++) t[q] += part[(long long)k * BND_NQ + q];
  for (int q = 0; q < BND_NQ; q++) sh[q][tid] = t[q];
  __syncthreads();
  for (int st = BND_SETUP_THREADS / 2; st > 0; st >>= 1) {
    if (tid < st)
      for (int q = 0; q < BND_NQ; q++) sh[q][tid] += sh[q][tid + st];
    __syncthreads();
  }
  if (tid != 0) return;
  for (int q = 0; q < BND_NQ; q++) t[q] = sh[q][0];
  const double n = (double)(c.g.ny * c.g.nz);
  if (dyn->bnd_ini) {
    const double b0 = t[2] / n, b1 = t[3] / n;
    if (dyn->p_bc < 0.0) dyn->p_bc = b0 * sqrt(b0 / b1);
    if (dyn->s_bc < 0.0) dyn->s_bc = (t[4] > 0.0) ? t[5] / t[4] : t[6] / n;
    dyn->bnd_ini = 0;
  }
  const double cn = 1.0 / n;
  dyn->pmean1 = t[0] * cn;
  dyn->pmean2 = t[1] * cn;
}

}  // namespace gpumhd
