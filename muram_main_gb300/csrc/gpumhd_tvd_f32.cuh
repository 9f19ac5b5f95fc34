// FP32 TVD sweeps (TVDlimit, src/tvdlimit_SR.C:199-695) for log-density runs.
//
// The FP32 sweeps are bound by instruction issue (792 instructions per cell in
// a y or z sweep, 973 in x, at 75 % issue), so this is the arithmetic of
// tvd_cell / tvd_slope / tvd_flux / tvd_update written for few instructions:
//
//  * sums and products of the eight variables in pairs (f32x2), minima and
//    maxima of three arguments in one instruction;
//  * the logarithms of density and energy enter only as differences across an
//    interface and in the interface's mean: ln(b/a) = 2 atanh((b-a)/(b+a)), a short
//    series, and exp(mean of logs + slopes) = a exp((ln(b/a) + slopes) / 2), so no
//    log of a cell is formed and nothing is lost to its size (ln rho ~ -15);
//  * an interface's differences serve the slopes of both its cells and its flux;
//  * the flux's ratio r = sl_lim / sl comes from one approximate reciprocal per
//    variable, and its clamp to [0, 1] gives the limited difference;
//  * the boundary-profile mixing of the diffusivities is linear in the cell's
//    Boris / density factor: two coefficients per quantity, fixed along y and z.
//
// Measured against those, 128 x 384 x 384: x 0.603 -> 0.386 ms, y 0.488 -> 0.368, z
// 0.477 -> 0.358 (3.3 to 3.6 TB/s; 17 words per cell); y 520 instructions per cell
// at 56 % issue before the window's registers rotated by unrolling two cells
// (0.461 ms) and the arrays had their own base pointers.  Blocks per SM (FP32,
// compensated): pencil 4, 3 (y 0.368, 0.288 ms at 128 x 256 x 256; 3 and 5: 0.415,
// 0.69; compensated with 4 spills: 0.39); x 5, 6 (with 6: 0.395; without the
// prefetch of the next pencil 0.446).
//
// DIAG adds an output step's diagnostics (src/tvdlimit_SR.C:577-667) to the same
// arithmetic, so that asking for them leaves the state's bits alone.
//
// k_tvd_sweep<float> and k_tvd_sweep_xlanes<float> stay for runs without the
// logarithm (rho_log = 0).
#pragma once

namespace gpumhd {
namespace tvdf {

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// One instruction each, within 1 ulp (rcp) and 2 ulp (2^x, x near 0), or 2^-23
// relative (sqrt); subnormal arguments count as zero, which here are densities
// and squares far below anything the floors let pass.
__device__ __forceinline__ float rcp(float a) { return f_rcp(a); }
__device__ __forceinline__ float sqrt_(float a) { return f_sqrt(a); }
__device__ __forceinline__ float exp2_(float a) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}

// The eight state arrays and the pressure at a byte offset (see at()).
__device__ __forceinline__ void load9(const float* __restrict__ U, const float* __restrict__ P, long long N, unsigned off,
                                      Raw9<float>& r) {
#pragma unroll
  for (int v = 0; v < NV; v++) r.v[v] = *at(U + v * N, off);
  r.v[8] = *at(P, off);
}
__device__ __forceinline__ void load8(const float* __restrict__ U, long long N, unsigned off, float* u) {
#pragma unroll
  for (int v = 0; v < NV; v++) u[v] = *at(U + v * N, off);
}
__device__ __forceinline__ void store8(float* __restrict__ U, long long N, unsigned off, const float* u) {
#pragma unroll
  for (int v = 0; v < NV; v++) *at(U + v * N, off) = u[v];
}

// Coefficients (at factor rf = 0 and per rf) of the slope factor, the energy /
// density, velocity and field diffusivities at a vertical position, and the
// heating profile there.
struct Prof {
  float c0, c1, e0, e1, v0, v1, b0, b1, qt;
};
__device__ __forceinline__ Prof prof_of(const KC<float>& k, int xi) {
  const float hb = k.hfb[xi], ht = k.hft[xi], hh = 1.0f - hb - ht;
  const float h0 = hb * k.tvd_h[0], h1 = k.tvd_h[1], h2 = k.tvd_h[2], h3 = ht * k.tvd_h[3];
  Prof p;
  p.c0 = hb * k.tvd_cs[0] + k.tvd_cs[2] * hh + ht * k.tvd_cs[3];
  p.c1 = (k.tvd_cs[1] - k.tvd_cs[2]) * hh;
  p.e0 = h0 + h2 * hh + h3;
  p.e1 = (h1 - h2) * hh;
  p.v0 = h0 + h2 * k.pm_v * hh + h3 * k.pm_v;
  p.v1 = (h1 - h2 * k.pm_v) * hh;
  p.b0 = h0 + h2 * k.pm_B * hh + h3 * k.pm_B;
  p.b1 = (h1 - h2 * k.pm_B) * hh;
  p.qt = k.qft[xi];
  return p;
}

// A cell: rho, v, energy per mass, B in pairs, and its TVD quantities.
struct Cell {
  float2 q[4];  // (rho, v1) (v2, v3) (e, B1) (B2, B3)
  float he, hv, hB, cm, BC2, bsqr, vsqr, hd, qt;
};

// Scalars of a sweep; the time step is folded into the fluxes.
struct Sweep {
  float dtt, cmax_t, fac0, inv_va2max, vsqr_diff;
  bool hyper;
};

// tvd_cell (src/tvdlimit_SR.C:269-377)
__device__ __forceinline__ void cell_of(const KC<float>& k, const Raw9<float>& r, const Prof& p, const Sweep& s, Cell& t) {
  const float d = fmaxf(k.rho_min, r.v[0]);
  const float dn = rcp(d);
  const float v1 = r.v[1] * dn, v2 = r.v[2] * dn, v3 = r.v[3] * dn;
  const float vv = v1 * v1 + v2 * v2 + v3 * v3;
  const float bb = r.v[5] * r.v[5] + r.v[6] * r.v[6] + r.v[7] * r.v[7];
  t.q[0] = f2(d, v1);
  t.q[1] = f2(v2, v3);
  t.q[2] = f2(r.v[4] * dn - 0.5f * vv, r.v[5]);
  t.q[3] = f2(r.v[6], r.v[7]);
  t.vsqr = vv;
  t.bsqr = bb;
  t.qt = p.qt;
  const float va2 = bb * dn;
  const float x2 = va2 * s.inv_va2max, sx = 1.0f + x2;
  const float lf = sx * rcp(sx + x2 * x2);
  float cs2 = (float)(5.0 / 3.0) * r.v[8] * dn;
  const float vabs = sqrt_(vv);
  const float dd = d * d;
  const float rf = fminf(lf, dd * rcp(dd + k.rho_lev));
  float cf = fmaf(rf, p.c1, p.c0);
  t.he = fmaf(rf, p.e1, p.e0);
  t.hv = fmaf(rf, p.v1, p.v0);
  t.hB = fmaf(rf, p.b1, p.b0);
  float CME = 0.0f;
  if (k.CZ != 1.0f) {  // Mach-number damping above the photosphere, not of the field's diffusivity
    CME = (1.0f - k.CZ) * ((float)(vabs >= k.CME_thresh * sqrt_(va2 + cs2)));
    t.he *= 1.0f - CME;
    t.hv *= 1.0f - CME;
  }
  cf = fmaxf(cf, CME);
  cs2 *= cf * cf;
  t.cm = vabs + sqrt_(fmaxf(cs2, lf * (cs2 + va2)));
  t.BC2 = 1.0f - lf;
  t.hd = 0.0f;
  if (s.hyper) t.hd = s.fac0 * fmaxf(0.0f, fminf(k.vhyp * vabs, s.cmax_t - t.cm));
}

// Differences across the interface of cells a | b: ln(rho), v, ln(e), B.
// |z| <= 0.2 in the series 2 (z + z^3/3 + ...): next term below 2e-8 relative;
// other jumps, and arguments the logarithm refuses, go through logf.
__device__ __forceinline__ void diff(const Cell& a, const Cell& b, float2 d[4]) {
#pragma unroll
  for (int p = 0; p < 4; p++) d[p] = sub(b.q[p], a.q[p]);
  const float2 sm = f2(a.q[0].x + b.q[0].x, a.q[2].x + b.q[2].x), df = f2(d[0].x, d[2].x);
  if (fabsf(df.x) <= 0.2f * sm.x && fabsf(df.y) <= 0.2f * sm.y) {
    const float2 z = mul(df, f2(rcp(sm.x), rcp(sm.y)));
    const float2 w = mul(z, z);
    float2 q = fma2(w, f2(2.0f / 9.0f), f2(2.0f / 7.0f));
    q = fma2(w, q, f2(2.0f / 5.0f));
    q = fma2(w, q, f2(2.0f / 3.0f));
    q = fma2(w, q, f2(2.0f));
    q = mul(q, z);
    d[0].x = q.x;
    d[2].x = q.y;
  } else {
    d[0].x = logf(b.q[0].x) - logf(a.q[0].x);
    d[2].x = logf(b.q[2].x) - logf(a.q[2].x);
  }
}

// tvd_slope (src/tvdlimit_SR.C:388-434) from the differences at the cell's left
// (l) and right (r) interfaces: the one of smallest size among l, r and their
// mean's half where l and r agree in sign, else 0.
__device__ __forceinline__ float limited(float l, float r, float m) {
  return fmaxf(min3(l, r, m), fminf(0.0f, max3(l, r, m)));
}
__device__ __forceinline__ void slope(const KC<float>& k, const float2 l[4], const float2 r[4], float vsqr, float vsqr_diff,
                                      int xi, float2 s[4]) {
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const float2 m = mul(add(l[p], r[p]), f2(0.25f));
    s[p].x = limited(l[p].x, r[p].x, m.x);
    s[p].y = limited(l[p].y, r[p].y, m.y);
  }
  if (k.has_visc_slope) {
    const float cf = (1.0f - k.visc_slope_bot * k.hfb[xi]) * (1.0f - k.visc_slope_top * k.hft[xi]);
    s[0].y *= cf; s[1].x *= cf; s[1].y *= cf;
  }
  if (k.has_eta_slope) {
    const float cf = (1.0f - k.eta_slope_bot * k.hfb[xi]) * (1.0f - k.eta_slope_top * k.hft[xi]);
    s[2].y *= cf; s[3].x *= cf; s[3].y *= cf;
  }
  if (fabsf(r[0].x) > k.q_rho_max) s[0].x = 0.0f;
  if (k.has_vmax_lim && vsqr > vsqr_diff) { s[0].y = 0.0f; s[1].x = 0.0f; s[1].y = 0.0f; }
}

// Limited diffusive difference of a pair (src/tvdlimit_SR.C:436-470):
// max(0, 1 + h (r - 1)) times l clamped between 0 and d, with l = d - slopes and
// r = l / d; below the reference's floor |d| < 1e-30 both vanish with d.
__device__ __forceinline__ float2 limited_diff(float2 d, float2 sa, float2 sb, float2 h) {
  const float2 l = sub(d, add(sa, sb));
  const float2 rc = f2(rcp(fmaxf(fabsf(d.x), 1e-30f)), rcp(fmaxf(fabsf(d.y), 1e-30f)));
  const float2 r = mul(mul(l, rc), mul(d, rc));
  float2 g = fma2(h, r, sub(f2(1.0f), h));
  g = f2(fmaxf(0.0f, g.x), fmaxf(0.0f, g.y));
  return mul(mul(g, f2(__saturatef(r.x), __saturatef(r.y))), d);
}

// tvd_flux (src/tvdlimit_SR.C:436-563), times dtt, between cells a (index ia,
// vertical index xi) and b; dm, dp: the density, velocity and energy differences
// of the interfaces left of a and right of b (hyperdiffusion).  DIAG: qvis
// receives the viscous heating at the interface.
template <int DIR, bool DIAG = false>
__device__ __forceinline__ void flux(const Consts& c, const KC<float>& k, const Cell& a, float b_cm, float b_hd,
                                     const float2 d[4], const float2 sa[4], const float2 sb[4], const float* dm,
                                     const float* dp, int ia, int xi, int sz, int istart, const Sweep& s, float2 F[4],
                                     float& qres, float* qvis = nullptr) {
  F[0] = limited_diff(d[0], sa[0], sb[0], f2(a.he, a.hv));
  F[1] = limited_diff(d[1], sa[1], sb[1], f2(a.hv, a.hv));
  F[2] = limited_diff(d[2], sa[2], sb[2], f2(a.he, a.hB));
  F[3] = limited_diff(d[3], sa[3], sb[3], f2(a.hB, a.hB));
  const float2 fac = f2(s.dtt * s.fac0 * fminf(s.cmax_t, fmaxf(a.cm, b_cm)));
#pragma unroll
  for (int p = 0; p < 4; p++) F[p] = mul(F[p], fac);
  if (DIR == 0) F[2].y *= k.B_par_diff;
  else if (DIR == 1) F[3].x *= k.B_par_diff;
  else F[3].y *= k.B_par_diff;
  if (c.need_coeff) {
    const float hb = k.hfb[xi], ht = k.hft[xi];
    F[0].x *= k.tvd_coeff[0];
    float cf = fmaxf(k.tvd_coeff[1], k.visc_coeff_bot * hb + k.visc_coeff_top * ht);
    F[0].y *= cf; F[1].x *= cf; F[1].y *= cf;
    F[2].x *= k.tvd_coeff[2];
    cf = fmaxf(k.tvd_coeff[3], k.eta_coeff_bot * hb + k.eta_coeff_top * ht);
    F[2].y *= cf; F[3].x *= cf; F[3].y *= cf;
  }
  if (DIR == 0 && s.hyper && ia >= istart) {
    // 0.125 (bp - am) - 0.375 (b - a)
    const float dn = s.dtt * fmaxf(a.hd, b_hd);
    F[0].x -= dn * (0.125f * (dm[0] + dp[0]) - 0.25f * d[0].x);
    F[0].y -= dn * (0.125f * (dm[1] + dp[1]) - 0.25f * d[0].y);
    F[2].x -= dn * (0.125f * (dm[2] + dp[2]) - 0.25f * d[2].x);
  }
  // interface values: a exp((d + sa - sb) / 2) for rho and e, a + (d + sa - sb) / 2 for v
  const float2 t0 = add(d[0], sub(sa[0], sb[0])), t1 = add(d[1], sub(sa[1], sb[1]));
  const float t4 = d[2].x + (sa[2].x - sb[2].x);
  const float2 u23 = fma2(t1, f2(0.5f), a.q[1]);
  const float u1 = fmaf(t0.y, 0.5f, a.q[0].y);
  const float u0 = a.q[0].x * exp2_(0.72134752f * t0.x), u4 = a.q[2].x * exp2_(0.72134752f * t4);
  const float f0 = F[0].x * u0;
  const float mc = f0 * k.CZ;
  const float2 f23 = fma2(u23, f2(mc), mul(F[1], f2(u0)));
  const float f1 = fmaf(u1, mc, F[0].y * u0);
  float f4 = F[2].x * u4 * u0;
  f4 += u4 * mc + a.qt * (u1 * f1 + u23.x * f23.x + u23.y * f23.y);
  F[0] = f2(f0, f1);
  F[1] = f23;
  F[2].x = f4;
  if (DIR == 0 && !c.g.periodic_x && (ia == sz - GH - 1 || ia == GH - 1)) F[2].y = 0.0f;
  qres = d[2].y * F[2].y + d[3].x * F[3].x + d[3].y * F[3].y;
  if (DIAG) *qvis = d[0].y * F[0].y + d[1].x * F[1].x + d[1].y * F[1].y;
}

// tvd_update (src/tvdlimit_SR.C:565-657); Fp / Fm, qp / qm carry the time step.
// Cin, Cout: the compensated mode's remainders, as in tvd_update.  DIAG: dg, the
// cell's diagnostics (arrays N apart), per unit of the full step's time; qvp, qvm:
// the viscous heating at the cell's interfaces, times dtt.
template <bool DIAG = false>
__device__ __forceinline__ void update(const KC<float>& k, const float2 Fp[4], const float2 Fm[4], float qp, float qm,
                                       const Cell& c0, const float* u_in, float* u, const Rem<float>* Cin,
                                       Rem<float>* Cout, long long N, float* dg = nullptr, float idt = 0.0f,
                                       float qvp = 0.0f, float qvm = 0.0f) {
  float res[NV];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const float2 r = sub(Fp[p], Fm[p]);
    res[2 * p] = r.x;
    res[2 * p + 1] = r.y;
  }
  const float v1 = c0.q[0].y, v2 = c0.q[1].x, v3 = c0.q[1].y, b1 = c0.q[2].y, b2 = c0.q[3].x, b3 = c0.q[3].y;
  if (DIAG) {
    dg[7 * N] += (res[4] + (1.0f - c0.qt) * (res[1] * v1 + res[2] * v2 + res[3] * v3)) * idt;
    dg[8 * N] += 0.5f * (qp + qm) * c0.qt * idt;
    dg[9 * N] += 0.5f * (qvp + qvm) * c0.qt * idt;
  }
  res[4] += (1.0f - c0.qt) * (res[1] * v1 + res[2] * v2 + res[3] * v3) + 0.5f * (qp + qm) * c0.qt;
  const float dn = (res[1] * b1 + res[2] * b2 + res[3] * b3) * rcp(fmaxf(1e-30f, c0.bsqr));
  const float g1 = c0.BC2 * (dn * b1 - res[1]), g2 = c0.BC2 * (dn * b2 - res[2]), g3 = c0.BC2 * (dn * b3 - res[3]);
  res[1] += g1;
  res[2] += g2;
  res[3] += g3;
  if (DIAG) dg[5 * N] += (g1 * v1 + g2 * v2 + g3 * v3) * idt;
  res[4] += g1 * v1 + g2 * v2 + g3 * v3;
  float rem[NV];
  if (Cin) {
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const float y = res[v] + rem_ld<float>(Cin + (long long)v * N);
      u[v] = u_in[v] + y;
      rem[v] = y - (u[v] - u_in[v]);
    }
  } else {
#pragma unroll
    for (int v = 0; v < NV; v++) u[v] = u_in[v] + res[v];
  }
  const float d0 = u[0], e0 = u[4];
  u[0] = fmaxf(k.rho_min, d0);
  u[4] = fmaxf(e0, k.eps_min * u[0] + 0.5f * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) * rcp(u[0]));
  if (DIAG) dg[6 * N] += (u[4] - e0) * idt;
  if (Cin && Cout) {
    if (u[0] != d0) rem[0] = 0.0f;
    if (u[4] != e0) rem[4] = 0.0f;
#pragma unroll
    for (int v = 0; v < NV; v++) rem_st<float>(Cout + (long long)v * N, rem[v]);
  }
}

__device__ __forceinline__ Sweep sweep_of(const DynR<float>& dr, const KC<float>& k, int dir) {
  return Sweep{dr.dt_tvd, dr.cmax_t[dir], dr.fac0[dir], dr.inv_va2max, dr.vsqr_diff, dir == 0 && k.has_vhyp};
}

}  // namespace tvdf

// Sweep along y (DIR 1) or z (DIR 2): one thread per pencil chunk, marching with
// a window of cells; the next cell's stored values are loaded a step ahead.
template <int DIR, bool COMP, bool DIAG = false>
__global__ void __launch_bounds__(128, COMP || DIAG ? 3 : 4) k_tvd_pencil_f32(Consts c, const float* __restrict__ Uin,
                                                           const float* __restrict__ Pst, float* __restrict__ Uout,
                                                           Dyn* __restrict__ dyn, TvdArgs ta,
                                                           const Rem<float>* Ci, Rem<float>* Co, TvdDiag<float> dg) {
  using namespace tvdf;
  if (dyn->err) return;
  if (ta.only_two_half && !dyn->two_half) return;  // second half pass not taken this step
  const Geom& g = c.g;
  const KC<float>& k = c.kf;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned nch = (unsigned)((ta.n1 + ta.td - 1) / ta.td);
  if (t >= (unsigned)ta.na * (unsigned)ta.nb * nch) return;
  const unsigned r = t / (unsigned)ta.na, ch = r / (unsigned)ta.nb;
  const int aa = ta.a0 + (int)(t - r * (unsigned)ta.na), bb = ta.b0 + (int)(r - ch * (unsigned)ta.nb);
  const int p0 = GH + (int)ch * ta.td, p1 = min(p0 + ta.td, GH + ta.n1);
  const unsigned sd = (unsigned)ta.sd * 4u;  // bytes
  const unsigned base = ((unsigned)aa * (unsigned)ta.sa + (unsigned)bb * (unsigned)ta.sb) * 4u;
  const long long N = g.N;
  const Sweep s = sweep_of(dyn->rf, k, DIR);
  // after the first of two half passes the z sweep also writes the periodic
  // images (the exchange between the halves); otherwise the interior only
  const bool half_images = (ta.mode == 1) && dyn->two_half;
  const Prof pr = prof_of(k, aa);
  Cell c0, c1;
  float2 d0[4], s0[4], F0[4];
  float q0, qv0 = 0.0f;  // qv: viscous heating, for the diagnostics
  Raw9<float> nxt;
  unsigned off = base + (unsigned)p0 * sd;
  {
    Cell ca, cb;
    float2 da[4], db[4], sm[4];
    Raw9<float> ra, rb, rc;
    load9(Uin, Pst, N, off - 2u * sd, ra);
    load9(Uin, Pst, N, off - sd, rb);
    load9(Uin, Pst, N, off, rc);
    load9(Uin, Pst, N, off + sd, nxt);
    cell_of(k, ra, pr, s, ca);
    cell_of(k, rb, pr, s, cb);
    diff(ca, cb, da);
    cell_of(k, rc, pr, s, c0);
    diff(cb, c0, db);
    slope(k, da, db, cb.vsqr, s.vsqr_diff, aa, sm);
    cell_of(k, nxt, pr, s, c1);
    load9(Uin, Pst, N, off + 2u * sd, nxt);
    diff(c0, c1, d0);
    slope(k, db, d0, c0.vsqr, s.vsqr_diff, aa, s0);
    flux<DIR, DIAG>(c, k, cb, c0.cm, 0.0f, db, sm, s0, nullptr, nullptr, p0 - 1, aa, 0, 0, s, F0, q0, &qv0);
  }
  // one cell: window a | b | n (n read from nxt), interface a | b with differences
  // da and slopes sa, sb; the values a later cell needs go to n, dn, sb, F, q
  auto step = [&](int pos, const Cell& a, const Cell& b, Cell& n, const float2* da, float2* db, const float2* sa,
                  float2* sb, const float2* Fm, float2* F, float qm, float& q, float qvm, float& qv) {
    float uc[NV], u[NV];
    load8(Uin, N, off, uc);
    cell_of(k, nxt, pr, s, n);
    if (pos + 1 < p1) load9(Uin, Pst, N, off + 3u * sd, nxt);
    diff(b, n, db);
    slope(k, da, db, b.vsqr, s.vsqr_diff, aa, sb);
    flux<DIR, DIAG>(c, k, a, b.cm, 0.0f, da, sa, sb, nullptr, nullptr, pos, aa, 0, 0, s, F, q, &qv);
    const int cj = DIR == 1 ? pos : bb, ck = DIR == 2 ? pos : bb;
    const Rem<float>* cin = nullptr;
    Rem<float>* cout = nullptr;
    if (COMP) {  // the remainders of the interior cell this one is or images
      const int sj = wrap_interior(cj, g.ny), sk = wrap_interior(ck, g.nz);
      cin = Ci + cidx32(g, aa, sj, sk);
      if (sj == cj && sk == ck) cout = Co + cidx32(g, aa, cj, ck);
    }
    update<DIAG>(k, F, Fm, q, qm, a, uc, u, cin, cout, N, DIAG ? dg.d + off / 4u : nullptr, dg.idt_full, qv, qvm);
    if (!half_images) store8(Uout, N, off, u);
    else store_state<float, true>(g, Uout, aa, cj, ck, images_of(g, aa, cj, ck, false), u);
    off += sd;
  };
  // two cells per turn, so that the window's registers rotate without copies
  for (int pos = p0; pos < p1; pos += 2) {
    Cell c2;
    float2 d1[4], s1[4], F1[4];
    float q1, qv1 = 0.0f;
    step(pos, c0, c1, c2, d0, d1, s0, s1, F0, F1, q0, q1, qv0, qv1);
    if (pos + 1 >= p1) break;
    step(pos + 1, c1, c2, c0, d1, d0, s1, s0, F1, F0, q1, q0, qv1, qv0);
    c1 = c0;
    c0 = c2;
  }
}

// Sweep along x: 32 consecutive cells of a pencil per warp, one per lane; the
// two lanes at each end are the stencil's halo (28 updates per warp), as in
// k_tvd_sweep_xlanes.
template <bool COMP, bool DIAG = false>
__global__ void __launch_bounds__(128, COMP ? 6 : 5) k_tvd_xlanes_f32(Consts c, const float* __restrict__ Uin,
                                                           const float* __restrict__ Pst, float* __restrict__ Uout,
                                                           Dyn* __restrict__ dyn, int only_two_half,
                                                           const Rem<float>* Ci, Rem<float>* Co, TvdDiag<float> dg) {
  using namespace tvdf;
  if (dyn->err) return;
  if (only_two_half && !dyn->two_half) return;
  const Geom& g = c.g;
  const KC<float>& k = c.kf;
  constexpr int OUT = 28;
  constexpr unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned nseg = (unsigned)((g.nx + OUT - 1) / OUT);
  // each warp keeps its segment and strides over the pencils, so that what
  // depends on x only is formed once
  const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned stride = ((gridDim.x * blockDim.x) >> 5) / nseg, npen = (unsigned)g.sy * (unsigned)g.sz;
  const unsigned seg = warp % nseg, pen0 = warp / nseg;
  if (pen0 >= stride) return;
  const int pos = OUT * (int)seg + lane;   // this lane's cell along x (the first is GH - 2)
  const int posc = min(pos, g.wx - 1);     // clamped for the tail of the last segment
  const bool out = lane >= 2 && lane < 30 && pos < GH + g.nx;
  const Prof pr = prof_of(k, posc);
  const Sweep s = sweep_of(dyn->rf, k, 0);
  const int istart = 1 + (g.periodic_x ? 0 : GH);
  auto dn1 = [&](float2 v) { return f2(__shfl_down_sync(ALL, v.x, 1), __shfl_down_sync(ALL, v.y, 1)); };
  auto up1 = [&](float2 v) { return f2(__shfl_up_sync(ALL, v.x, 1), __shfl_up_sync(ALL, v.y, 1)); };
  // the next pencil's values are loaded during this one's work
  Raw9<float> raw;
  load9(Uin, Pst, g.N, ((unsigned)g.sx * min(pen0, npen - 1) + (unsigned)posc) * 4u, raw);
  for (unsigned pen = pen0; pen < npen; pen += stride) {
    const unsigned base = (unsigned)g.sx * pen;
    Cell c0, cr;
    cell_of(k, raw, pr, s, c0);
    float uin[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) uin[v] = raw.v[v];
    if (pen + stride < npen) load9(Uin, Pst, g.N, ((unsigned)g.sx * (pen + stride) + (unsigned)posc) * 4u, raw);
    // from the right neighbour its values, speed and hyperdiffusivity; lane 31's
    // own values stand in for its missing one (its results are not used)
#pragma unroll
    for (int p = 0; p < 4; p++) cr.q[p] = dn1(c0.q[p]);
    const float r_cm = __shfl_down_sync(ALL, c0.cm, 1);
    float2 dr[4], dl[4], s0[4], s1[4], F[4], Fm[4];
    diff(c0, cr, dr);
#pragma unroll
    for (int p = 0; p < 4; p++) dl[p] = up1(dr[p]);
    slope(k, dl, dr, c0.vsqr, s.vsqr_diff, posc, s0);
#pragma unroll
    for (int p = 0; p < 4; p++) s1[p] = dn1(s0[p]);
    float r_hd = 0.0f, dm[3] = {0.0f, 0.0f, 0.0f}, dp[3] = {0.0f, 0.0f, 0.0f};
    if (s.hyper) {
      r_hd = __shfl_down_sync(ALL, c0.hd, 1);
      dm[0] = dl[0].x; dm[1] = dl[0].y; dm[2] = dl[2].x;
      dp[0] = __shfl_down_sync(ALL, dr[0].x, 1);
      dp[1] = __shfl_down_sync(ALL, dr[0].y, 1);
      dp[2] = __shfl_down_sync(ALL, dr[2].x, 1);
    }
    float q, qv = 0.0f;
    flux<0, DIAG>(c, k, c0, r_cm, r_hd, dr, s0, s1, dm, dp, pos, posc, g.nx + 2 * GH, istart, s, F, q, &qv);
#pragma unroll
    for (int p = 0; p < 4; p++) Fm[p] = up1(F[p]);
    const float qm = __shfl_up_sync(ALL, q, 1);
    const float qvm = DIAG ? __shfl_up_sync(ALL, qv, 1) : 0.0f;
    if (!out) continue;
    const unsigned id = base + (unsigned)pos;
    const Rem<float>* cin = nullptr;
    Rem<float>* cout = nullptr;
    if (COMP) {  // the remainders of the interior cell this one is or images
      const int kz = (int)(pen / (unsigned)g.sy), j = (int)pen - kz * g.sy;
      const int sj = wrap_interior(j, g.ny), sk = wrap_interior(kz, g.nz);
      cin = Ci + cidx32(g, pos, sj, sk);
      if (sj == j && sk == kz) cout = Co + id;
    }
    float u[NV];
    update<DIAG>(k, F, Fm, q, qm, c0, uin, u, cin, cout, g.N, DIAG ? dg.d + id : nullptr, dg.idt_full, qv, qvm);
    store8(Uout, g.N, id * 4u, u);
  }
}

}  // namespace gpumhd
