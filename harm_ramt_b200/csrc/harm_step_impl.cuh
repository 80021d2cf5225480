// Templated kernels of the step, shared by the FP64 translation unit
// (harm_step.cu, built without multiply-add contraction so that it rounds
// as the reference does) and the mixed-precision one (harm_step_mixed.cu,
// built with contraction and fast FP32 division/square root).
#pragma once
#include <cuda_runtime.h>
#include <float.h>
#include "harm_exact.cuh"
#include "harm_kernels.cuh"
#include "harm_smem.h"
#include "harm_tma.cuh"

namespace harm {

// ---------------------------------------------------------------- fluxes
// The interface states (step_ch.c:812-823 slopes and 893-904 interface
// values) of N consecutive zones of one variable, a thread
// walking along the zones (src: the first zone's value, step st; one more
// value on each side is read for MC, two for PARA).  The slopes and, for
// PARA, the raw interface values that neighbouring zones share are formed
// once; put(c, l, r) takes zone c's states.  The values are mc_slope's and
// para4's: 2 min(|a|, |b|) is min(|2 a|, |2 b|), (4 a) b is (2 a)(2 b), and
// the sign of a slope is copied instead of multiplied.
template <typename T>
__device__ __forceinline__ T para_dq_shared(T a, T b, T ym, T yp)
{
  const T s = (T(4.) * a) * b, c = T(0.5) * (yp - ym);
  const T m = T(2.) * rmin(fabs(a), fabs(b));
  return (s <= T(0.)) ? T(0.) : copysign(rmin(fabs(c), m), c);
}
template <typename T, bool PARA, int N, typename Put>
__device__ __forceinline__ void row_states(const double* src, int st, Put put)
{
  T ym = (T)src[-st], y = (T)src[0], a = y - ym;
  if (!PARA) {
#pragma unroll
    for (int c = 0; c < N; c++) {
      const T yp = (T)src[(c + 1) * st], b = yp - y;
      const T h = T(0.5) * minmod(T(0.5) * (yp - ym), minmod(T(2.) * a, T(2.) * b));
      put(c, y - h, y + h);
      ym = y;
      y = yp;
      a = b;
    }
  } else {
    T yp = (T)src[st], b = yp - y;
    const T ymm = (T)src[-2 * st];
    T d0 = para_dq_shared(ym - ymm, a, ymm, y), d = para_dq_shared(a, b, ym, yp);
    T l = para_face(ym, y, d0, d);
#pragma unroll
    for (int c = 0; c < N; c++) {
      const T ypp = (T)src[(c + 2) * st], e = ypp - yp;
      const T d1 = para_dq_shared(b, e, y, ypp);
      const T r = para_face(y, yp, d, d1);
      T lo, ro;
      para_limit(ym, y, yp, l, r, lo, ro);
      put(c, lo, ro);
      ym = y;
      y = yp;
      yp = ypp;
      b = e;
      d = d1;
      l = r;
    }
  }
}

// What face_flux takes from its two states (after the Lorentz limits, rc), by
// the form for any metric: fluxes F_l and F_r, the conserved vectors'
// difference dU, the wavespeeds c (left, then right).  Returns the fail code.
template <typename T, bool FFDE>
__device__ __noinline__ int face_sides_general(const StepArgs& a, long long z, int dir, const T* p_l, const T* p_r, T* F_l,
                                               T* F_r, T* dU, T* c, int rc)
{
  Geo<T> g;
  load_geo32<false>(a, dir == 1 ? FACE1 : FACE2, z, g);
  const T gam = (T)a.pp.gam;
  State<T> q;
  T U_r[NPR];
  state_of(p_l, g, q);
  flux_of<T, FFDE>(p_l, q, dir, g, gam, F_l);
  flux_of<T, FFDE>(p_l, q, 0, g, gam, dU);
  if (!rc) rc = vchar_of(p_l, q, dir, g, gam, c[0], c[1]);
  state_of(p_r, g, q);
  flux_of<T, FFDE>(p_r, q, dir, g, gam, F_r);
  flux_of<T, FFDE>(p_r, q, 0, g, gam, U_r);
  for (int k = 0; k < NPR; k++) dU[k] = U_r[k] - dU[k];
  if (!rc) rc = vchar_of(p_r, q, dir, g, gam, c[2], c[3]);
  return rc;
}

// Flux through one face from its two interface states (the rest of the
// fluxcalc face loop, step_ch.c:944-1065).  The left state is finished
// (state, fluxes, wavespeeds) before the right one starts, and U_r - U_l is
// formed as soon as U_r exists, so only one state is live at a time; the
// values and the order of the fatal checks (both Lorentz limits, then the
// left and the right wavespeeds) are the reference's.
template <typename T, bool FFDE, bool SP = false>
__device__ __forceinline__ void face_flux(const StepArgs& a, int i, int j, int dir, T* p_l, T* p_r, T* Fo,
                                          double& dtij, int rf)
{
  const long long z = a.gr.at(i, j);
  Geo<T> g;
  if constexpr (sizeof(T) == 4) load_geo32<SP>(a, dir == 1 ? FACE1 : FACE2, z, g);
  else load_geo(a, dir == 1 ? FACE1 : FACE2, z, g);
  // B^dir continuity (BDIRCONT, step_ch.c:944-947)
  if (dir == 1) p_l[B1] = p_r[B1] = T(0.5) * (p_l[B1] + p_r[B1]);
  else p_l[B2] = p_r[B2] = T(0.5) * (p_l[B2] + p_r[B2]);
  const T gmax = (T)a.pp.gammamax, gam = (T)a.pp.gam;
  int rc = limit_gamma<T, SP>(gmax, p_l, g);
  if (!rc) rc = limit_gamma<T, SP>(gmax, p_r, g);
  const int rc0 = rc;
  T F_l[NPR], F_r[NPR], dU[NPR];
  T cmax_l, cmin_l, cmax_r, cmin_r;
  bool finite = true;
  {
    State<T> q;
    state_of<T, SP>(p_l, g, q);
    if (SP) finite = fabs(dot4(q.bcon, q.bcov)) <= T(FLT_MAX);
    flux_of<T, FFDE>(p_l, q, dir, g, gam, F_l);
    flux_of<T, FFDE>(p_l, q, 0, g, gam, dU);  // U_l for now
    if (!rc) rc = vchar_of<T, SP>(p_l, q, dir, g, gam, cmax_l, cmin_l);
  }
  {
    State<T> q;
    T U_r[NPR];
    state_of<T, SP>(p_r, g, q);
    if (SP) finite = finite && fabs(dot4(q.bcon, q.bcov)) <= T(FLT_MAX);
    flux_of<T, FFDE>(p_r, q, dir, g, gam, F_r);
    flux_of<T, FFDE>(p_r, q, 0, g, gam, U_r);
#pragma unroll
    for (int k = 0; k < NPR; k++) dU[k] = U_r[k] - dU[k];
    if (!rc) rc = vchar_of<T, SP>(p_r, q, dir, g, gam, cmax_r, cmin_r);
  }
  if constexpr (SP) {
    // where b^2 is finite on both sides so is every value that a product left
    // out would have as its factor; else that product is not a number, and
    // the form that has it decides (the check costs a mixed step of the 512^2
    // torus 1 of 327 us, the dipole 0.4 of 105)
    if (!finite) {
      T l[NPR], r[NPR], fl[NPR], fr[NPR], d[NPR], c[4] = {cmax_l, cmin_l, cmax_r, cmin_r};
#pragma unroll
      for (int k = 0; k < NPR; k++) {
        l[k] = p_l[k];
        r[k] = p_r[k];
      }
      rc = face_sides_general<T, FFDE>(a, z, dir, l, r, fl, fr, d, c, rc0);
#pragma unroll
      for (int k = 0; k < NPR; k++) {
        F_l[k] = fl[k];
        F_r[k] = fr[k];
        dU[k] = d[k];
      }
      cmax_l = c[0];
      cmin_l = c[1];
      cmax_r = c[2];
      cmin_r = c[3];
    }
  }
  if (rc) {
    report_fail(a.sc, a.phase0 + (dir == 1 ? PH_FACE1 : PH_FACE2), rc, zone_order(i, j));
    cmax_l = cmin_l = cmax_r = cmin_r = T(0.);
  }
  // cminmax_calc, step_ch.c:1095-1148
  T lmin = rmin(cmin_l, cmin_r), lmax = rmax(cmax_l, cmax_r);
  lmin = fabs(rmax(T(0.), -lmin));
  lmax = fabs(rmax(T(0.), lmax));
  T cmin = lmin, cmax = lmax, ctop = rmax(lmax, lmin);
  // choose_flux, step_ch.c:703-738: rf is fluxmethod, or with FLUXADJUST
  // (HYDROFLUXADJUSTONLY 1) FLAGREALFLUX of zone (i, j), the face's own
  // zone, for the hydro variables
  if (cmax + cmin != T(0.0)) {
#pragma unroll
    for (int k = 0; k < NPR; k++) {
      const int m = (k < B1) ? rf : a.pp.fluxmethod;
      const T hllfrac = (m == 1) ? T(1.0) : T(0.0), laxffrac = (m == 1) ? T(0.0) : T(1.0);
      Fo[k] = hllfrac * ((cmax * F_l[k] + cmin * F_r[k] - cmax * cmin * dU[k]) / (cmax + cmin)) +
              laxffrac * (T(0.5) * (F_l[k] + F_r[k] - ctop * dU[k]));
    }
  } else {
#pragma unroll
    for (int k = 0; k < NPR; k++) Fo[k] = T(0.5) * (F_l[k] + F_r[k] - ctop * dU[k]);
  }
  // face Courant limit, step_ch.c:1062-1065 (kept in FP64)
  double cm = (double)rmax(cmax, cmin);
  dtij = a.pp.cour * (dir == 1 ? a.pp.dx1 : a.pp.dx2) / cm;
}

// ---- the FP64 face without branches (harm_exact.cuh)
// The functions below evaluate get_state, primtoflux, vchar and the Riemann
// flux (the templates of harm_device.cuh and face_flux above) with the same
// operands in the same order, every quotient and root through `ex`.  While
// ex.ok() holds every value is finite and in range, so sums leave out the
// terms that are a value times an exact zero or an exact zero itself (the
// unit covectors of vchar, the Kronecker delta of mhd_calc_0, the B^dir row).
// Where the templates branch (a Lorentz limit, a wavespeed outside its
// bounds) ex.ok() is false and the face goes through face_flux.

// SP: a metric that couples x2 to nothing else and t not to phi in g^{mu nu}
// (g_{t2} = g_{12} = g_{23} = 0, g^{t2} = g^{t3} = g^{12} = g^{23} = 0 at every
// face and centre: Kerr-Schild on a grid stretched along x1 and x2, flat
// space), found when the geometry is uploaded.  Its sums leave out the terms
// that are a finite value times an exact zero, and those planes are not read:
// k_flux of the 512^2 torus 87 -> 79.5 us, 1024^2 292 -> 268, the 512 x 256
// dipole 40 -> 34.5; k_update 51 and 58 -> 49 and 53, 1024^2 178 -> 160 (the
// faces have since gained checks: 1024^2 270).
constexpr int SP_COV = (1 << 2) | (1 << 5) | (1 << 8), SP_CON = SP_COV | (1 << 3);
template <bool SP>
__device__ __forceinline__ void lower_cov(const double* v, const double* c, double* w)
{
  if (!SP) {
    lower_v(v, c, w);
    return;
  }
  w[0] = c[0] * v[0] + c[1] * v[1] + c[3] * v[3];
  w[1] = c[1] * v[0] + c[4] * v[1] + c[6] * v[3];
  w[2] = c[7] * v[2];
  w[3] = c[3] * v[0] + c[6] * v[1] + c[9] * v[3];
}
template <bool SP>
__device__ __forceinline__ void raise_con(const double* v, const double* g, double* w)
{
  if (!SP) {
    lower_v(v, g, w);
    return;
  }
  w[0] = g[0] * v[0] + g[1] * v[1];
  w[1] = g[1] * v[0] + g[4] * v[1] + g[6] * v[3];
  w[2] = g[7] * v[2];
  w[3] = g[6] * v[1] + g[9] * v[3];
}
// the space part of lower_cov for a vector without a time component
template <bool SP>
__device__ __forceinline__ void lower_space(const double* b, const double* c, double* w)
{
  if (SP) {
    w[0] = c[4] * b[0] + c[6] * b[2];
    w[1] = c[7] * b[1];
    w[2] = c[6] * b[0] + c[9] * b[2];
  } else {
    w[0] = c[4] * b[0] + c[5] * b[1] + c[6] * b[2];
    w[1] = c[5] * b[0] + c[7] * b[1] + c[8] * b[2];
    w[2] = c[6] * b[0] + c[8] * b[1] + c[9] * b[2];
  }
}
// the q^2 of gamma_calc
template <bool SP>
__device__ __forceinline__ double qsq_x(const double* pr, const double* c)
{
  const double d = c[4] * pr[U1] * pr[U1] + c[7] * pr[U2] * pr[U2] + c[9] * pr[U3] * pr[U3];
  if (SP) return d + 2. * (c[6] * pr[U1] * pr[U3]);
  return d + 2. * (c[5] * pr[U1] * pr[U2] + c[6] * pr[U1] * pr[U3] + c[8] * pr[U2] * pr[U3]);
}

// lapse and shift of a location, as ucon_calc_rel4vel forms them
struct LapseX {
  Recip alpha;
  double beta[3];
};
template <bool SP>
__device__ __forceinline__ LapseX lapse_x(Exact& ex, const double* gcon)
{
  LapseX l;
  const double alpha = Exact::quot(1., ex.rcp(ex.sqrt_of(-gcon[0])));
  l.alpha = ex.rcp(alpha);
#pragma unroll
  for (int k = 0; k < (SP ? 1 : 3); k++) {
    l.beta[k] = gcon[1 + k] * alpha * alpha;
    ex.numerator<-600>(l.beta[k]);
  }
  return l;
}

struct StateX : State<double> {
  Recip ut;  // u^t
  double bsq, gamma;
};
// get_state; limit: GAMMAMAX where the caller limits the Lorentz factor first
template <bool SP, typename EX>
__device__ __forceinline__ void state_x(EX& ex, const double* pr, const double* c, const LapseX& l, double limit,
                                        StateX& q)
{
  const double gamma = ex.sqrt_of(1. + qsq_x<SP>(pr, c));
  ex.need(gamma <= limit);
  q.gamma = gamma;
  q.ucon[0] = EX::quot(gamma, l.alpha);
#pragma unroll
  for (int k = 0; k < 3; k++)
    q.ucon[1 + k] = (SP && k > 0) ? pr[U1 + k] : pr[U1 + k] - EX::quot(gamma * l.beta[k], l.alpha);
  lower_cov<SP>(q.ucon, c, q.ucov);
  q.bcon[0] = pr[B1] * q.ucov[1] + pr[B2] * q.ucov[2] + pr[B3] * q.ucov[3];
  q.ut = ex.rcp(q.ucon[0]);
#pragma unroll
  for (int k = 1; k < 4; k++) q.bcon[k] = ex.div(pr[B1 - 1 + k] + q.bcon[0] * q.ucon[k], q.ut);
  lower_cov<SP>(q.bcon, c, q.bcov);
  q.bsq = dot4(q.bcon, q.bcov);
}

// primtoflux in time: the conserved vector
template <bool FFDE>
__device__ __forceinline__ void conserved_x(const double* pr, const StateX& q, double sg, double gam, double* U)
{
  const double r = FFDE ? 0. : pr[RHO], u = FFDE ? 0. : pr[UU], P = (gam - 1.) * u, w = P + r + u;
  const double eta = FFDE ? q.bsq : w + q.bsq, ptot = FFDE ? q.bsq * 0.5 : P + q.bsq * 0.5;
  const double m = pr[RHO] * q.ucon[0], eu = eta * q.ucon[0];
  U[RHO] = m * sg;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    double t = eu * q.ucov[j];
    if (j == 0) t = t + ptot;
    t = t - q.bcon[0] * q.bcov[j];
    if (!FFDE && j == 0) t = t + m;
    U[UU + j] = t * sg;
  }
#pragma unroll
  for (int k = B1; k <= B3; k++) U[k] = pr[k] * sg;
}

// bsq_flag (a tiny b^2's quotients only have to come out below the limits)
__device__ __forceinline__ unsigned char bsq_flag_x(Exact& ex, const StepArgs& a, const double* pr, double bsq)
{
  const double rl = a.pp.bsqorholimit, ul = a.pp.bsqoulimit;
  ex.numerator((fabs(bsq) < 1.e-200 && rl > 1.e-150 && ul > 1.e-150) ? 0. : bsq);
  const double br = Exact::quot(bsq, ex.rcp(pr[RHO])), bu = Exact::quot(bsq, ex.rcp(pr[UU]));
  const int f0 = (br > rl) ? 2 : ((br > 0.9 * rl) ? 1 : 0), f3 = (bu > ul) ? 2 : ((bu > 0.9 * ul) ? 1 : 0);
  return (unsigned char)(f0 | (f3 << 2));
}

// What a face takes from one interface state.  The B^dir row of the flux and
// of the conserved vectors' difference is zero on both sides (B^dir is
// continuous), so two field components are kept: the other one of the plane
// and B3.
constexpr int NX = NPR - 1, XB = B1, XB3 = B1 + 1;
struct SideX {
  double F[NX], U[NX], vmax, vmin;
};

// primtoflux in direction dir (1 or 2) and in time, and vchar; sg: sqrt(-g);
// gd, gdd: g^{t dir} and g^{dir dir}
template <bool FFDE, bool SP, typename EX>
__device__ __forceinline__ void side_x(EX& ex, const double* pr, const StateX& q, int dir, double sg, double gtt,
                                       double gd, double gdd, double gam, SideX& x)
{
  const bool d1 = (dir == 1);
  {
    const double r = FFDE ? 0. : pr[RHO], u = FFDE ? 0. : pr[UU], P = (gam - 1.) * u, w = P + r + u;
    const double eta = FFDE ? q.bsq : w + q.bsq, ptot = FFDE ? q.bsq * 0.5 : P + q.bsq * 0.5;
    const double ud = d1 ? q.ucon[1] : q.ucon[2], bd = d1 ? q.bcon[1] : q.bcon[2];
    const double m = pr[RHO] * ud, eu = eta * ud, m0 = pr[RHO] * q.ucon[0], eu0 = eta * q.ucon[0];
    x.F[RHO] = m * sg;
    x.U[RHO] = m0 * sg;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      double t = eu * q.ucov[j];
      if (j == 1 && d1) t = t + ptot;
      if (j == 2 && !d1) t = t + ptot;
      t = t - bd * q.bcov[j];
      if (!FFDE && j == 0) t = t + m;
      x.F[UU + j] = t * sg;
      t = eu0 * q.ucov[j];
      if (j == 0) t = t + ptot;
      t = t - q.bcon[0] * q.bcov[j];
      if (!FFDE && j == 0) t = t + m0;
      x.U[UU + j] = t * sg;
    }
    const double Bd = d1 ? pr[B1] : pr[B2], Bo = d1 ? pr[B2] : pr[B1], uo = d1 ? q.ucon[2] : q.ucon[1];
    x.F[XB] = ex.div(Bo * ud - Bd * uo, q.ut) * sg;
    x.F[XB3] = ex.div(pr[B3] * ud - Bd * q.ucon[3], q.ut) * sg;
    x.U[XB] = Bo * sg;
    x.U[XB3] = pr[B3] * sg;
  }
  // (a density or internal energy without bound can leave the wavespeeds in
  // range -- where the sum below is not positive -- and the fluxes infinite)
  ex.bounded(FFDE ? pr[RHO] : (gam - 1.) * pr[UU] + pr[RHO] + pr[UU]);
  // vchar and simplefast
  const double WW0 = pr[RHO] + gam * pr[UU];
  const bool wpos = WW0 > 0.;
  const double WW = wpos ? WW0 : 0.;
  const double cs2q = Exact::quot(gam * (gam - 1.) * pr[UU], ex.rcp(wpos ? WW0 : 1.));
  const double cs2 = wpos ? cs2q : 0.;
  const double EF = q.bsq + WW;
  const bool epos = EF > 0.;
  const double va2q = Exact::quot(q.bsq, ex.rcp(epos ? EF : 1.));
  const double va2 = epos ? va2q : 0.;
  // numerators unwatched: where the larger of the two squares exceeds 1e-150
  // its quotient is exact, and one so small that its quotient might not be
  // leaves cms2 at the other to the last bit (the upper ends are cms2's)
  ex.need((cs2 > va2 ? cs2 : va2) > 1.e-150);
  const double cms2 = cs2 + va2 - cs2 * va2;
  ex.need(cms2 >= 0. && cms2 <= 1.);
  const double Au = d1 ? q.ucon[1] : q.ucon[2], Bu = q.ucon[0];
  const double Au2 = Au * Au, Bu2 = Bu * Bu, AuBu = Au * Bu;
  const double A = Bu2 - (gtt + Bu2) * cms2;
  const double B = 2. * (AuBu - ((SP && !d1) ? AuBu : gd + AuBu) * cms2);
  const double C = Au2 - (gdd + Au2) * cms2;
  const double s = ex.sqrt_of(B * B - 4. * A * C);
  const Recip A2 = ex.rcp(2. * A);
  // s >= 2^-100, so neither sum is tiny unless it is zero
  const double vm = Exact::quot(B - s, A2), vp = Exact::quot(B + s, A2);
  x.vmax = (vp < vm) ? vm : vp;
  x.vmin = (vp < vm) ? vp : vm;
}

// what a face reads of its location's metric: g_{mu nu}, g^{t mu}, g^{dir dir}
// and sqrt(-g)
struct FaceGeo {
  double c[10], gcon[4], gdd, sg;
};
// loads that start where they are written (asm: the compiler would load each
// value at its use, in small batches)
template <bool SP>
__device__ __forceinline__ void load_face_geo(const StepArgs& a, int dir, long long z, FaceGeo& g)
{
  const long long pl = a.gr.plane;
  const double* b = a.geo + (long long)(dir == 1 ? FACE1 : FACE2) * GEO_PER_LOC * pl + z;
#pragma unroll
  for (int k = 0; k < 10; k++)
    if (!SP || !(SP_COV >> k & 1)) asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(g.c[k]) : "l"(b + k * pl));
#pragma unroll
  for (int k = 0; k < (SP ? 2 : 4); k++) asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(g.gcon[k]) : "l"(b + (10 + k) * pl));
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(g.gdd) : "l"(b + (dir == 1 ? 14 : 17) * pl));
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(g.sg) : "l"(b + 20 * pl));
}

// face_flux without branches: left and right point at the two interface
// states (planes ks doubles apart), dir 1 or 2, g its metric.  F and dtij are
// valid where ex.ok().
template <bool FFDE, bool SP, typename EX>
__device__ __forceinline__ void face_flux_x(EX& ex, const StepArgs& a, const FaceGeo& g, int dir, const double* left,
                                            const double* right, int ks, double* F, double& dtij, int rf)
{
  const double gd = (dir == 1) ? g.gcon[1] : (SP ? 0. : g.gcon[2]);
  const double gam = a.pp.gam, limit = (a.pp.gammamax <= 1.) ? 1.e300 : a.pp.gammamax;
  const int bd = (B1 - 1 + dir) * ks;
  const double Bd = 0.5 * (left[bd] + right[bd]);
  const LapseX l = lapse_x<SP>(ex, g.gcon);
  SideX sl, sr;
#pragma unroll
  for (int s = 0; s < 2; s++) {
    const double* src = s ? right : left;
    double p[NPR];
#pragma unroll
    for (int k = 0; k < NPR; k++) p[k] = src[k * ks];
    if (dir == 1) p[B1] = Bd;
    else p[B2] = Bd;
    StateX q;
    state_x<SP>(ex, p, g.c, l, limit, q);
    sl = sr;
    side_x<FFDE, SP>(ex, p, q, dir, g.sg, g.gcon[0], gd, g.gdd, gam, sr);
  }
  double cmin = rmin(sl.vmin, sr.vmin), cmax = rmax(sl.vmax, sr.vmax);
  cmin = fabs(rmax(0., -cmin));
  cmax = fabs(rmax(0., cmax));
  const double ctop = rmax(cmax, cmin), cc = cmax * cmin;
  const Recip sum = ex.rcp(cmax + cmin);
  // an in-range divisor and bounded states keep both forms finite, so the form
  // that choose_flux weighs with 0 adds nothing
#pragma unroll
  for (int k = 0; k < NX; k++) {
    const double dU = sr.U[k] - sl.U[k];
    if (((k < B1) ? rf : a.pp.fluxmethod) == 1) F[k] = ex.div(cmax * sl.F[k] + cmin * sr.F[k] - cc * dU, sum);
    else F[k] = 0.5 * (sl.F[k] + sr.F[k] - ctop * dU);
  }
  dtij = Exact::quot(a.pp.cour * (dir == 1 ? a.pp.dx1 : a.pp.dx2), ex.rcp(ctop));
}

// fix_flux's face-local rules (fixup.c:1357-1410) on the flux through the
// face (i, j): the mass-flux sign clamps at the two x1 ends; only u~2's flux
// crosses the polar and equatorial x2 faces
template <typename T>
__device__ __forceinline__ void fix_face(const StepArgs& a, int i, int j, int dir, T* Fo)
{
  const int n1 = a.gr.n1, n2 = a.gr.n2;
  if (dir == 1) {
    if (i == 0 && a.pp.bc == 0 && j >= -1 && j < n2 && Fo[RHO] > 0) Fo[RHO] = 0;
    if (i == n1 && j >= -1 && j < n2 && Fo[RHO] < 0) Fo[RHO] = 0;
  } else {
    const bool polar = (j == 0 || j == n2) && (i < n1);
    const bool equator = (j == (n2 - 1) / 2) && (i >= 0) && (i < n1);
    if (polar || equator) {
#pragma unroll
      for (int k = 0; k < NPR; k++)
        if (k != U2) Fo[k] = T(0.);
    }
  }
}

__device__ __forceinline__ void store_face_x(const StepArgs& a, int i, int j, int dir, long long z, const double* Fx)
{
  double Fo[NPR];
#pragma unroll
  for (int k = 0; k <= U3; k++) Fo[k] = Fx[k];
  Fo[B1] = (dir == 1) ? 0. : Fx[XB];
  Fo[B2] = (dir == 1) ? Fx[XB] : 0.;
  Fo[B3] = Fx[XB3];
  fix_face(a, i, j, dir, Fo);
  double* F = ((dir == 1) ? a.F1 : a.F2) + z;
#pragma unroll
  for (int k = 0; k < NPR; k++) F[k * a.gr.plane] = Fo[k];
}

// The face (i, j) in direction dir that face_flux_x could not take (left: its
// left state, the right one NPR planes on).  Stores the flux and returns the
// face's Courant limit.
template <bool FFDE>
__device__ __noinline__ double face_general(const StepArgs& a, const double* left, int ks, int i, int j, int dir, int rf)
{
  const long long z = a.gr.at(i, j);
  double pl[NPR], pr[NPR], Fo[NPR], dtij;
#pragma unroll
  for (int k = 0; k < NPR; k++) {
    pl[k] = left[k * ks];
    pr[k] = left[(NPR + k) * ks];
  }
  face_flux<double, FFDE>(a, i, j, dir, pl, pr, Fo, dtij, rf);
  fix_face(a, i, j, dir, Fo);
  double* F = ((dir == 1) ? a.F1 : a.F2) + z;
#pragma unroll
  for (int k = 0; k < NPR; k++) F[k * a.gr.plane] = Fo[k];
  return dtij;
}

__device__ __forceinline__ double block_min(double v, double* sh)
{
  // exact minimum (no rounding), NaN-ignoring like `if (x < m) m = x`
  for (int o = 16; o > 0; o >>= 1) {
    double w = __shfl_down_sync(0xffffffffu, v, o);
    v = (w < v) ? w : v;
  }
  const int lane = (threadIdx.y * blockDim.x + threadIdx.x) & 31, warp = (threadIdx.y * blockDim.x + threadIdx.x) >> 5;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  const int nw = (blockDim.x * blockDim.y + 31) >> 5;
  if (warp == 0) {
    v = (lane < nw) ? sh[lane] : 1.e9;
    for (int o = 16; o > 0; o >>= 1) {
      double w = __shfl_down_sync(0xffffffffu, v, o);
      v = (w < v) ? w : v;
    }
  }
  return v;
}

// fluxcalc for both directions over i in [-1,N1], j in [-1,N2]: x1 faces
// with i >= 0, x2 faces with j >= 0 (FZLOOP ranges), then the fix_flux
// rules that do not read another face (fixup.c:1357-1410; the inner x1 mass
// flux clamp only where that end is OUTFLOW, i.e. for the torus).  Blocks are
// 32 (x1) x BY (x2) zones.  The block's primitive tile -- its zones, the
// two-zone stencil halo on every side and one more row below, for the x2
// neighbour of its first row -- arrives in shared memory by one TMA copy
// (flux_tile_*, below); every zone reconstructs its own interface states
// once from the tile (the first row also those of the zones below it).
// Lane 0's zone is also the previous block's lane 31 (blocks step by FLUX_BX
// = 31 along x1): lane 0 only lends its right state, and its faces are the
// previous block's (block 0's lane 0 is zone -1, which has no x1 face but an
// x2 face).  BY = 4 or 8 rows per block (flux_rows).

// the block's tile: issues its TMA copy (one thread); the zone's value of
// plane 0 is at the returned pointer
template <int BY>
__device__ __forceinline__ const double* flux_tile_load(double* tile, const CUtensorMap* map, uint64_t* bar)
{
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int cx = (int)(blockIdx.x * FLUX_BX) & ~1;  // the tile's first column (even)
  if (tx == 0 && ty == 0) {
    mbar_init(bar, 1);
    mbar_expect_tx(bar, (uint32_t)flux_tile_bytes(BY));
    tma_load_3d(tile, map, cx, (int)(blockIdx.y * BY) - 1, 0, bar);
  }
  // row ty + 3, column tx + 2 + (the block's first column - cx)
  return tile + (ty + 3) * FLUX_TILE_W + tx + 2 + ((int)(blockIdx.x * FLUX_BX) - cx);
}

// a row of a slot plane: 33 values, so that lanes in successive rows hit
// successive banks
constexpr int FLUX_SLOT_W = 33;
// The interface states of the block's zones, from the tile (tz: the thread's
// zone) into four slots a zone in shared memory: state s (0 left, 1 right) of
// its face in direction dir is slot[(2 * dir - 2 + s) * NPR * KS + k * KS],
// KS = BY * FLUX_SLOT_W.  A warp forms the states of one variable (BY = 8) or
// two at all of the block's zones: along x2 a lane per column (and the zones
// below the first row, for their right states), along x1 a lane per BY zones
// of a row.  A zone's right state is the left state of the next zone's face.
template <typename T, bool PARA, int BY>
__device__ __forceinline__ void block_states(const double* tz, T* slot, bool does1 = true, bool does2 = true)
{
  const int tx = threadIdx.x, ty = threadIdx.y;
  constexpr int PS = flux_tile_rows(BY) * FLUX_TILE_W, SW = FLUX_SLOT_W, KS = BY * SW;
#pragma unroll 1
  for (int k = ty; k < NPR; k += BY) {
    const double* t = tz + (k * PS - ty * FLUX_TILE_W - tx);  // the block's first zone
    T* d = slot + (k * KS - ty * SW - tx);
    if (does2) {
      T* d2 = d + 2 * NPR * KS + tx;
      row_states<T, PARA, BY + 1>(t + tx - FLUX_TILE_W, FLUX_TILE_W, [&](int c, T l, T r) {
        if (c > 0) d2[NPR * KS + (c - 1) * SW] = l;
        if (c < BY) d2[c * SW] = r;
      });
    }
    if (!does1) continue;
    const int row = tx % BY, c0 = (tx / BY) * BY;
    d += row * SW + c0;
    row_states<T, PARA, BY>(t + row * FLUX_TILE_W + c0, 1, [&](int c, T l, T r) {
      d[NPR * KS + c] = l;
      d[c + 1] = r;  // (the last zone's goes to the row's padding)
    });
  }
}

// the block's Courant minima
__device__ __forceinline__ void flux_block_dt(const StepArgs& a, double dt1, double dt2, double (*sh)[32])
{
  dt1 = block_min(dt1, sh[0]);
  dt2 = block_min(dt2, sh[1]);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    const int b = blockIdx.y * gridDim.x + blockIdx.x;
    if (blockIdx.z == 0) a.blockmin[b] = dt1;
    if (blockIdx.z == gridDim.z - 1) a.blockmin[a.nblocks_flux + b] = dt2;
  }
}

// The b^2 flags and the flux choice of the zone at tz, formed in the first
// substep of a step with the per-zone switch (from the step's p, which is
// that substep's tile; get_bsqflags, fixup.c:1197-1295, with the b^2 flags
// the repairs read later): (flags) | (choice) << 8
__device__ __forceinline__ int flux_flags(const StepArgs& a, const double* tz, int ps, long long z)
{
  double pr[NPR];
#pragma unroll
  for (int k = 0; k < NPR; k++) pr[k] = tz[k * ps];
  Geo<double> gz;
  load_geo(a, CENT, z, gz);
  unsigned char b = 0;
  if (!a.pp.eom) {
    State<double> q;
    state_of(pr, gz, q);
    b = bsq_flag(a, pr, q);
  }
  const double gamma = gamma_of(pr, gz);
  const int f1 = (gamma > 2.0 * a.pp.gammadamp) ? 2 : ((gamma > a.pp.gammadamp) ? 1 : 0);
  const int rf = ((b & 3) == 2 || f1 == 2 || (b >> 2) == 2) ? a.pp.fluxmethod - 1 : a.pp.fluxmethod;
  return b | ((rf < 0) ? 0 : rf) << 8;
}

// flux_flags for the FP64 faces: without branches, or flux_flags itself
static __device__ __noinline__ int flux_flags_x(const StepArgs& a, const double* tz, int ps, long long z)
{
  const double* base = a.geo + (long long)CENT * GEO_PER_LOC * a.gr.plane + z;
  double pr[NPR], c[10], gcon[4];
#pragma unroll
  for (int k = 0; k < NPR; k++) pr[k] = tz[k * ps];
#pragma unroll
  for (int k = 0; k < 10; k++) c[k] = __ldg(base + k * a.gr.plane);
#pragma unroll
  for (int k = 0; k < 4; k++) gcon[k] = __ldg(base + (10 + k) * a.gr.plane);
  Exact ex;
  StateX q;
  state_x<false>(ex, pr, c, lapse_x<false>(ex, gcon), 1.e300, q);
  const unsigned char b = bsq_flag_x(ex, a, pr, q.bsq);
  if (a.pp.eom || !ex.ok()) return flux_flags(a, tz, ps, z);
  const int f1 = (q.gamma > 2.0 * a.pp.gammadamp) ? 2 : ((q.gamma > a.pp.gammadamp) ? 1 : 0);
  const int rf = ((b & 3) == 2 || f1 == 2 || (b >> 2) == 2) ? a.pp.fluxmethod - 1 : a.pp.fluxmethod;
  return b | ((rf < 0) ? 0 : rf) << 8;
}

// FP32 faces (mixed form): both directions through one copy of the face
// code, dir a run-time value (the direction-dependent reads are selects),
// which halves the kernel's instruction footprint.  96 registers a thread:
// five 4-row blocks per SM.  Leaving out the sparse metric's planes and
// products takes 6 us off a mixed step at 512^2 and 6.4 off the 512 x 256
// dipole's, forming PARA's states by block_states 24 at 512^2; all with the
// same bits.  49 us a launch at 512^2 PARA with the switch, 23 on the dipole.
template <typename T, bool PARA, bool FFDE, int BY, bool SP>
__global__ void __launch_bounds__(32 * BY, 5)
    k_flux(const __grid_constant__ StepArgs a, const __grid_constant__ CUtensorMap prim_map)
{
  extern __shared__ __align__(128) double tile[];
  __shared__ double sh[2][32];
  __shared__ uint64_t bar;
  const int tx = threadIdx.x, ty = threadIdx.y;
  constexpr int PS = flux_tile_rows(BY) * FLUX_TILE_W, SW = FLUX_SLOT_W, KS = BY * SW;
  const double* tz = flux_tile_load<BY>(tile, &prim_map, &bar);
  T* slot = reinterpret_cast<T*>(tile + NPR * PS) + ty * SW + tx;  // as in k_flux_fp64
  const int i = blockIdx.x * FLUX_BX + tx - 1;
  const int j = blockIdx.y * BY + ty - 1;
  const int n1 = a.gr.n1, n2 = a.gr.n2;
  const bool in = (i <= n1) && (j <= n2);
  const bool own = (tx > 0) || (blockIdx.x == 0);  // lane 0 of a later block repeats a zone
  const long long z = a.gr.at(in ? i : -1, in ? j : -1);
  double dt1 = 1.e9, dt2 = 1.e9;
  T L[NPR], pl[NPR];
  T Fo[NPR];
  double dtij;
  T* F1 = reinterpret_cast<T*>(a.F1);
  T* F2 = reinterpret_cast<T*>(a.F2);
  __syncthreads();  // the barrier is initialised before anyone polls it
  if (!mbar_wait(&bar, 0)) {
    if (tx == 0 && ty == 0) report_fail(a.sc, a.phase0 + PH_FACE1, FAIL_TMA_TIMEOUT, zone_order(i, j));
    return;
  }
  if constexpr (PARA) block_states<T, PARA, BY>(tz, slot);
  // the flux choice of this zone, which both of its faces use: fluxmethod,
  // or with the per-zone switch FLAGREALFLUX, formed in the first substep
  // and read back in the second
  int rf = a.pp.fluxmethod;
  if (a.pp.fluxadjust && in) {
    if (a.flags_here) {
      const int f = flux_flags(a, tz, PS, z);
      rf = f >> 8;
      if (own) {
        a.bsqf[z] = (unsigned char)(f & 255);
        a.fluxf[z] = (unsigned char)rf;
      }
    } else {
      rf = (int)a.fluxf[z];
    }
  }
  if constexpr (PARA) __syncthreads();
#pragma unroll 1
  for (int dir = 1; dir <= 2; dir++) {
    if constexpr (PARA) {
      const T* left = slot + (2 * dir - 2) * NPR * KS;
#pragma unroll
      for (int k = 0; k < NPR; k++) {
        pl[k] = left[k * KS];
        L[k] = left[(NPR + k) * KS];
      }
    } else {
      // MC's slopes are cheap: each thread forms its own zone's, and the left
      // state comes by shuffle or through shared memory (the mixed 512 x 256
      // dipole 88.2 us a step then, with block_states 90.9)
      const int st = (dir == 1) ? 1 : FLUX_TILE_W;
      T R[NPR];
#pragma unroll
      for (int k = 0; k < NPR; k++)
        row_states<T, false, 1>(tz + k * PS, st, [&](int, T l, T r) {
          L[k] = l;
          R[k] = r;
        });
      if (dir == 1) {
#pragma unroll
        for (int k = 0; k < NPR; k++) pl[k] = __shfl_up_sync(0xffffffffu, R[k], 1);
      } else {
#pragma unroll
        for (int k = 0; k < NPR; k++) slot[k * KS] = R[k];
        __syncthreads();
        if (ty > 0) {
#pragma unroll
          for (int k = 0; k < NPR; k++) pl[k] = slot[k * KS - SW];
        } else {
#pragma unroll
          for (int k = 0; k < NPR; k++)
            row_states<T, false, 1>(tz + k * PS - st, st, [&](int, T, T r) { pl[k] = r; });
        }
      }
    }
    const bool act = (dir == 1) ? (in && i >= 0 && tx > 0) : (in && j >= 0 && own);
    if (act) {
      face_flux<T, FFDE, SP>(a, i, j, dir, pl, L, Fo, dtij, rf);
      T* F;
      if (dir == 1) {
        dt1 = (dtij < dt1) ? dtij : dt1;
        F = F1;
      } else {
        dt2 = (dtij < dt2) ? dtij : dt2;
        F = F2;
      }
      fix_face(a, i, j, dir, Fo);
#pragma unroll
      for (int k = 0; k < NPR; k++) F[k * a.gr.plane + z] = Fo[k];
    }
  }
  flux_block_dt(a, dt1, dt2, sh);
}

// FP64 faces.  FP64 issue and latency bound: 2255 FP64-pipe instructions a
// zone (2065 with the sparse metric; 512^2 PARA, a launch that forms no
// flags) at 128 registers (16 warps per SM).  What the layout is for:
//  * all interface states are formed first, into shared memory (four slots a
//    zone: the left and right state of its x1 and x2 face).  A warp takes one
//    variable of the whole block and walks along the zones, so each slope and
//    raw interface value is formed once (93 instead of 172 FP64 instructions
//    a variable and zone), and the block meets at one barrier while its warps
//    are still together;
//  * then each thread takes its two faces in one stretch of code without a
//    branch (harm_exact.cuh).  Warps with states so small that quotients
//    leave Exact's range (the field ahead of its front: 5% of the warps of
//    the 512^2 torus at t = 3, 13% of the 1024^2 one at t = 0.8) take the
//    ExactTiny form, and what neither can take goes to face_general, whose
//    code is cold: 0.2% of the warps there cost 20% of the kernel.
// Time per launch, developed flow, mean of both substeps (one face at a time,
// each quotient and root with its own branches -> this form): 512^2 PARA
// with the switch 152 -> 88 us, 1024^2 626 -> 299 us, 128^2 MC 26 -> 16 us,
// the force-free 512 x 256 dipole 63.5 -> 38 us.
template <bool PARA, bool FFDE, int BY, bool SPLIT, bool SP>
__global__ void __launch_bounds__(32 * BY, 512 / (32 * BY))
    k_flux_fp64(const __grid_constant__ StepArgs a, const __grid_constant__ CUtensorMap prim_map)
{
  extern __shared__ __align__(128) double tile[];
  __shared__ double sh[2][32];
  __shared__ uint64_t bar;
  const int tx = threadIdx.x, ty = threadIdx.y;
  constexpr int PS = flux_tile_rows(BY) * FLUX_TILE_W, SW = FLUX_SLOT_W, KS = BY * SW;
  const double* tz = flux_tile_load<BY>(tile, &prim_map, &bar);
  double* slot = tile + NPR * PS + ty * SW + tx;  // state s of direction dir: slot[(2 * dir - 2 + s) * NPR * KS + k * KS]
  const int i = blockIdx.x * FLUX_BX + tx - 1;
  const int j = blockIdx.y * BY + ty - 1;
  const int n1 = a.gr.n1, n2 = a.gr.n2;
  const bool in = (i <= n1) && (j <= n2);
  const bool own = (tx > 0) || (blockIdx.x == 0);  // lane 0 of a later block repeats a zone
  const long long z = a.gr.at(in ? i : -1, in ? j : -1);
  double dt1 = 1.e9, dt2 = 1.e9;
  // SPLIT: a layer of blocks for each direction (flux_launch_by)
  const bool does1 = !SPLIT || blockIdx.z == 0, does2 = !SPLIT || blockIdx.z == 1;
  // the first face's metric is on its way while the states are formed (8-row
  // blocks: 1024^2 298 -> 291 us; the small grids of 4-row ones keep their
  // metric in L2, and their steps were 2% slower with it)
  FaceGeo g;
  if (BY == FLUX_BY_LARGE) load_face_geo<SP>(a, does1 ? 1 : 2, z, g);
  __syncthreads();  // the barrier is initialised before anyone polls it
  if (!mbar_wait(&bar, 0)) {
    if (tx == 0 && ty == 0) report_fail(a.sc, a.phase0 + PH_FACE1, FAIL_TMA_TIMEOUT, zone_order(i, j));
    return;
  }
  block_states<double, PARA, BY>(tz, slot, does1, does2);
  // the flux choice of this zone (as in k_flux)
  int rf = a.pp.fluxmethod;
  if (a.pp.fluxadjust && in) {
    if (a.flags_here) {
      const int f = flux_flags_x(a, tz, PS, z);
      rf = f >> 8;
      if (own && does1) {
        a.bsqf[z] = (unsigned char)(f & 255);
        a.fluxf[z] = (unsigned char)rf;
      }
    } else {
      rf = (int)a.fluxf[z];
    }
  }
  __syncthreads();
  // whether one of the states of the warp's faces holds a velocity or field
  // so small that quotients may leave Exact's range (lane 0 has no x1 face and
  // its left slot is not written: it looks at lane 1's)
  const double* slot0 = slot + (tx == 0);
  bool small = false;
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int k = U1; k <= B3; k++) {
      if (!(q < 2 ? does1 : does2)) continue;
      // (volatile: these values are read again where they are used)
      const double v = *const_cast<const volatile double*>((q == 0 ? slot0 : slot) + (q * NPR + k) * KS);
      const uint32_t t = hi_word(v) & 0x7fffffffu;
      small |= (t < Exact::word(-850)) && ((t | lo_word(v)) != 0);
    }
  const bool tiny = __any_sync(0xffffffffu, small);
  // both faces in one stretch of code; what it could not take comes after it
  bool todo1 = does1 && in && i >= 0 && tx > 0, todo2 = does2 && in && j >= 0 && own;
  auto faces = [&](auto ex0) {
#pragma unroll
    for (int dir = 1; dir <= 2; dir++) {
      bool& todo = (dir == 1) ? todo1 : todo2;
      if (!todo) continue;
      const double* left = slot + (2 * dir - 2) * NPR * KS;
      double Fx[NX], dtij;
      if ((dir == 2 && does1) || BY != FLUX_BY_LARGE) load_face_geo<SP>(a, dir, z, g);
      auto ex = ex0;
      face_flux_x<FFDE, SP>(ex, a, g, dir, left, left + NPR * KS, KS, Fx, dtij, rf);
      if (ex.ok()) {
        store_face_x(a, i, j, dir, z, Fx);
        if (dir == 1) dt1 = (dtij < dt1) ? dtij : dt1;
        else dt2 = (dtij < dt2) ? dtij : dt2;
        todo = false;
      }
    }
  };
  if (!SP || __ldg(a.geo_full) == 0) {  // (a geometry uploaded since the kernel was chosen)
    if (!tiny) faces(Exact());
    else faces(ExactTiny());
  }
#pragma unroll 1
  for (int dir = 1; dir <= 2; dir++) {
    if (!((dir == 1) ? todo1 : todo2)) continue;
    const double dtij = face_general<FFDE>(a, slot + (2 * dir - 2) * NPR * KS, KS, i, j, dir, rf);
    if (dir == 1) dt1 = (dtij < dt1) ? dtij : dt1;
    else dt2 = (dtij < dt2) ? dtij : dt2;
  }
  flux_block_dt(a, dt1, dt2, sh);
}

// the k_flux instance of the block's row count (b.y) and the metric's form
template <typename T, bool PARA, bool FFDE, int BY, bool SP>
inline void flux_launch_by(dim3 g, dim3 b, cudaStream_t s, const StepArgs& a, const CUtensorMap& map)
{
  constexpr bool fp64 = sizeof(T) == 8;
  // (MC's FP32 faces pass one state on: the rest of the SM's memory is L1)
  constexpr int slots = (fp64 || PARA) ? 4 : 1;
  constexpr size_t sm = flux_tile_bytes(BY) + slots * NPR * BY * FLUX_SLOT_W * sizeof(T);
  void (*kern)(StepArgs, CUtensorMap);
  // Where the blocks would take at most half of the SMs' slots (four 4-row
  // blocks each), each direction gets a layer of blocks of its own, and a
  // block half the work: a step of the 64^2 torus 71.3 -> 65.3 us, 128^2 79.6
  // -> 75.2, 245 x 131 90.9 -> 86.2 (the next size up fills the SMs anyway).
  // An ensemble's members fill the SMs together, and the layers only repeat
  // the tile's copy, where their blocks no longer all fit at once (a step of
  // 2 tori of 64^2 with layers 71.8 us, without 78.4; 4 of 96^2 92.6, 93.5; 3
  // of 128^2 102.9, 103.7; 4 of 128^2 123.0, 119.8; 16 of 128^2 with the switch
  // 396, 360; 16 uneven ones 919, 884).
  constexpr bool small = fp64 && BY == FLUX_BY_SMALL;
  if (small && g.x * g.y <= 2 * 148 && a.ens_blocks <= 4 * 148) g.z = 2;
  if constexpr (small) kern = (g.z == 2) ? k_flux_fp64<PARA, FFDE, BY, true, SP> : k_flux_fp64<PARA, FFDE, BY, false, SP>;
  else if constexpr (fp64) kern = k_flux_fp64<PARA, FFDE, BY, false, SP>;
  else kern = k_flux<T, PARA, FFDE, BY, SP>;
  static SmemLimit limit[2];
  limit[g.z - 1].raise((const void*)kern, sm);
  kern<<<g, b, sm, s>>>(a, map);
}
template <typename T, bool PARA, bool FFDE, bool SP>
inline void flux_rows_launch(dim3 g, dim3 b, cudaStream_t s, const StepArgs& a, const CUtensorMap& map)
{
  // (the FP32 faces' blocks have 4 rows on any grid, flux_rows)
  if constexpr (sizeof(T) == 8) {
    if (b.y == FLUX_BY_LARGE) {
      flux_launch_by<T, PARA, FFDE, FLUX_BY_LARGE, SP>(g, b, s, a, map);
      return;
    }
  }
  flux_launch_by<T, PARA, FFDE, FLUX_BY_SMALL, SP>(g, b, s, a, map);
}

// flux_ct corner EMF, step_ch.c:1214-1234, over i in [0,N1], j in [0,N2].
// F1 on the rows j = -1 and j = N2 carries fix_flux's mirrored B2 for i < N1.
// The grid spans i, j from -1: with bsqf_fused set (the first substep of an
// FP64 GRMHD step) the threads of the ring one zone outside the active grid
// (i or j in {-1, N}) set the b^2 flags of their zone from the step's p, as
// get_bsqflags does over its DQZLOOP range (fixup.c:1197-1233); the first
// substep's k_update sets those of the active zones.
template <typename FT>
__global__ void k_emf(StepArgs a, const double* __restrict__ pv)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x - 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y - 1;
  const int n1 = a.gr.n1, n2 = a.gr.n2;
  if (i == 0 && j == 0) a.sc->ndeferred = 0;
  if (i > n1 || j > n2) return;
  if (a.bsqf_fused && (i == -1 || i == n1 || j == -1 || j == n2)) {
    const long long z = a.gr.at(i, j);
    double pr[NPR];
#pragma unroll
    for (int k = 0; k < NPR; k++) pr[k] = __ldg(pv + k * a.gr.plane + z);
    Geo<double> g;
    load_geo(a, CENT, z, g);
    State<double> q;
    state_of(pr, g, q);
    a.bsqf[z] = bsq_flag(a, pr, q);
  }
  if (i < 0 || j < 0) return;
  const long long pl = a.gr.plane;
  const FT* F1b2 = reinterpret_cast<const FT*>(a.F1) + B2 * pl;
  const FT* F2b1 = reinterpret_cast<const FT*>(a.F2) + B1 * pl;
  // the mirrored rows by their address, so that all loads start together
  const bool top = j == n2 && i < n1, bottom = j - 1 == -1 && i < n1;
  double f1a = __ldg(F1b2 + a.gr.at(i, top ? n2 - 1 : j)), f1b = __ldg(F1b2 + a.gr.at(i, bottom ? 0 : j - 1));
  const double f2a = __ldg(F2b1 + a.gr.at(i, j)), f2b = __ldg(F2b1 + a.gr.at(i - 1, j));
  const double gc = gdet_at(a, CORN, a.gr.at(i, j));
  const double g1 = gdet_at(a, FACE1, a.gr.at(i, j)), g2 = gdet_at(a, FACE1, a.gr.at(i, j - 1));
  const double g3 = gdet_at(a, FACE2, a.gr.at(i, j)), g4 = gdet_at(a, FACE2, a.gr.at(i - 1, j));
  f1a = top ? -f1a : f1a;
  f1b = bottom ? -f1b : f1b;
  // quotients without branches (harm_exact.cuh): fluxes ahead of the field's
  // front are subnormal, which the operator handles apart (1024^2 with the
  // launch 26.6 -> 22.0 us, 512^2 11.8 -> 10.5)
  ExactTiny ex;
  double e = ex.div(f1a, ex.rcp(g1)) + ex.div(f1b, ex.rcp(g2)) - ex.div(f2a, ex.rcp(g3)) - ex.div(f2b, ex.rcp(g4));
  if (!ex.ok()) e = f1a / (g1) + f1b / (g2) - f2a / (g3) - f2b / (g4);
  a.emf[a.gr.at(i, j)] = 0.25 * (gc) * (e);
}

// ---------------------------------------------------------------- update
// Newton iterations a zone may take inside k_update before it is handed to
// k_update_tail, which continues the solve from the saved state (the
// reference's limit is 200; typical zones need 2-4).
#ifndef HARM_NEWTON_CAP
#define HARM_NEWTON_CAP 16
#endif
constexpr int NEWTON_MAIN_CAP = HARM_NEWTON_CAP;

// pflag store + fixup1zone (fixup.c:274-377: floors then the Lorentz factor
// limit) + store of the new primitives; frho, fu: the zone's floors
__device__ __forceinline__ void finish_zone(const StepArgs& a, const Geo<double>& g, long long z, int i, int j, double* pfz,
                                            int pfl, double* pf, double frho, double fu)
{
  const long long pl = a.gr.plane;
  if (a.rec_pinv) {
#pragma unroll
    for (int k = 0; k < NPR; k++) a.rec_pinv[k * pl + z] = pfz[k];
  }
  a.pflag[z] = pfl;
  if (frho > pfz[RHO]) pfz[RHO] = frho;
  if (fu > pfz[UU]) pfz[UU] = fu;
  int rc = limit_gamma(a.pp.gammamax, pfz, g);
  if (rc) report_fail(a.sc, a.phase0 + PH_UPDATE, rc, zone_order(i, j));
#pragma unroll
  for (int k = 0; k < NPR; k++) pf[k * pl + z] = pfz[k];
}

// ---- the zone update without branches (harm_exact.cuh)
// utoprim_2d (harm_device.cuh) with the same operands in the same order,
// every quotient and root through `ex`; its rare exits (a bad guess, an
// iterate out of bounds) leave ex.ok() false.  The result, pflag and iteration
// count hold where ex.ok().
//
// Numerators of the Newton step are not watched.  Q.B^2 may be arbitrarily
// small, but a W in range keeps the terms with it below 2^-700 where its
// quotients are not exact, and there they change nothing to the last bit:
// they are added to terms of order W or W^2, to a residual that is zero or
// larger, or to a vsq that is zero (the new vsq is then below the range that
// its reciprocal is watched for) or at least 2^-200.  A dx whose own quotient
// is not exact is far below the tolerance either way.
__device__ __forceinline__ double utsq_calc_x(ExactTiny& ex, const U2PCtx& c, double W)
{
  const double Wsq = W * W, W4 = Wsq * Wsq;
  const double den = W4 + 2. * c.Bsq * Wsq * W + Wsq * (c.Bsq * c.Bsq - c.Qtsq) - c.QdotBsq * (2. * W + c.Bsq);
  return ex.div_normal(c.Bsq * c.QdotBsq + W * (2. * c.QdotBsq + c.Qtsq * W), ex.rcp(den));
}

__device__ __forceinline__ int newton_vsq_x(ExactTiny& ex, const U2PCtx& c, double& x0, double& x1, double gammafail,
                                            int& niter_out, int maxit, double* st, long long ss, bool resume)
{
  constexpr int MAX_NEWT_ITER = 200;
  constexpr double NEWT_TOL = 1.0e-15, MIN_NEWT_TOL = 1.0e-10, W_TOO_BIG = 1.e9;
  const double vsq_too_big = (1.0 - 1.0 / (gammafail - 1.0));
  const double Bsq = c.Bsq, QdotBsq = c.QdotBsq, gam = c.gam;
  double errx = 1., errx_old = 2., errx_oldest;
  int n_iter = 0;
  if (resume) {
    x0 = st[0];
    x1 = st[ss];
    errx = st[2 * ss];
    errx_old = st[3 * ss];
    n_iter = (int)st[4 * ss];
  }
  const Recip rgam = ex.rcp(gam), rwg = ex.rcp(c.wglobal);
  Recip rW = ex.rcp(x0);
#pragma unroll 1
  while ((errx > NEWT_TOL) && (n_iter < maxit)) {
    // func_vsq
    const double W = x0, vsq = x1, Wsq = W * W, W3 = Wsq * W, gtmp = 1. - vsq;
    const double sq = ex.sqrt_of(gtmp);
    const Recip r2 = ex.rcp_from(Wsq, rW.y * rW.y), r3 = ex.rcp_from(W3, r2.y * rW.y);
    const double p_tmp = ExactTiny::quot((gam - 1.) * (W * gtmp - c.D * sq), rgam);
    const double dPdW = ExactTiny::quot((gam - 1.) * gtmp, rgam);
    const double dPdvsq = ExactTiny::quot((gam - 1.) * (ExactTiny::quot(0.5 * c.D, ex.rcp(sq)) - W), rgam);
    const double BW = Bsq + W;
    const double t2 = c.Qtsq - vsq * (BW * BW) + ExactTiny::quot(QdotBsq * (Bsq + 2 * W), r2);
    const double t3 = c.Qdotn - (Bsq * (1 + vsq)) / 2. + 0.5 * ExactTiny::quot(QdotBsq, r2) - W + p_tmp;
    const double QW3 = ExactTiny::quot(QdotBsq, r3), s = -1 + dPdW - QW3;
    double dx0 = (-Bsq / 2. + dPdvsq) * t2 + (BW * BW) * t3;
    double dx1 = -(s * t2) - 2 * (vsq + QW3) * BW * t3;
    const double detJ = BW * (s * BW + ExactTiny::quot((Bsq - 2 * dPdvsq) * (QdotBsq + vsq * W3), r3));
    const Recip rd = ex.rcp(fabs(detJ));
    dx0 = ExactTiny::quot((detJ < 0.) ? dx0 : -dx0, rd);
    dx1 = ExactTiny::quot((detJ < 0.) ? dx1 : -dx1, rd);
    if (((n_iter + 1) % 10) == 0) {
      const double r = cycle_break_uniform(x0, x1, n_iter);
      dx0 *= r;
      dx1 *= r;
    }
    errx_oldest = errx_old;
    errx_old = errx;
    x0 = fabs(x0 + dx0);
    rW = ex.rcp(x0);
    x1 += dx1;
    // where x1 is zero the reference takes |dx1| itself
    errx = (ExactTiny::quot(fabs(dx0), rW) + ExactTiny::quot(fabs(dx1), ex.rcp((x1 == 0.) ? 1. : fabs(x1)))) / 2.;
    ex.need(!(ExactTiny::quot(x0, rwg) > W_TOO_BIG));
    x1 = (x1 < 0.) ? 0.0 : x1;
    x1 = (x1 > 1.) ? vsq_too_big : x1;
    if (((errx_old == errx) || (errx_oldest == errx)) && (errx < MIN_NEWT_TOL)) errx = -errx;
    n_iter++;
  }
  niter_out = n_iter;
  if (maxit < MAX_NEWT_ITER && n_iter >= maxit && errx > NEWT_TOL) {
    if (st && ex.ok()) {
      st[0] = x0;
      st[ss] = x1;
      st[2 * ss] = errx;
      st[3 * ss] = errx_old;
      st[4 * ss] = (double)n_iter;
    }
    return NEWTON_DEFERRED;
  }
  if (n_iter >= MAX_NEWT_ITER) return (errx > MIN_NEWT_TOL) ? 1 : 0;
  return 0;
}

// c, gn: the packed g_{mu nu} and g^{mu nu}; sg: sqrt(-g)
template <bool SP>
__device__ __forceinline__ int utoprim_2d_x(ExactTiny& ex, const double* U, const double* c, const double* gn, double sg,
                                            double* pr, double gam, double gammafail, int* niter, int maxit, double* nst,
                                            long long nss, bool resume)
{
  constexpr double W_TOO_BIG = 1.e9, FAIL_VAL = 1.e30;
  double Ut[NPR];
  const Recip rs = ex.rcp(sg);
  const double ngn = -gn[0];
  const Recip ral = ex.rcp(ExactTiny::quot(1., ex.rcp(ex.sqrt_of(ngn))));  // alpha
  const double alpha = ral.b;
  {
    double Ug[NPR];
#pragma unroll
    for (int k = 0; k < B1; k++) Ug[k] = ex.div_normal(U[k], rs);
#pragma unroll
    for (int k = B1; k <= B3; k++) Ug[k] = ex.div(U[k], rs);
    Ug[UU] += -Ug[RHO];
    Ut[RHO] = Ug[RHO] * alpha;
#pragma unroll
    for (int k = UU; k <= U3; k++) Ut[k] = -alpha * Ug[k];
#pragma unroll
    for (int k = B1; k <= B3; k++) Ut[k] = alpha * Ug[k];
  }
  const double* B = Ut + B1;
  const double* Q = Ut + UU;
  U2PCtx x;
  x.gam = gam;
  double Bv[3];
  lower_space<SP>(B, c, Bv);
  x.Bsq = B[0] * Bv[0] + B[1] * Bv[1] + B[2] * Bv[2];
  double Qcon[4];
  raise_con<SP>(Q, gn, Qcon);
  const double QdotB = Q[1] * B[0] + Q[2] * B[1] + Q[3] * B[2];
  x.QdotBsq = QdotB * QdotB;
  const double nlapse = -ex.sqrt_of(ExactTiny::quot(1., ex.rcp(ngn)));
  x.Qdotn = Qcon[0] * nlapse;
  x.Qtsq = Q[0] * Qcon[0] + Q[1] * Qcon[1] + Q[2] * Qcon[2] + Q[3] * Qcon[3] + x.Qdotn * x.Qdotn;
  x.D = Ut[RHO];
  double utsq = 0.;
#pragma unroll
  for (int i = 1; i < 4; i++)
#pragma unroll
    for (int j = 1; j < 4; j++) {
      if (SP && (SP_COV >> sym(i, j) & 1)) continue;
      const double t = c[sym(i, j)] * pr[U1 + i - 1] * pr[U1 + j - 1];
      utsq = (i == 1 && j == 1) ? t : utsq + t;
    }
  const double utsq_too_big = ((gammafail - 1.0) * (gammafail - 1.0));
  ex.need(utsq >= 0. && utsq <= utsq_too_big);
  const double p0 = (gam - 1.) * pr[UU], w0 = pr[RHO] + pr[UU] + p0;
  x.wglobal = w0;
  double W = w0 * (1. + utsq);
  double x0 = fabs(W), ut = fabs(utsq_calc_x(ex, x, W));
  double x1 = ex.div_normal(ut, ex.rcp(ut + 1.));
  const int ret = newton_vsq_x(ex, x, x0, x1, gammafail, *niter, maxit, nst, nss, resume);
  if (ret == NEWTON_DEFERRED) return NEWTON_DEFERRED;
#pragma unroll
  for (int k = B1; k <= B3; k++) pr[k] = ex.div(Ut[k], ral);
  if (ret != 0) return ret * 100 + 1;
  W = x0;
  if (W == FAIL_VAL) return 1;
  if (ExactTiny::quot(W, ex.rcp(w0)) > W_TOO_BIG) return PF_CONVW;
  utsq = utsq_calc_x(ex, x, W);
  if ((utsq < 0.) && (fabs(utsq) < 1.0e-13)) utsq = fabs(utsq);
  if (utsq < 0. || utsq > utsq_too_big) return PF_CONVUTSQ2;
  const double gamma = ex.sqrt_of(1. + utsq);
  const double rho0 = ex.div_normal(x.D, ex.rcp(gamma));
  const double w = ExactTiny::quot(W, ex.rcp(gamma * gamma));
  const double p = ex.div_normal((gam - 1.) * (w - rho0), ex.rcp(gam));
  const double u = w - (rho0 + p);
  int pfl = 0;
  if ((rho0 <= 0.) || (u <= 0.)) {
    if ((rho0 <= 0.) && (u >= 0.)) pfl = PF_RHONEG;
    if ((rho0 >= 0.) && (u <= 0.)) pfl = PF_UNEG;
    if ((rho0 <= 0.) && (u <= 0.)) pfl = PF_RHOUNEG;
  }
  pr[RHO] = rho0;
  pr[UU] = u;
  const double WB = W + x.Bsq;
  const Recip r1 = ex.rcp(WB), r2 = ex.rcp(W * WB);
#pragma unroll
  for (int i = 1; i < 4; i++) {
    const double Qt = (SP && i > 1) ? Qcon[i] : Qcon[i] + (gn[i] * nlapse) * x.Qdotn;
    const double t1 = ex.div_normal(-gamma * Qt, r1), n2 = gamma * QdotB * B[i - 1];
    // the field's part is watched only where the other does not drown it
    ex.numerator((fabs(t1) > 1.e-150) ? 0. : n2);
    pr[U1 + i - 1] = t1 - ExactTiny::quot(n2, r2);
  }
  return pfl;
}

// utoprim_ffde and fixup1zone's Lorentz limit the same way
template <bool SP>
__device__ __forceinline__ void utoprim_ffde_x(ExactTiny& ex, const double* U, const double* c, const double* gn,
                                               double sg, double* pr, double gammamax)
{
  const Recip rs = ex.rcp(sg);
  double S[3], B[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    S[k] = ex.div(U[U1 + k], rs);
    B[k] = ex.div(U[B1 + k], rs);
  }
  const double alphasq = ExactTiny::quot(1., ex.rcp(-gn[0]));
  double bv[3];
  lower_space<SP>(B, c, bv);
  const double b1 = bv[0], b2 = bv[1], b3 = bv[2];
  const double Bsq = b1 * B[0] + b2 * B[1] + b3 * B[2];
  const double o = ExactTiny::quot(1., ex.rcp(Bsq * sg));
  const double E[3] = {(b2 * S[2] - b3 * S[1]) * o, (b3 * S[0] - b1 * S[2]) * o, (b1 * S[1] - b2 * S[0]) * o};
  double ev[3];
  lower_space<SP>(E, c, ev);
  const double e1 = ev[0], e2 = ev[1], e3 = ev[2];
  const double Esq = E[0] * e1 + E[1] * e2 + E[2] * e3;
  const double gammasq = ex.div_normal(Bsq, ex.rcp(Bsq - Esq));
  ex.need(gammasq <= gammamax * gammamax && gammasq >= 1.0);
  double v[4], uc[4];
  v[1] = alphasq * (-gn[1] + (e2 * b3 - e3 * b2) * o);
  v[2] = alphasq * (SP ? (e3 * b1 - e1 * b3) * o : -gn[2] + (e3 * b1 - e1 * b3) * o);
  v[3] = alphasq * (SP ? (e1 * b2 - e2 * b1) * o : -gn[3] + (e1 * b2 - e2 * b1) * o);
  const double d2 = SP ? c[1] * v[1] + c[3] * v[3] + c[6] * v[1] * v[3]
                       : c[1] * v[1] + c[2] * v[2] + c[3] * v[3] + c[5] * v[1] * v[2] + c[6] * v[1] * v[3] +
                             c[8] * v[2] * v[3];
  const double discr = +c[0] + c[4] * v[1] * v[1] + c[7] * v[2] * v[2] + c[9] * v[3] * v[3] + 2. * d2;
  uc[0] = ExactTiny::quot(1., ex.rcp(ex.sqrt_of(-discr)));
#pragma unroll
  for (int j = 1; j < 4; j++) pr[U1 - 1 + j] = v[j] * uc[0];
#pragma unroll
  for (int k = 0; k < 3; k++) pr[B1 + k] = B[k];
  ex.need(gammamax <= 1.0 || ex.sqrt_of(1. + qsq_x<SP>(pr, c)) <= gammamax);
}

// flux divergence with flux-CT B fluxes (step_ch.c:1403-1413)
template <typename FT>
__device__ __forceinline__ void flux_divergence(const StepArgs& a, int i, int j, long long z, double* dUr)
{
  const FT* F1 = reinterpret_cast<const FT*>(a.F1);
  const FT* F2 = reinterpret_cast<const FT*>(a.F2);
  const long long pl = a.gr.plane;
  const double idx1 = 1.0 / a.pp.dx1, idx2 = 1.0 / a.pp.dx2;
  const long long zi1 = a.gr.at(i + 1, j), zj1 = a.gr.at(i, j + 1), zij = a.gr.at(i + 1, j + 1);
  const double e00 = __ldg(a.emf + z), e10 = __ldg(a.emf + zi1), e01 = __ldg(a.emf + zj1), e11 = __ldg(a.emf + zij);
#pragma unroll
  for (int k = 0; k < NPR; k++) {
    double f1p, f1m, f2p, f2m;
    if (k == B1) {
      f1p = 0.;
      f1m = 0.;
      f2m = -0.5 * (e00 + e10);
      f2p = -0.5 * (e01 + e11);
    } else if (k == B2) {
      f1m = 0.5 * (e00 + e01);
      f1p = 0.5 * (e10 + e11);
      f2p = 0.;
      f2m = 0.;
    } else {
      f1p = __ldg(F1 + k * pl + zi1);
      f1m = __ldg(F1 + k * pl + z);
      f2p = __ldg(F2 + k * pl + zj1);
      f2m = __ldg(F2 + k * pl + z);
    }
    const double dU1 = (-(f1p - f1m) * idx1);
    const double dU2 = (-(f2p - f2m) * idx2);
    dUr[k] = dU1 + dU2;
  }
}

// source_conn, phys.c:520-619: acc[l] = sum_j sum_k T^j_k Gamma^k_{lj}, T row
// jj given, the connection planes in shared memory (sz, plane_s apart)
__device__ __forceinline__ void source_row(const double* row, int jj, const double* sz, int plane_s, double* acc)
{
#pragma unroll
  for (int l = 0; l < 4; l++)
#pragma unroll
    for (int k = 0; k < 4; k++) acc[l] += row[k] * sz[(conn_plane(k, l, jj) - GEO_CONN) * plane_s];
}

// a deferred (or, with the retry chain, failed) inversion goes to
// k_update_tail, so that this warp is not held for up to 200 iterations by
// one lane; -1 in the last state plane: to be solved afresh
__device__ __forceinline__ void defer_zone(const StepArgs& a, long long z, int pfl, const double* U)
{
  const long long pl = a.gr.plane;
  if (pfl != NEWTON_DEFERRED) a.fixbuf[(NEWTON_STATE - 1) * pl + z] = -1.0;
#pragma unroll
  for (int k = 0; k < NPR; k++) a.ubuf[k * pl + z] = U[k];
  a.worklist[atomicAdd(&a.sc->ndeferred, 1)] = (int)z;
}

// one zone's update by the general templates; returns its Newton iterations
// (the mixed form's update is this one too, in k_update_mixed's own text)
template <bool FFDE>
__device__ __noinline__ int update_general(const StepArgs& a, int i, int j, const double* pi, const double* pb,
                                           double* pf, double c2, const double* sz, int plane_s)
{
  const long long pl = a.gr.plane, z = a.gr.at(i, j);
  const double dt = a.sc->dt, gam = a.pp.gam;
  Geo<double> g;
  load_geo(a, CENT, z, g);
  double U[NPR], pfz[NPR], dUr[NPR], dUg[NPR];
  {
    // Ui = U(pi)
    double pr[NPR];
#pragma unroll
    for (int k = 0; k < NPR; k++) pr[k] = __ldg(pi + k * pl + z);
#pragma unroll
    for (int k = 0; k < NPR; k++) pfz[k] = pr[k];
    State<double> q;
    state_of(pr, g, q);
    flux_of<double, FFDE>(pr, q, 0, g, gam, U);
    if (a.bsqf_fused) a.bsqf_fused[z] = bsq_flag(a, pr, q);  // get_bsqflags of the step's p
  }
  flux_divergence<double>(a, i, j, z, dUr);
  {
    double pr[NPR];
#pragma unroll
    for (int k = 0; k < NPR; k++) pr[k] = __ldg(pb + k * pl + z);
    State<double> q;
    state_of(pr, g, q);
    double acc[4] = {0., 0., 0., 0.};
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      double row[4];
      mhd_row<double, FFDE>(pr, jj, q, gam, row);
      source_row(row, jj, sz, plane_s, acc);
    }
    dUg[RHO] = 0. + g.g * 0.;
    dUg[B1] = dUg[B2] = dUg[B3] = dUg[RHO];
#pragma unroll
    for (int l = 0; l < 4; l++) dUg[UU + l] = 0. + g.g * acc[l];
  }
  {
    // the RK combine of dUtoU, advance.c:273-286
    const double cdt = c2 * dt;
#pragma unroll
    for (int k = 0; k < NPR; k++) U[k] = 1.0 * U[k] + 0.0 * 0.0 + cdt * (dUr[k] + dUg[k]);
  }
  if constexpr (FFDE) {
    // Utoprim_ffde, then fixup1zone's Lorentz-factor limit (the floors are
    // GRMHD-only, fixup.c:293); pflag is left as it was
    int rc = utoprim_ffde(U, g, pfz, a.pp.gammamax);
    if (!rc) rc = limit_gamma(a.pp.gammamax, pfz, g);
    if (rc) report_fail(a.sc, a.phase0 + PH_UPDATE, rc, zone_order(i, j));
#pragma unroll
    for (int k = 0; k < NPR; k++) pf[k * pl + z] = pfz[k];
    return 0;
  } else {
    int niter;
    // a deferred solve leaves its Newton state in the repair scratch (idle
    // until k_fixup_compute), NEWTON_STATE planes
    const int pfl = utoprim_2d(U, g, pfz, gam, a.pp.gammafail, &niter, NEWTON_MAIN_CAP, a.fixbuf + z, pl);
    if (pfl == NEWTON_DEFERRED || (a.pp.tryagain && pfl != 0)) {
      defer_zone(a, z, pfl, U);
      return 0;
    }
    finish_zone(a, g, z, i, j, pfz, pfl, pf, sz[(GEO_FLOOR - GEO_CONN) * plane_s],
                sz[(GEO_FLOOR + 1 - GEO_CONN) * plane_s]);
    return niter;
  }
}

// block rows in launch order from both poles inward (0, last, 1, last-1,
// ...): the zones near the axis take the most Newton iterations, and started
// first their blocks no longer trail the kernel's last wave (developed 512^2
// flow: 0.5256-0.5309 against 0.5333-0.5366 ms a step)
__device__ __forceinline__ unsigned update_block_row()
{
  return (blockIdx.y & 1u) ? gridDim.y - 1u - (blockIdx.y >> 1) : (blockIdx.y >> 1);
}
// the block's connection and floor planes: issues the TMA copy (one thread)
__device__ __forceinline__ void update_geo_load(double* sgeo, const CUtensorMap* map, unsigned by, uint64_t* bar)
{
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    mbar_init(bar, 1);
    mbar_expect_tx(bar, (uint32_t)upd_smem_bytes(blockDim.x, blockDim.y));
    tma_load_3d(sgeo, map, (int)((blockIdx.x * blockDim.x + NG) & ~1u), (int)(by * blockDim.y + NG), GEO_CONN, bar);
  }
}
// Newton iteration count (the reference's nstroke), one atomic per warp
__device__ __forceinline__ void count_newton(const StepArgs& a, int niter)
{
  const unsigned mask = __activemask();
  const unsigned it = __reduce_add_sync(mask, (unsigned)niter);
  if ((int)(threadIdx.x & 31) == __ffs(mask) - 1) atomicAdd(&a.sc->newton_iters, (unsigned long long)it);
}

// advance_standard zone loop, advance.c:114-181, for one RK2 substep.
// CUf = {1, 0, c2}: Uf = Ui + c2*dt*dU; on the last substep unew = Uf.
// The connection coefficients and floors arrive by TMA (geo_map, a 3D map
// over the geometry block with the box above) while U(p_i) is formed; the
// block width is even.  Bound by memory latency, then by HBM (836 B a zone):
// every global load starts before anything is computed, without branches in
// between (harm_exact.cuh), at 168 registers (12 warps per SM; at 128 the
// loads come in small batches and 172 B of registers spill: 66.6 against 61.5
// us with the tail at 512^2).  A zone whose values leave the exact range goes
// to update_general.  512^2 developed flow, the kernel for any metric: 86 -> 50
// us (first substep) and 58 us (second), 3.9 TB/s; 1024^2 with the tail 300 ->
// 178 us.  The torus's and the star's metrics take the SP kernel: 49 and 53
// us, 1024^2 with the tail 160.
template <bool FFDE, bool SP>
__global__ void __launch_bounds__(128, 3) k_update(const __grid_constant__ StepArgs a,
                                                   const __grid_constant__ CUtensorMap geo_map,
                                                   const double* __restrict__ pi, const double* __restrict__ pb,
                                                   double* __restrict__ pf, double c2)
{
  extern __shared__ __align__(128) double sgeo[];
  __shared__ uint64_t bar;
  const unsigned by = update_block_row();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = by * blockDim.y + threadIdx.y;
  const int W = upd_box_w(blockDim.x);
  update_geo_load(sgeo, &geo_map, by, &bar);
  const bool active = (i < a.gr.n1 && j < a.gr.n2);
  const long long pl = a.gr.plane, z = a.gr.at(active ? i : 0, active ? j : 0);
  const double dt = a.sc->dt, gam = a.pp.gam;
  double c[10], gn[10], sg;
  double U[NPR], pfz[NPR], dUr[NPR];
  ExactTiny ex;
  StateX q;
  LapseX lp;
  unsigned char bf = 0;
  // the flux divergence first, while few registers are taken: its 28 loads
  // then start together (formed after U(pi), in small batches, they cost 20
  // of the kernel's 79 us at 512^2)
  flux_divergence<double>(a, active ? i : 0, active ? j : 0, z, dUr);
  {
    const double* base = a.geo + (long long)CENT * GEO_PER_LOC * pl + z;
#pragma unroll
    for (int k = 0; k < 10; k++) {
      if (!SP || !(SP_COV >> k & 1)) c[k] = __ldg(base + k * pl);
      if (!SP || !(SP_CON >> k & 1)) gn[k] = __ldg(base + (10 + k) * pl);
    }
    sg = __ldg(base + 20 * pl);
#pragma unroll
    for (int k = 0; k < NPR; k++) pfz[k] = __ldg(pi + k * pl + z);
  }
  // p_b is on its way meanwhile (asm: the compiler would load it at its use)
  double prb[NPR];
#pragma unroll
  for (int k = 0; k < NPR; k++) asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(prb[k]) : "l"(pb + k * pl + z));
  __syncthreads();  // the barrier is initialised before anyone polls it
  if (active) {
    if (SP) ex.need(__ldg(a.geo_full) == 0);  // (a geometry uploaded since the kernel was chosen)
    lp = lapse_x<SP>(ex, gn);
    state_x<SP>(ex, pfz, c, lp, 1.e300, q);
    // Ui = U(pi)
    conserved_x<FFDE>(pfz, q, sg, gam, U);
    if (a.bsqf_fused) bf = bsq_flag_x(ex, a, pfz, q.bsq);  // get_bsqflags of the step's p
  }
  if (!mbar_wait(&bar, 0)) {
    if (active) report_fail(a.sc, a.phase0 + PH_UPDATE, FAIL_TMA_TIMEOUT, zone_order(i, j));
    return;
  }
  if (!active) return;
  const int plane_s = blockDim.y * W;
  const double* sz = sgeo + threadIdx.y * W + threadIdx.x + 1;
  {
    // (the first substep's pb is pi, whose state is at hand)
    if (pb != pi) state_x<SP>(ex, prb, c, lp, 1.e300, q);
    const double r = FFDE ? 0. : prb[RHO], u = FFDE ? 0. : prb[UU], P = (gam - 1.) * u, w = P + r + u;
    const double eta = FFDE ? q.bsq : w + q.bsq, ptot = FFDE ? q.bsq * 0.5 : P + q.bsq * 0.5;
    double acc[4] = {0., 0., 0., 0.};
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      const double eu = eta * q.ucon[jj];
      double row[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        double t = eu * q.ucov[k];
        if (k == jj) t = t + ptot;
        row[k] = t - q.bcon[jj] * q.bcov[k];
      }
      source_row(row, jj, sz, plane_s, acc);
    }
    // the RK combine of dUtoU, advance.c:273-286
    const double cdt = c2 * dt;
#pragma unroll
    for (int k = 0; k < NPR; k++) {
      const double d = (k >= UU && k <= U3) ? dUr[k] + sg * acc[k - UU] : dUr[k];
      U[k] = (U[k] + 0.) + cdt * d;  // (+ 0., as dUtoU has it: no zero stays negative)
    }
  }
  if constexpr (FFDE) {
    utoprim_ffde_x<SP>(ex, U, c, gn, sg, pfz, a.pp.gammamax);
    if (!ex.ok()) {
      update_general<FFDE>(a, i, j, pi, pb, pf, c2, sz, plane_s);
      return;
    }
#pragma unroll
    for (int k = 0; k < NPR; k++) pf[k * pl + z] = pfz[k];
  } else {
    int niter;
    // a deferred solve leaves its Newton state in the repair scratch (idle
    // until k_fixup_compute), NEWTON_STATE planes
    const int pfl = utoprim_2d_x<SP>(ex, U, c, gn, sg, pfz, gam, a.pp.gammafail, &niter, NEWTON_MAIN_CAP, a.fixbuf + z, pl,
                                 false);
    if (!ex.ok()) {
      niter = update_general<FFDE>(a, i, j, pi, pb, pf, c2, sz, plane_s);
    } else {
      if (a.bsqf_fused) a.bsqf_fused[z] = bf;
      if (pfl == NEWTON_DEFERRED || (a.pp.tryagain && pfl != 0)) {
        defer_zone(a, z, pfl, U);
        niter = 0;
      } else {
        Geo<double> g;
#pragma unroll
        for (int k = 0; k < 10; k++) g.gcov[k] = (SP && (SP_COV >> k & 1)) ? 0. : c[k];
        finish_zone(a, g, z, i, j, pfz, pfl, pf, sz[(GEO_FLOOR - GEO_CONN) * plane_s],
                    sz[(GEO_FLOOR + 1 - GEO_CONN) * plane_s]);
      }
    }
    count_newton(a, niter);
  }
}

// launches a k_update instance (its dynamic shared memory limit raised to the
// largest box of the tile shapes harm_set_tiles accepts, an even width and at
// most 128 threads: 64 rows of 2)
inline void update_launch(void (*kern)(StepArgs, CUtensorMap, const double*, const double*, double*, double),
                          SmemLimit& limit, dim3 g, dim3 b, cudaStream_t s, const StepArgs& a, const CUtensorMap& map,
                          const double* pi, const double* pb, double* pf, double c2)
{
  limit.raise((const void*)kern, upd_smem_bytes(2, 64));
  kern<<<g, b, upd_smem_bytes(b.x, b.y), s>>>(a, map, pi, pb, pf, c2);
}

// ---------------------------------------------------------------- end of step
// diag_flux() for the global region's inner x1 face (diag.c:576-833): the
// face fluxes in diagnostic form (UtoU UEVOLVE->UDIAG) and the energy-
// equation stress terms 3 and 6 from the zone-centred state pr of row j.
template <typename FT>
__device__ __forceinline__ void horizon_terms(const StepArgs& a, const double* pr, int j, double* t4)
{
  const FT* F1 = reinterpret_cast<const FT*>(a.F1);
  const long long pl = a.gr.plane;
  const double surface = a.pp.dx2 * (2.0 * 3.14159265358979323846);
  const long long z = a.gr.at(0, j);
  const double gf = gdet_at(a, FACE1, z);
  const double Fr = (double)F1[RHO * pl + z] * surface, Fu = (double)F1[UU * pl + z] * surface;
  const double gr = Fr / gf;
  double gu = Fu / gf;
  gu += -gr;
  t4[0] = gr * gf;
  t4[1] = gu * gf;
  Geo<double> g;
  load_geo(a, CENT, z, g);
  State<double> q;
  state_of(pr, g, q);
  double bsq = 0;
#pragma unroll
  for (int l = 0; l < 4; l++) bsq += (q.bcon[l]) * (q.bcov[l]);
  const double surgdet = (g.g) * surface;
  t4[2] = bsq * (q.ucon[1]) * (q.ucov[0]) * surgdet;
  t4[3] = -(q.bcon[1]) * (q.bcov[0]) * surgdet;
}

// The end of a step in three parts.  step_sums, by every thread of one
// block, after the horizon terms of every row j sit in t[k * ts + j] (k < 4):
// their sums in j order as the reference's loop adds them (so the sums are
// exact), pcum += pdot * dt (diag.c:576-833).  step_dt, by one block: the new
// dt from the flux blocks' Courant minima (advance.c:190, step_ch.c:174-183).
// step_commit, one thread, after both and after everything that reads the
// step's scalars: t += dt and the new dt.  L2: the terms were written by other
// blocks of the same kernel (read past L1).
template <bool L2>
__device__ __forceinline__ void step_sums(const StepArgs& a, const double* t, long long ts)
{
  constexpr int CHUNK = 256;
  __shared__ double acc[4];
  __shared__ double stage[4][CHUNK + 1];  // rows one double apart in banks: the four adding lanes do not conflict
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
  const int n2 = a.gr.n2;
  // chunks of the four term rows are staged in shared memory by the whole
  // block (independent loads), then four threads add them one after another
  // in j order
  double s = 0.;
  for (int j0 = 0; j0 < n2; j0 += CHUNK) {
    const int m = (n2 - j0 < CHUNK) ? n2 - j0 : CHUNK;
#pragma unroll 8
    for (int q = tid; q < 4 * m; q += nt) {
      const int k = q / m, jj = q - k * m;
      const double* src = t + k * ts + j0 + jj;
      stage[k][jj] = L2 ? __ldcg(src) : *src;
    }
    __syncthreads();
    if (tid < 4) {
      const double* b = stage[tid];
      int q = 0;
      for (; q + 8 <= m; q += 8) {
        double v[8];
#pragma unroll
        for (int r = 0; r < 8; r++) v[r] = b[q + r];
#pragma unroll
        for (int r = 0; r < 8; r++) s += v[r];
      }
      for (; q < m; q++) s += b[q];
    }
    __syncthreads();
  }
  if (tid < 4) acc[tid] = s;
  __syncthreads();
  if (tid == 0) {
    DevScalars* sc = a.sc;
    for (int k = 0; k < 4; k++) sc->hz[k] = acc[k];
    sc->hz[4] += acc[0] * sc->dt;
    sc->hz[5] += acc[1] * sc->dt;
    sc->hz[6] += (acc[2] + acc[3]) * sc->dt;
  }
}

__device__ __forceinline__ void step_dt(const StepArgs& a)
{
  __shared__ double sh[2][32];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
  double m1 = 1.e9, m2 = 1.e9;
#pragma unroll 4
  for (int b = tid; b < a.nblocks_flux; b += nt) {
    double v1 = __ldcg(a.blockmin + b), v2 = __ldcg(a.blockmin + a.nblocks_flux + b);
    m1 = (v1 < m1) ? v1 : m1;
    m2 = (v2 < m2) ? v2 : m2;
  }
  m1 = block_min(m1, sh[0]);
  m2 = block_min(m2, sh[1]);
  if (tid == 0) a.sc->ndt = a.pp.defcon * 1. / (1. / m1 + 1. / m2);
}

__device__ __forceinline__ void step_commit(const StepArgs& a)
{
  DevScalars* s = a.sc;
  double ndt = __ldcg(&s->ndt);
  const bool moved = s->dt > 0.;
  s->t += s->dt;
  s->realnstep += 1;
  if (ndt > a.pp.safe * s->dt) ndt = a.pp.safe * s->dt;
  s->dt = ndt;
  if (moved) s->dt_free = ndt;  // a step at dt = 0 (past the end time) keeps the last one
  if (s->t + s->dt > a.pp.tf) s->dt = a.pp.tf - s->t;
}

// After the last substep, one block: the horizon terms of every row j (into
// the inversion scratch ubuf, idle by now), then the three parts.
constexpr int STEP_END_THREADS = 512;
template <typename FT>
__global__ void __launch_bounds__(STEP_END_THREADS) k_step_end(StepArgs a, const double* __restrict__ pv)
{
  const long long pl = a.gr.plane;
  for (int j = threadIdx.x; j < a.gr.n2; j += blockDim.x) {
    const long long z = a.gr.at(0, j);
    double pr[NPR], t4[4];
#pragma unroll
    for (int k = 0; k < NPR; k++) pr[k] = pv[k * pl + z];
    horizon_terms<FT>(a, pr, j, t4);
#pragma unroll
    for (int k = 0; k < 4; k++) a.ubuf[k * pl + j] = t4[k];
  }
  __syncthreads();
  step_sums<false>(a, a.ubuf, pl);
  step_dt(a);
  __syncthreads();
  if (threadIdx.x == 0) step_commit(a);
}

}  // namespace harm
