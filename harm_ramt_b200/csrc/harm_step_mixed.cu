// Mixed-precision instantiations of the step kernels: FP32 interface states,
// wavespeeds and face fluxes (FP32 face geometry, FP32 flux storage), with
// the con-to-prim solve, conserved update, geometric source, EMF and dt in
// FP64.  This translation unit is built with multiply-add contraction and
// fast FP32 division and square root; it is not bit-identical to the
// reference (harm_step.cu is).
#include "harm_step_impl.cuh"

namespace harm {

template <bool SP>
static void flux_fp32(int para, int ffde, dim3 g, dim3 b, cudaStream_t s, const StepArgs& a, const CUtensorMap& prim_map)
{
  if (ffde) {
    if (para) flux_rows_launch<float, true, true, SP>(g, b, s, a, prim_map);
    else flux_rows_launch<float, false, true, SP>(g, b, s, a, prim_map);
  } else if (para) flux_rows_launch<float, true, false, SP>(g, b, s, a, prim_map);
  else flux_rows_launch<float, false, false, SP>(g, b, s, a, prim_map);
}

void launch_flux_mixed(int para, int ffde, dim3 g, dim3 b, cudaStream_t s, const StepArgs& a,
                       const CUtensorMap& prim_map)
{
  if (a.sparse32) flux_fp32<true>(para, ffde, g, b, s, a, prim_map);
  else flux_fp32<false>(para, ffde, g, b, s, a, prim_map);
}

void launch_emf_mixed(dim3 g, dim3 b, cudaStream_t s, const StepArgs& a, const double* pv)
{
  k_emf<float><<<g, b, 0, s>>>(a, pv);
}

// k_update of the mixed form (the zone update after FP32 fluxes).  Its FP64
// sums are contracted as the compiler finds them, which depends on the text
// and on the registers allowed (three blocks per SM instead of four: other
// bits), and a run from the initial state magnifies another choice to 1e-4
// within some tens of steps.  So this kernel stays as it is while k_update is
// the branch-free one: k_update's text here (a mixed step of the 512^2 torus
// 244 us, of the 512 x 256 dipole 88) gave other results than this one (324
// and 104); starting every load first gave the same ones and no gain (330
// and 102).
template <bool FFDE>
__global__ void __launch_bounds__(128, 4) k_update_mixed(StepArgs a, const __grid_constant__ CUtensorMap geo_map,
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
  __syncthreads();  // the barrier is initialised before anyone polls it
  const bool active = (i < a.gr.n1 && j < a.gr.n2);
  const long long pl = a.gr.plane, z = a.gr.at(active ? i : 0, active ? j : 0);
  const double dt = a.sc->dt, gam = a.pp.gam;
  Geo<double> g;
  double U[NPR], pfz[NPR], dUr[NPR], dUg[NPR];
  if (active) {
    load_geo(a, CENT, z, g);
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
    flux_divergence<float>(a, i, j, z, dUr);
  }
  if (!mbar_wait(&bar, 0)) {
    if (active) report_fail(a.sc, a.phase0 + PH_UPDATE, FAIL_TMA_TIMEOUT, zone_order(i, j));
    return;
  }
  if (!active) return;
  const int plane_s = blockDim.y * W;
  const double* sz = sgeo + threadIdx.y * W + threadIdx.x + 1;
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
  } else {
    int niter;
    const int pfl = utoprim_2d(U, g, pfz, gam, a.pp.gammafail, &niter, NEWTON_MAIN_CAP, a.fixbuf + z, pl);
    if (pfl == NEWTON_DEFERRED || (a.pp.tryagain && pfl != 0)) {
      defer_zone(a, z, pfl, U);
      niter = 0;
    } else {
      finish_zone(a, g, z, i, j, pfz, pfl, pf, sz[(GEO_FLOOR - GEO_CONN) * plane_s],
                  sz[(GEO_FLOOR + 1 - GEO_CONN) * plane_s]);
    }
    count_newton(a, niter);
  }
}

void launch_update_mixed(int ffde, dim3 g, dim3 b, cudaStream_t s, const StepArgs& a, const CUtensorMap& map,
                         const double* pi, const double* pb, double* pf, double c2)
{
  auto kern = ffde ? k_update_mixed<true> : k_update_mixed<false>;
  static SmemLimit limit[2];
  update_launch(kern, limit[ffde != 0], g, b, s, a, map, pi, pb, pf, c2);
}

}  // namespace harm
