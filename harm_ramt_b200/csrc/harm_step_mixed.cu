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
    conserved_general<FFDE>(a, z, g, pi, pfz, U);
    flux_divergence<float>(a, i, j, z, dUr);
  }
  if (!mbar_wait(&bar, 0)) {
    if (active) report_fail(a.sc, a.phase0 + PH_UPDATE, FAIL_TMA_TIMEOUT, zone_order(i, j));
    return;
  }
  if (!active) return;
  const int plane_s = blockDim.y * W;
  const double* sz = sgeo + threadIdx.y * W + threadIdx.x + 1;
  source_general<FFDE>(a, z, g, pb, sz, plane_s, dUg);
  combine_general(c2 * dt, dUr, dUg, U);
  const int niter = invert_general<FFDE>(a, i, j, z, g, U, pfz, pf, sz, plane_s);
  if (!FFDE) count_newton(a, niter);
}

void launch_update_mixed(int ffde, dim3 g, dim3 b, cudaStream_t s, const StepArgs& a, const CUtensorMap& map,
                         const double* pi, const double* pb, double* pf, double c2)
{
  auto kern = ffde ? k_update_mixed<true> : k_update_mixed<false>;
  static bool attr[2] = {false, false};
  update_launch(kern, attr[ffde != 0], g, b, s, a, map, pi, pb, pf, c2);
}

}  // namespace harm
