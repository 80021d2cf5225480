// One side of an FP32 face by the form for a sparse metric and by the form for
// any metric, on the host: the Lorentz limit, the state, the fluxes and the
// wavespeeds.  What the sparse form's faces rely on is reported a state:
// bit 0: b^2 is finite (the sparse form is used); bit 1: then both forms give
// the same; bit 2: else the general form gives the same from the state that
// the sparse Lorentz limit left as from its own.
#include <math.h>
#include <string.h>

#include "../harm_ramt_b200/csrc/harm_device.cuh"

using namespace harm;

struct Side {
  float F[NPR], U[NPR], vmax, vmin;
  int rc;
};

static bool same(float a, float b) { return a == b || (isnan(a) && isnan(b)); }

template <bool FFDE, bool SP>
static void side(const float* p, const Geo<float>& g, int dir, float gam, int rc, Side& x)
{
  State<float> q;
  state_of<float, SP>(p, g, q);
  flux_of<float, FFDE>(p, q, dir, g, gam, x.F);
  flux_of<float, FFDE>(p, q, 0, g, gam, x.U);
  x.vmax = x.vmin = 0.f;
  x.rc = rc ? rc : vchar_of<float, SP>(p, q, dir, g, gam, x.vmax, x.vmin);
}

static bool equal(const Side& a, const Side& b)
{
  bool ok = a.rc == b.rc && same(a.vmax, b.vmax) && same(a.vmin, b.vmin);
  for (int k = 0; k < NPR; k++) ok = ok && same(a.F[k], b.F[k]) && same(a.U[k], b.U[k]);
  return ok;
}

template <bool FFDE>
static unsigned char one(const float* p, const Geo<float>& g, int dir, float gammamax, float gam)
{
  float ps[NPR], pg[NPR];
  memcpy(ps, p, sizeof ps);
  memcpy(pg, p, sizeof pg);
  const int rs = limit_gamma<float, true>(gammamax, ps, g), rg = limit_gamma<float, false>(gammamax, pg, g);
  Side general, s;
  side<FFDE, false>(pg, g, dir, gam, rg, general);
  State<float> q;
  state_of<float, true>(ps, g, q);
  const bool finite = fabs(dot4(q.bcon, q.bcov)) <= 3.402823466e38f;
  if (finite) side<FFDE, true>(ps, g, dir, gam, rs, s);
  else side<FFDE, false>(ps, g, dir, gam, rs, s);
  return (finite ? 1 : 0) | (equal(general, s) ? (finite ? 2 : 4) : 0);
}

extern "C" void sparse_sides(int n, const float* p, const float* gcov, const float* gcon, const float* gdet,
                             const int* dir, float gammamax, float gam, int ffde, unsigned char* out)
{
  for (int k = 0; k < n; k++) {
    Geo<float> g;
    memcpy(g.gcov, gcov + 10 * k, sizeof g.gcov);
    memcpy(g.gcon, gcon + 10 * k, sizeof g.gcon);
    g.g = gdet[k];
    out[k] = ffde ? one<true>(p + NPR * k, g, dir[k], gammamax, gam) : one<false>(p + NPR * k, g, dir[k], gammamax, gam);
  }
}
