"""FP64 fluxes of states whose density or internal energy is infinite, not a
number or near the end of the range, with either solver: equal to the
oracle's, NaN for NaN (a flux form that the solver's choice weighs with zero
still spoils the flux where it is infinite).  The force-free step carries such
values along, as does the first substep of the torus."""
import numpy as np
import pytest

import harmtest as ht

pytestmark = pytest.mark.gpu
VALUES = [np.inf, -np.inf, np.nan, 1e305, -1e305, 1e200, -1e200, -1e120]


@pytest.mark.parametrize("kind", ["dipole", "torus"])
@pytest.mark.parametrize("lim,flux,switch", [(3, 0, 0), (4, 0, 3), (4, 1, 0), (3, 1, 3)])
@pytest.mark.parametrize("what", [0, 1])
def test_fluxes(harm, kind, lim, flux, switch, what):
    n1, n2 = 45, 30
    par = getattr(harm, kind + "_params")(n1, n2)
    geom = getattr(harm, kind + "_geometry")(par)
    p0 = getattr(harm, kind + "_init")(par, geom)
    opt = dict(lim=lim, fluxmethod=flux, fluxadjust=switch, gam=par.gam, gammamax=par.gammamax)
    if kind == "dipole":
        opt.update(eom=1, bc=1, omegastar=par.omegastar)
    r = np.random.default_rng(10 * lim + flux)
    m = np.zeros(p0.shape[:2], bool)
    m[3 + 4:n1:7, 3 + 3:n2:7] = True  # every one surrounded by ordinary zones
    p0[m, what] = r.choice(VALUES, m.sum())
    if kind == "torus":  # a field there and around, so that the wavespeeds stay finite
        p0[..., 5:8] = 0.01 * r.uniform(0.5, 1.0, p0[..., 5:8].shape)
    o = ht.Oracle(n1, n2, geom, dx1=geom["dx1"], dx2=geom["dx2"], **opt)
    po = o.bound(p0)
    fo = np.zeros(po.shape[:2] + (5,), dtype=np.int32)
    o.step(po, fo, 0.0, 1e-5)
    h = harm.HarmGPU(n1, n2, geom["dx1"], geom["dx2"], **opt)
    h.upload_geometry(geom["gcov"], geom["gcon"], geom["gdet"], geom["conn"], geom["floors"])
    h.set_prims(p0)
    h.bound_prims()
    h.set_time(0.0, 1e-5, 0)
    h.step_ch(1)
    st = h.sync(raise_on_fail=False)
    if o.fail()[0] == 0:
        for a, b in zip(h.get_fluxes(), o.fluxes()):
            a, b = ht.interior(a), ht.interior(b)
            assert np.array_equal(a, b, equal_nan=True), np.argwhere(~((a == b) | (np.isnan(a) & np.isnan(b))))[:5].tolist()
    assert (st["fail_code"] != 0) == (o.fail()[0] != 0)
    h.close()
