"""The FP32 faces for the sparse metric leave out products with its zeros; for
states that overflow FP32 or are infinite those products are not zero.  An
ensemble's FP32 faces use the form for any metric: a context's own step gives
the same bytes, NaN for NaN, from states full of such values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("kind", ["torus", "dipole"])
@pytest.mark.parametrize("lim,flux", [(3, 0), (4, 1)])
@pytest.mark.parametrize("gammamax", [25.0, 1.0])
@pytest.mark.parametrize("what,seed", [("huge", 1), ("huge", 2), ("huge", 3), ("infinite", 1)])
def test_both_forms(harm, kind, lim, flux, gammamax, what, seed):
    n1, n2 = 360, 300
    par = getattr(harm, kind + "_params")(n1, n2)
    geom = getattr(harm, kind + "_geometry")(par)
    r = np.random.default_rng(seed)
    p0 = np.zeros((n1 + 6, n2 + 6, 8))
    p0[..., 0] = 10.0 ** r.uniform(-5, 0, p0.shape[:2])
    p0[..., 1] = 0.1 * p0[..., 0]
    p0[..., 2:5] = r.uniform(-1, 1, p0[..., 2:5].shape)
    p0[..., 5:8] = r.uniform(-0.1, 0.1, p0[..., 5:8].shape)
    p0[r.random(p0.shape) < 0.2] = 0.0
    m = r.random(p0.shape) < 0.25
    m[..., :2] &= r.random(m[..., :2].shape) < 0.2
    lone = np.zeros(m.shape[:2], bool)
    lone[4::3, 4::3] = True  # between ordinary zones
    m &= lone[..., None]
    v = 10.0 ** r.uniform(10, 38, m.sum()) if what == "huge" else np.full(m.sum(), np.inf)
    p0[m] = v * r.choice([-1.0, 1.0], m.sum())
    opt = dict(eom=harm.EOM_FFDE, bc=harm.BC_STAR, omegastar=par.omegastar) if kind == "dipole" else {}
    h = [harm.HarmGPU(n1, n2, geom["dx1"], geom["dx2"], lim=lim, fluxmethod=flux, gam=par.gam, gammamax=gammamax,
                      precision=harm.PREC_MIXED, **opt) for _ in range(2)]
    for c in h:
        c.upload_geometry(geom["gcov"], geom["gcon"], geom["gdet"], geom["conn"], geom["floors"])
        c.set_prims(p0)
        c.bound_prims()
        c.set_time(0.0, 1e-30, 0)
    e = harm.Ensemble(h[:1])
    e.step(1)
    h[1].step_ch(1)
    st = e.sync(raise_on_fail=False)[0], h[1].sync(raise_on_fail=False)
    for a, b in zip(h[0].get_fluxes() + h[0].get_prims(), h[1].get_fluxes() + h[1].get_prims()):
        assert _same(a, b), np.argwhere(~((a == b) | (np.isnan(a) & np.isnan(b))))[:5].tolist()
    assert [st[0][k] for k in ("fail_code", "fail_i", "fail_j", "dt")] == [st[1][k] for k in ("fail_code", "fail_i", "fail_j", "dt")]
    e.close()
