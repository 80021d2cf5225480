"""The kernels for a metric with every entry, over the layouts of the face
kernel (a layer of 4-row blocks per direction, one layer of them, 8-row
blocks), for the torus and the force-free star: equal to the oracle bit for
bit.  The mixed form after a change of metric equals a context that never had
another, and stays near FP64."""
import numpy as np
import pytest

import harmtest as ht
from test_gpu_metric_forms import _full, _upload

pytestmark = pytest.mark.gpu


def _problem(harm, kind, n1, n2):
    par = getattr(harm, kind + "_params")(n1, n2)
    geom = getattr(harm, kind + "_geometry")(par)
    p0 = getattr(harm, kind + "_init")(par, geom)
    opt = dict(gam=par.gam, gammamax=par.gammamax)
    if kind == "dipole":
        opt.update(eom=1, bc=1, omegastar=par.omegastar)
    return geom, p0, opt


@pytest.mark.parametrize("kind,n1,n2,lim,flux,switch", [
    ("torus", 61, 37, 4, 0, 3), ("torus", 260, 260, 3, 1, 0), ("torus", 260, 260, 4, 0, 3), ("torus", 365, 365, 4, 1, 3),
    ("torus", 365, 365, 3, 0, 0), ("dipole", 64, 40, 3, 0, 0), ("dipole", 64, 40, 4, 1, 0), ("dipole", 260, 260, 4, 0, 0),
    ("dipole", 400, 350, 3, 1, 0)])
def test_equal_to_the_oracle(harm, kind, n1, n2, lim, flux, switch):
    geom, p0, opt = _problem(harm, kind, n1, n2)
    geom = _full(geom)
    opt.update(lim=lim, fluxmethod=flux, fluxadjust=switch)
    o = ht.Oracle(n1, n2, geom, dx1=geom["dx1"], dx2=geom["dx2"], **opt)
    po = o.bound(p0)
    fo = np.zeros(po.shape[:2] + (5,), dtype=np.int32)
    h = harm.HarmGPU(n1, n2, geom["dx1"], geom["dx2"], **opt)
    _upload(h, geom)
    h.set_prims(p0)
    h.bound_prims()
    t, dt = 0.0, 1e-5
    h.set_time(t, dt, 0)
    for _ in range(2):
        rc, t, dt = o.step(po, fo, t, dt)
        assert rc == 0
    h.step_ch(2)
    st = h.sync()
    pg, fg = h.get_prims()
    assert np.array_equal(pg, po) and (st["t"], st["dt"]) == (t, dt)
    assert np.array_equal(ht.interior(fg)[..., 0], ht.interior(fo)[..., 0])
    for a, b in zip(h.get_fluxes(), o.fluxes()):
        assert np.array_equal(ht.interior(a), ht.interior(b))
    h.close()


@pytest.mark.parametrize("kind,n1,n2,lim,flux", [("torus", 61, 37, 4, 1), ("torus", 365, 365, 3, 1), ("dipole", 96, 64, 3, 0)])
def test_mixed_form_after_a_change_of_metric(harm, kind, n1, n2, lim, flux):
    sparse, p0, opt = _problem(harm, kind, n1, n2)
    full = _full(sparse)

    def run(geoms, precision):
        h = harm.HarmGPU(n1, n2, full["dx1"], full["dx2"], lim=lim, fluxmethod=flux, precision=precision, **opt)
        for g in geoms:
            _upload(h, g)
            h.set_prims(p0)
            h.bound_prims()
            h.set_time(0.0, 1e-5, 0)
            h.step_ch(5)
            st = h.sync()
        p = h.get_prims()[0]
        h.close()
        return p, st["t"], st["dt"]

    p, t, dt = run([sparse, full], harm.PREC_MIXED)
    fresh = run([full], harm.PREC_MIXED)
    assert np.array_equal(p, fresh[0]) and (t, dt) == fresh[1:]
    # five steps' rounding of FP32 fluxes (6e-8 each) on steps of dt ~ 1e-5
    exact = run([full], harm.PREC_FP64)[0]
    for k in (0, 1, 5, 6):
        a, b = ht.interior(p)[..., k], ht.interior(exact)[..., k]
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b) + 1e-300, k
