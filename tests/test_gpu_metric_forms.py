"""The kernels for a metric that couples x2 to nothing (the torus's and the
star's) and those for any metric: both equal the oracle bit for bit, also when
a context, or a member of an ensemble whose graph exists, gets a metric of the
other form."""
import numpy as np
import pytest

import harmtest as ht

pytestmark = pytest.mark.gpu
N1, N2 = 45, 21


def _full(geom):
    """The same tables with small x2 and t-phi entries everywhere."""
    g = {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in geom.items()}
    r = np.random.default_rng(3)
    for t in ("gcov", "gcon"):
        for i, j in ((0, 2), (0, 3), (1, 2), (2, 3)):
            d = 1e-4 * r.uniform(-1, 1, g[t].shape[:3]) * np.sqrt(np.abs(g[t][..., i, i] * g[t][..., j, j]))
            g[t][..., i, j] += d
            g[t][..., j, i] = g[t][..., i, j]
    return g


def _upload(h, g):
    h.upload_geometry(g["gcov"], g["gcon"], g["gdet"], g["conn"], g["floors"])


def _start(h, p0):
    h.set_prims(p0)
    h.bound_prims()
    h.set_time(0.0, 1e-5, 0)


def _oracle(g, p0, lim, flux, nsteps):
    o = ht.Oracle(N1, N2, g, lim=lim, fluxmethod=flux, dx1=g["dx1"], dx2=g["dx2"])
    p = o.bound(p0)
    f = np.zeros(p.shape[:2] + (5,), dtype=np.int32)
    t, dt = 0.0, 1e-5
    for _ in range(nsteps):
        rc, t, dt = o.step(p, f, t, dt)
        assert rc == 0
    return p, t, dt


@pytest.mark.parametrize("lim,flux", [(3, 0), (4, 1)])
def test_both_forms_and_a_change_of_form(harm, lim, flux):
    par = harm.torus_params(N1, N2)
    sparse = harm.torus_geometry(par)
    full, p0 = _full(sparse), harm.torus_init(par, sparse)
    h = harm.HarmGPU(N1, N2, sparse["dx1"], sparse["dx2"], lim=lim, fluxmethod=flux)
    for g in (sparse, full, sparse):
        _upload(h, g)
        _start(h, p0)
        h.step_ch(4)
        st = h.sync()
        p, t, dt = _oracle(g, p0, lim, flux, 4)
        assert np.array_equal(h.get_prims()[0], p) and (st["t"], st["dt"]) == (t, dt)
    h.close()


def test_ensemble_member_changes_form(harm):
    par = harm.torus_params(N1, N2)
    sparse = harm.torus_geometry(par)
    full, p0 = _full(sparse), harm.torus_init(par, sparse)
    m = [harm.HarmGPU(N1, N2, sparse["dx1"], sparse["dx2"], lim=4, fluxmethod=1) for _ in range(2)]
    for h in m:
        _upload(h, sparse)
    e = harm.Ensemble(m, steps_per_launch=2)
    _upload(m[1], full)
    for h in m:
        _start(h, p0)
    e.step(4)
    e.sync()
    for h, g in zip(m, (sparse, full)):
        assert np.array_equal(h.get_prims()[0], _oracle(g, p0, 4, 1, 4)[0])
    e.close()


def test_mixed_forms_agree(harm):
    """An ensemble's FP32 faces use the form for any metric, a context's own
    step the sparse one: the same bits."""
    par = harm.torus_params(N1, N2)
    g = harm.torus_geometry(par)
    p0 = harm.torus_init(par, g)
    m = [harm.HarmGPU(N1, N2, g["dx1"], g["dx2"], lim=4, fluxmethod=1, precision=harm.PREC_MIXED) for _ in range(2)]
    for h in m:
        _upload(h, g)
        _start(h, p0)
    e = harm.Ensemble(m[:1], steps_per_launch=3)
    e.step(30)
    e.sync()
    m[1].step_ch(30)
    m[1].sync()
    assert np.array_equal(m[0].get_prims()[0], m[1].get_prims()[0])
    e.close()
