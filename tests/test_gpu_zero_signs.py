"""A zero of the FP64 primitives has the oracle's sign (a dump shows it): the
bytes of the state are compared, not its values, from states with zeros of
either sign and fields down to the smallest subnormal numbers, where fluxes,
conserved fields and quotients become zero."""
import numpy as np
import pytest

import harmtest as ht

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lim,flux,switch", [(3, 1, 0), (4, 0, 0), (4, 1, 3), (3, 0, 3)])
@pytest.mark.parametrize("seed", [1, 2])
def test_signs_of_the_primitives_zeros(harm, lim, flux, switch, seed):
    n1, n2 = 70, 45
    par = harm.torus_params(n1, n2)
    geom = harm.torus_geometry(par)
    p0 = harm.torus_init(par, geom)
    r = np.random.default_rng(seed)
    for k in range(4, 8):
        m = r.random(p0.shape[:2])
        p0[..., k] = np.where(m < 0.3, np.where(m < 0.15, -0.0, 0.0),
                              np.where(m < 0.6, np.ldexp(r.uniform(-1, 1, m.shape), r.integers(-1080, -1000, m.shape)),
                                       p0[..., k]))
    o = ht.Oracle(n1, n2, geom, lim=lim, fluxmethod=flux, fluxadjust=switch, dx1=geom["dx1"], dx2=geom["dx2"])
    po = o.bound(p0)
    fo = np.zeros(po.shape[:2] + (5,), dtype=np.int32)
    h = harm.HarmGPU(n1, n2, geom["dx1"], geom["dx2"], lim=lim, fluxmethod=flux, fluxadjust=switch)
    h.upload_geometry(geom["gcov"], geom["gcon"], geom["gdet"], geom["conn"], geom["floors"])
    h.set_prims(p0)
    h.bound_prims()
    t, dt = 0.0, 1e-3
    h.set_time(t, dt, 0)
    for _ in range(3):
        rc, t, dt = o.step(po, fo, t, dt)
        assert rc == 0
        h.step_ch(1)
        h.sync()
        pg = h.get_prims()[0]
        assert np.array_equal(pg, po)
        assert np.array_equal(pg.view(np.uint64), po.view(np.uint64)), np.argwhere(np.signbit(pg) != np.signbit(po))[:4].tolist()
    h.close()
