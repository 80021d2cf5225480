"""The FP64 face kernel at the edges of its blocks (31 faces x 8 or 4 rows) and
over the whole exponent range: equal to the oracle bit for bit on grids one
off its tile sizes, and from states whose fields and azimuthal velocity run
from ordinary values down to the smallest subnormal numbers and zero (every
form of its quotients, in the same warps and alone)."""
import numpy as np
import pytest

import harmtest as ht

pytestmark = pytest.mark.gpu


def _run(harm, n1, n2, lim, flux, nsteps, change=None):
    par = harm.torus_params(n1, n2)
    geom = harm.torus_geometry(par)
    p0 = harm.torus_init(par, geom)
    if change is not None:
        change(p0)
    o = ht.Oracle(n1, n2, geom, lim=lim, fluxmethod=flux, dx1=geom["dx1"], dx2=geom["dx2"])
    po = o.bound(p0)
    fo = np.zeros(po.shape[:2] + (5,), dtype=np.int32)
    h = harm.HarmGPU(n1, n2, geom["dx1"], geom["dx2"], lim=lim, fluxmethod=flux)
    h.upload_geometry(geom["gcov"], geom["gcon"], geom["gdet"], geom["conn"], geom["floors"])
    h.set_prims(p0)
    h.bound_prims()
    t, dt = 0.0, 1e-5
    h.set_time(t, dt, 0)
    for s in range(nsteps):
        rc, t, dt = o.step(po, fo, t, dt)
        assert rc == 0
        h.step_ch(1)
        st = h.sync()
        pg, fg = h.get_prims()
        assert np.array_equal(pg, po), f"step {s + 1}: {np.argwhere(pg != po)[:4].tolist()}"
        assert np.array_equal(ht.interior(fg)[..., 0], ht.interior(fo)[..., 0])
        assert st["t"] == t and st["dt"] == dt
    h.close()


@pytest.mark.parametrize("n1,n2", [(4, 4), (29, 6), (30, 7), (31, 8), (32, 9), (61, 5), (62, 14), (93, 31), (300, 130)])
@pytest.mark.parametrize("lim,flux", [(3, 0), (4, 1)])
def test_block_edges(harm, n1, n2, lim, flux):
    _run(harm, n1, n2, lim, flux, 4)


@pytest.mark.parametrize("lim,flux", [(3, 1), (4, 0), (4, 1)])
@pytest.mark.parametrize("mode", ["mixed", "rows", "columns"])
def test_tiny_numbers(harm, lim, flux, mode):
    def change(p):
        r = np.random.default_rng(5)
        n1, n2 = p.shape[:2]
        e = {"mixed": r.integers(-1080, -1, (n1, n2)), "rows": np.linspace(-1085, -20, n2)[None, :] * np.ones((n1, 1)),
             "columns": np.linspace(-20, -1085, n1)[:, None] * np.ones((1, n2))}[mode].astype(int)
        for k in (4, 5, 6, 7):
            p[..., k] = np.ldexp(r.uniform(-1, 1, (n1, n2)), e)
        p[r.random((n1, n2)) < 0.1, 5:8] = 0.0

    _run(harm, 64, 48, lim, flux, 3, change)
