"""Adjoint runs with many checkpoint segments launch captured steps, short
ones issue their kernels one by one: the same objective, dt sequence and
final state, and the same gradient but for the order in which a step's
contributions to a zone are added (each sum of some ten terms rounds
differently by 1e-15, over 65 steps: 1e-12 is allowed), at either side of
the line between the two (16 launches of a slot's step), with a shorter last
segment, and for a second call of the same context."""
import numpy as np
import pytest

from test_gpu_adjoint import _ctx, _developed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsteps,ckpt", [(30, 1), (31, 1), (40, 1), (65, 2), (66, 2)])
def test_captured_and_issued_steps_agree(harm, nsteps, ckpt):
    n = 32
    geom, p, dt = _developed(harm, n, 40)
    lam = np.random.default_rng(nsteps).standard_normal(p.shape)
    run = {}
    for c in (ckpt, nsteps, 7):  # 7: ten segments at most
        h = _ctx(harm, n, geom, p, dt)
        run[c] = h.adjoint(nsteps, c, 1.0, 1.0, lam)[:3] + (h.get_prims()[0],)
        if c == ckpt:
            h.set_prims(p)
            h.set_time(0.0, dt, 0)
            again = h.adjoint(nsteps, c, 1.0, 1.0, lam)
        h.close()
    J, grad, dts, last = run[nsteps]
    assert np.isfinite(grad).all() and np.abs(grad).max() > 0
    for Jc, gc, dc, lc in (run[ckpt], run[7], again[:3] + (last,)):
        assert Jc == J and np.array_equal(dc, dts) and np.array_equal(lc, last)
        assert np.linalg.norm(gc - grad) <= 1e-12 * np.linalg.norm(grad)
