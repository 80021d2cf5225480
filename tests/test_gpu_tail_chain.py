"""The retry chain inside the step (k_update_tail_chain: a failed zone's methods
side by side) leaves the state that running them one after another left:
SHA-256 of the primitives (zeros without sign) after runs from init of the
one-thread-per-zone chain, itself equal to the reference built with
UTOPRIMTRYAGAIN 1.  The runs rescue failures by 5D1 (the first two) and hold
zones that fail every method (the last, 344 repairs)."""
import hashlib

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,lim,flux,nsteps,fixups,newton,sha", [
    (32, 32, 3, 1, 25, 0, 155672, "a7720fb131ffcc18ed0296260fffada5"),
    (96, 64, 4, 1, 40, 0, 1469132, "f629dbbae3b8aa59fa0b8bb766d5490a"),
    (245, 131, 4, 0, 230, 344, 46647513, "7ef4a011bd60fab04a0fa3e70512c864"),
])
def test_chain_in_the_step(harm, n1, n2, lim, flux, nsteps, fixups, newton, sha):
    h, _, _ = harm.torus_context(n1, n2, lim=lim, fluxmethod=flux, tryagain=True)
    h.step_ch(nsteps)
    st = h.sync()
    p, _ = h.get_prims()
    h.close()
    assert (st["fixups"], st["newton_iters"]) == (fixups, newton)
    assert hashlib.sha256((p + 0.0).tobytes()).hexdigest()[:32] == sha
