"""The FP32 faces' form for a sparse metric against the form for any metric, a
side at a time on the host: equal wherever b^2 is finite, and elsewhere the
general form from the state after the sparse Lorentz limit equals the general
form all the way, over ordinary states and states that overflow or hold
infinities and NaN, on every face of a torus's and a star's grid."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC, LIB = os.path.join(HERE, "sparse_sides.cu"), os.path.join(HERE, "_build", "libsparse_sides.so")
pytestmark = pytest.mark.skipif(shutil.which("/usr/local/cuda/bin/nvcc") is None, reason="needs nvcc")
N = 100000


def _lib():
    dev = os.path.join(HERE, "..", "harm_ramt_b200", "csrc", "harm_device.cuh")
    if not os.path.exists(LIB) or any(os.path.getmtime(f) > os.path.getmtime(LIB) for f in (SRC, dev)):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        tmp = LIB + ".tmp%d" % os.getpid()
        subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17",
                        "--fmad=false", "-Xcompiler", "-fPIC,-ffp-contract=off", "-shared", "-o", tmp, SRC], check=True)
        os.replace(tmp, LIB)
    return ctypes.CDLL(LIB)


def _states(r, what):
    p = np.empty((N, 8), np.float32)
    p[:, 0] = 10.0 ** r.uniform(-5, 0, N)
    p[:, 1] = 0.1 * p[:, 0]
    p[:, 2:5] = r.uniform(-1, 1, (N, 3)) * 10.0 ** r.uniform(-1, 1, (N, 1))
    p[:, 5:8] = r.uniform(-0.1, 0.1, (N, 3))
    p[r.random((N, 8)) < 0.2] = 0.0
    m = r.random((N, 8)) < {"ordinary": 0.0, "one": 0.0}.get(what, 0.25)
    m[:, :2] &= r.random((N, 2)) < 0.2
    if what == "one":
        m[np.arange(N), r.integers(2, 8, N)] = True
    k = m.sum()
    v = {"huge": 10.0 ** r.uniform(10, 38, k), "nan": np.full(k, np.nan)}.get(what, np.full(k, np.inf))
    p[m] = v * r.choice([-1.0, 1.0], k)
    return p


@pytest.mark.parametrize("kind", ["torus", "dipole"])
@pytest.mark.parametrize("gammamax", [25.0, 1.0])
@pytest.mark.parametrize("what", ["ordinary", "huge", "infinite", "one", "nan"])
def test_both_forms(kind, gammamax, what):
    import harm_ramt_b200 as hb
    par = getattr(hb, kind + "_params")(64, 48)
    g = getattr(hb, kind + "_geometry")(par)
    r = np.random.default_rng(3)
    i, j, dirs = r.integers(0, 70, N), r.integers(0, 54, N), r.integers(1, 3, N).astype(np.int32)
    tri = [(a, b) for a in range(4) for b in range(a, 4)]
    at = (i, j, dirs - 1)
    with np.errstate(over="ignore"):
        gcov = np.stack([g["gcov"][at + t] for t in tri], 1).astype(np.float32)
        gcon = np.stack([g["gcon"][at + t] for t in tri], 1).astype(np.float32)
        gdet = g["gdet"][at].astype(np.float32)
    assert not gcov[:, [2, 5, 8]].any() and not gcon[:, [2, 3, 5, 8]].any()
    out = np.empty(N, np.uint8)
    p = _states(r, what)
    ptr = [x.ctypes.data_as(ctypes.c_void_p) for x in (p, gcov, gcon, gdet, dirs, out)]
    _lib().sparse_sides(N, *ptr[:5], ctypes.c_float(gammamax), ctypes.c_float(par.gam), int(kind == "dipole"), ptr[5])
    finite = (out & 1).astype(bool)
    assert (what == "one" or finite.any()) and (what == "ordinary" or not finite.all())
    assert (out[finite] == 3).all(), (p[finite & (out != 3)][:3].tolist())
    assert (out[~finite] == 4).all(), (p[~finite & (out != 4)][:3].tolist())
