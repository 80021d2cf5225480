"""The branch-free quotients and roots of the FP64 kernels (harm_exact.cuh)
round as IEEE division and square root do: equal to the operators for every
operand reported in range, on the host with seeds a few units off and on the
device with its own approximations; operands out of range are reported."""
import shutil

import numpy as np
import pytest

import exact_cases as ec

needs_nvcc = pytest.mark.skipif(shutil.which("/usr/local/cuda/bin/nvcc") is None, reason="needs nvcc")
PLACES = [pytest.param("host", n, marks=needs_nvcc) for n in (1, 2, 3)] + [
    pytest.param("device", 0, marks=pytest.mark.gpu)]


@pytest.mark.parametrize("where,nudge", PLACES)
def test_quotients(where, nudge):
    for name, a, b in ec.operand_sets():
        q, ok = ec.evaluate(where, False, a, b, nudge)
        assert ok.all(), name
        assert np.array_equal(q, a / b), name


@pytest.mark.parametrize("where,nudge", PLACES)
def test_quotients_of_tiny_numbers(where, nudge):
    r = np.random.default_rng(9)
    n = 1 << 20
    a, b = ec.hard_quotients(500)
    sets = [(a * 2.0 ** -60, b)]
    # numerators and quotients across the subnormal range, and exact ties of it
    sets += [(a * 2.0 ** -k, b * 2.0 ** s) for k in range(1075, 1130, 3) for s in (-1, 0, 1, 5)]
    sets += [(r.uniform(1, 2, n) * 2.0 ** r.integers(-1074, -960, n), r.uniform(1, 2, n) * 2.0 ** r.integers(-40, 40, n))]
    sets += [(r.integers(-4000, 4000, n) * 5e-324, r.integers(1, 64, n).astype(float))]
    sets += [(r.uniform(1, 2, n) * 2.0 ** r.integers(-960, 190, n), r.uniform(1, 2, n) * 2.0 ** r.integers(-200, 60, n))]
    for a, b in sets:
        q, ok = ec.evaluate(where, 2, a, b, nudge)
        assert ok.all()
        assert np.array_equal(q, a / b)


@pytest.mark.parametrize("where,nudge", PLACES)
def test_roots(where, nudge):
    hard = ec.hard_roots()
    assert len(hard) > 80
    r = np.random.default_rng(8)
    n = 1 << 20
    for x in (hard, hard * 4.0 ** -33, hard * 4.0 ** 28, r.uniform(1, 4, n), r.uniform(1, 2, n) * 2.0 ** r.integers(-200, 60, n),
              1.0 + 2.0 ** -52 * np.arange(1000)):
        q, ok = ec.evaluate(where, True, x, x, nudge)
        assert ok.all()
        assert np.array_equal(q, np.sqrt(x))


@pytest.mark.parametrize("where,nudge", PLACES[-2:])
def test_out_of_range_is_reported(where, nudge):
    tiny = np.array([5e-324, 2.0 ** -1022, 2.0 ** -951, np.inf, -np.inf, np.nan, 2.0 ** 601])
    assert not ec.evaluate(where, False, tiny, np.ones(len(tiny)), nudge)[1].any()
    wild = np.array([0.0, -0.0, -1.0, 5e-324, 2.0 ** -201, 2.0 ** 61, np.inf, np.nan, -np.inf])
    assert not ec.evaluate(where, False, np.ones(len(wild)), wild, nudge)[1].any()
    wild = np.array([0.0, -0.0, -1.0, 5e-324, 2.0 ** -201, 2.0 ** 61, np.inf, np.nan])
    assert not ec.evaluate(where, True, wild, wild, nudge)[1].any()


def _same_bits(q, ref):
    return np.array_equal(q.view(np.uint64), ref.view(np.uint64))


@pytest.mark.parametrize("where,nudge", PLACES)
@pytest.mark.parametrize("root", [2, 3])
def test_signs_of_zero(where, nudge, root):
    """A quotient of zero, and one that rounds to zero, keeps its sign (in the
    form that the primitives are made with)."""
    r = np.random.default_rng(10)
    b = np.concatenate([r.uniform(1, 2, 500) * 2.0 ** r.integers(-60, 19, 500), 1.0 + np.arange(64) / 64.0])
    a = np.concatenate([np.zeros_like(b), -np.zeros_like(b)])
    b = np.tile(b, 2)
    q, ok = ec.evaluate(where, root, a, b, nudge)
    assert ok.all() and _same_bits(q, a / b)
    if root == 2:
        a, b = np.where(np.signbit(a), -5e-324, 5e-324), np.abs(b) + 2.5
        q, ok = ec.evaluate(where, root, a, np.minimum(b, 2.0 ** 59), nudge)
        assert ok.all() and _same_bits(q, a / np.minimum(b, 2.0 ** 59))


@pytest.mark.parametrize("where,nudge", PLACES)
def test_quotients_next_to_the_smallest_normal(where, nudge):
    """a / b half a spacing or less below 2^-1022 and a few spacings around it."""
    b = np.concatenate([1.0 + np.arange(1, 256) / 256.0, 1.0 + 2.0 ** -52 * np.arange(1, 64), 2.0 - 2.0 ** -52 * np.arange(1, 64)])
    b, k = (x.ravel() for x in np.meshgrid(b, np.arange(-8, 17), indexing="ij"))
    for sign in (1.0, -1.0):
        for s in (-1, 0, 3):
            a, d = sign * (b * 2.0 ** -1022 - k * 2.0 ** -1074), np.ldexp(b, s)
            a = np.ldexp(a, s) if s > 0 else a
            q, ok = ec.evaluate(where, 2, a, d, nudge)
            assert ok.all()
            assert np.array_equal(q, a / d)


@pytest.mark.parametrize("where,nudge", PLACES)
@pytest.mark.parametrize("root,power", [(4, 2), (5, 3)])
def test_quotients_by_powers(where, nudge, root, power):
    """Quotients by W^2 and W^3 whose reciprocals come from 1 / W, as in the
    Newton step: over random W, W next to powers of two and thirds, and
    numerators that put the quotient next to a tie."""
    r = np.random.default_rng(11)
    n = 1 << 18
    e = 2.0 ** -52 * np.arange(1, 4096)
    W = np.concatenate([r.uniform(1, 2, n) * 2.0 ** r.integers(-60, 19, n), 1.0 + e, 2.0 - e, 4.0 / 3.0 + e, 1.5 - e,
                        np.sqrt(2.0) + e, np.cbrt(2.0) - e])
    d = W * W if power == 2 else (W * W) * W
    a, b = ec.hard_quotients(200)
    near = (r.integers(1 << 52, 1 << 53, len(W)) + 0.5) * 2.0 ** -52 * d
    for num in (r.uniform(-1, 1, len(W)), near, d, np.nextafter(d, 0.0), -np.nextafter(d, np.inf), r.choice(a, len(W))):
        q, ok = ec.evaluate(where, root, num, W, nudge)
        assert ok.all()
        assert np.array_equal(q, num / d)
