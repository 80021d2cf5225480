"""Operands at which a quotient or a square root is hardest to round, and the
library of tests/exact_ops.cu that evaluates them.

A quotient of significands A / B lies at distance |N| / (B 2^p) from a tie M
when 2^s A = B M + N with M odd: the tests take every |N| <= 9 for random
and extreme B.  A root lies next to a tie when M^2 - 2^54 X = N is small:
every such X with |N| < 256 (well past the method's error bound of 64) is
found by lifting the square roots of N modulo 2^54."""
import ctypes
import os
import random
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
SRC, LIB = os.path.join(HERE, "exact_ops.cu"), os.path.join(HERE, "_build", "libexact_ops.so")


def library():
    if not os.environ.get("HARM_PREBUILT_ONLY") and (not os.path.exists(LIB) or any(
            os.path.getmtime(f) > os.path.getmtime(LIB) for f in
            (SRC, *(os.path.join(HERE, "..", "harm_ramt_b200", "csrc", h) for h in ("harm_exact.cuh", "harm_device.cuh"))))):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        tmp = LIB + ".tmp%d" % os.getpid()
        subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                        "--fmad=false", "-Xcompiler", "-fPIC,-ffp-contract=off", "-shared", "-o", tmp, SRC], check=True)
        os.replace(tmp, LIB)
    return ctypes.CDLL(LIB)


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def evaluate(where, root, a, b, nudge=0):
    """(values, ok) of a / b, or of sqrt(a), on the host or the device."""
    a, b = np.ascontiguousarray(a, dtype=float), np.ascontiguousarray(b, dtype=float)
    q, ok = np.empty_like(a), np.empty(len(a), np.uint8)
    lib = library()
    if where == "host":
        lib.exact_host(int(root), len(a), _ptr(a), _ptr(b), nudge, _ptr(q), _ptr(ok))
    else:
        assert lib.exact_device(int(root), len(a), _ptr(a), _ptr(b), _ptr(q), _ptr(ok)) == 0
    return q, ok.astype(bool)


def hard_quotients(count, seed=1, most=9):
    rng = random.Random(seed)
    A, B = [], []
    for _ in range(count):
        b = rng.choice([rng.randrange(1 << 52, 1 << 53) | 1, (1 << 53) - 2 * rng.randrange(1, 2000) + 1,
                        (1 << 52) + 2 * rng.randrange(0, 2000) + 1])
        for N in range(-most, most + 1):
            for s in (53, 54):
                M = (-N * pow(b, -1, 1 << s)) % (1 << s)
                a = (b * M + N) >> s
                if M % 2 and (1 << 53) <= M < (1 << 54) and (1 << 52) <= a < (1 << 53):
                    A.append(a)
                    B.append(b)
    return np.array(A, float), np.array(B, float) * 2.0 ** -52


def hard_roots(most=256):
    out = []
    for N in range(-most + 1, most):
        if N % 8 != 1:
            continue
        roots = {m for m in range(8) if (m * m - N) % 8 == 0}
        for k in range(4, 55):
            roots = {c % (1 << k) for m in roots for c in (m, m + (1 << (k - 2)), m + (1 << (k - 1)), m + 3 * (1 << (k - 2)))
                     if (c * c - N) % (1 << k) == 0}
        for M in roots:
            X = (M * M - N) >> 54
            if (1 << 53) <= M < (1 << 54) and int(float(X)) == X:
                out.append(X * 2.0 ** -52)
    return np.array(sorted(out))


def operand_sets():
    """(name, a, b) of quotients in range."""
    r = np.random.default_rng(7)
    n = 1 << 20
    a, b = hard_quotients(3000)
    yield "next to a tie", a, b
    yield "next to a tie, scaled", -a * 2.0 ** -900, b * 2.0 ** -70
    yield "over the range", r.uniform(1, 2, n) * 2.0 ** r.integers(-950, 600, n), r.uniform(1, 2, n) * 2.0 ** r.integers(-200, 60, n)
    top = (2.0 ** 53 - np.arange(1, 200)) * 2.0 ** -53
    yield "top of a binade", np.tile(top, 199), np.repeat(top, 199)
    yield "powers of two", np.full(199, 2.0 ** -30), top
    yield "zero", np.zeros(199), top
