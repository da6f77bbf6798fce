"""Correctly rounded FP64 division and square root (csrc/evp_fp64.cuh).

The device's results must have the bits of IEEE division and square root
(numpy's, on the host) wherever the range tests accept the operands: random
significands over the range, the square roots closest to the middle of two
doubles, quotients within a few units of a midpoint, all-ones divisors, and
operands at the edges of the range.  The hard cases' own construction is
checked on the CPU in exact integers.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT


def hard_square_roots(most=24):
    """x whose square root lies near n + 1/2: n*n + n - c = X, X in
    [2^104, 2^106) with 53 significant bits, |c| <= most.  Returned as
    (significand integer of 53 bits, X) pairs."""
    out = []
    for c in range(-most, most + 1, 2):
        sols = [0, 1]  # n*n + n - c = 0 (mod 2), lifted bit by bit to mod 2^52
        for k in range(1, 52):
            sols = [s + (b << k) for s in sols for b in (0, 1)
                    if ((s + (b << k)) ** 2 + s + (b << k) - c) % (1 << (k + 1)) == 0]
        for s in sols:
            n = s + (1 << 52)
            X = n * n + n - c
            if not (1 << 104) <= X < (1 << 106):
                continue
            unit = 52 if X < (1 << 105) else 53
            if X % (1 << unit) == 0:
                out.append((X >> unit, X))
    return out


def hard_quotients(count, rng):
    """(a, b) significand integers with a/b within |N| <= 15 of a midpoint of
    two 53-bit quotients: a * 2^54 = m*b + N, m odd of 54 bits."""
    out = []
    while len(out) < count:
        b = int(rng.integers(1 << 52, 1 << 53)) | 1
        N = int(rng.choice([-15, -7, -5, -3, -1, 1, 3, 5, 7, 15]))
        m = (-N * pow(b, -1, 1 << 54)) % (1 << 54)
        a = (m * b + N) >> 54
        if m >= 1 << 53 and 1 << 52 <= a < 1 << 53:
            out.append((a, b, m, N))
    return out


def test_hard_cases_are_hard():
    roots = hard_square_roots()
    assert len(roots) >= 20
    for sig, X in roots:
        assert sig.bit_length() == 53
        n = int(np.floor(np.sqrt(float(X))))
        assert min(abs(4 * X - (2 * k + 1) ** 2) for k in range(n - 2, n + 3)) <= 4 * 24 + 1
    for a, b, m, N in hard_quotients(50, np.random.default_rng(1)):
        assert (a << 54) - m * b == N and m % 2 == 1


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fp64") / "fp64_shim.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3",
                    "-std=c++17", "-fmad=false", "-shared", "-Xcompiler", "-fPIC", "-I",
                    os.path.join(PKG, "csrc"), os.path.join(ROOT, "tests", "native", "fp64_shim.cu"),
                    "-o", out], check=True)
    return C.CDLL(out)


def run(L, op, a, b=None):
    a = np.ascontiguousarray(a, dtype=np.float64)
    b = a if b is None else np.ascontiguousarray(b, dtype=np.float64)
    out, ok = np.empty_like(a), np.empty(a.size, dtype=np.int32)
    p = lambda x: x.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert L.fp64_run(op, a.size, p(a), p(b), p(out), p(ok)) == 0
    return out, ok.astype(bool)


def same(x, y):
    return x.view(np.int64) == y.view(np.int64)


def values(rng, n, lo=-500, hi=499, ones=0.05, powers=0.05):
    s = rng.integers(1 << 52, 1 << 53, n)
    pick = rng.random(n)
    s = np.where(pick < ones, (1 << 53) - 1 - rng.integers(0, 3, n), s)
    s = np.where(pick > 1 - powers, (1 << 52) + rng.integers(0, 3, n), s)
    return np.ldexp(s.astype(np.float64), rng.integers(lo, hi + 1, n) - 52)


@pytest.mark.gpu
def test_square_root_bits(shim):
    rng = np.random.default_rng(2)
    sig = np.array([s for s, _ in hard_square_roots()], dtype=np.float64)
    # a significand's parity of exponent decides which of its two roots is met
    hard = np.concatenate([np.ldexp(sig, e) for e in (-552, -301, -53, -52, 0, 1, 200, 446)])
    x = np.concatenate([hard, values(rng, 2_000_000), np.ldexp(1.0, np.arange(-500, 500)), [0.0]])
    got, ok = run(shim, 1, x)
    assert ok.all()
    assert same(got, np.sqrt(x)).all()
    for x in (-0.0, -1.0, np.inf, np.nan, 5e-324, np.ldexp(1.0, 500), np.ldexp(1.9, -501)):
        assert not run(shim, 1, [x])[1].any()


@pytest.mark.gpu
def test_quotient_bits(shim):
    rng = np.random.default_rng(3)
    h = hard_quotients(20000, rng)
    a = np.array([x[0] for x in h], dtype=np.float64)
    b = np.array([x[1] for x in h], dtype=np.float64)
    a = np.concatenate([np.ldexp(a, rng.integers(-500, 446, a.size)), values(rng, 2_000_000),
                        np.zeros(1000)])
    b = np.concatenate([np.ldexp(b, rng.integers(-500, 446, b.size)), values(rng, 2_000_000),
                        values(rng, 1000)])
    a[20000:1_000_000] *= rng.choice([-1.0, 1.0], 980_000)
    got, ok = run(shim, 0, a, b)
    assert ok.mean() > 0.95
    assert same(got, a / b)[ok].all()
    # a power of two over an all-ones divisor, and operands out of range, are refused
    ones = np.ldexp(float((1 << 53) - 1), -52)
    for x, y in ((1.0, ones), (-0.0, ones), (3.0, 0.0), (3.0, np.inf), (np.nan, 2.0),
                 (3.0, -2.0), (np.ldexp(1.5, 500), 3.0), (np.ldexp(1.5, -501), 3.0)):
        assert not run(shim, 0, [x], [y])[1].any(), (x, y)
