"""The short reciprocals, quotients and square roots of the FP64 kernels (div64.cuh) have the
rounding of `/` and sqrt(): bit for bit against the device's operators, on random operands
over the callers' ranges and on the hardest ones there are, whose exact results lie next to
a rounding boundary.  Those are built from the operands' integers: a / b is beside the
midpoint (2 M + 1) / 2 of two neighbouring doubles where a 2^k = (2 M + 1) b + d for a small
odd d, sqrt(x) where (2 M + 1)^2 = 4 x + d, and 1 / b where b lies just below a power of two.
"""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    from veritas_gb300 import build as vb

    so = tmp_path_factory.mktemp("quotients") / "quotients_check.so"
    subprocess.run([vb._nvcc(), *vb.ARCH, "-O3", "--fmad=false", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", str(vb.CSRC), str(ROOT / "tests" / "native" / "quotients_check.cu"), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).quotients_check
    ptr = np.ctypeslib.ndpointer(np.float64)
    fn.argtypes = [ctypes.c_int, ptr, ptr, ptr, ptr, np.ctypeslib.ndpointer(np.uint8), ctypes.c_int]

    def run(op, a, b):
        a, b = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(b, dtype=np.float64)
        got, want, hard = np.empty_like(a), np.empty_like(a), np.empty(a.size, np.uint8)
        assert fn(op, a, b, got, want, hard, a.size) == 0
        return got, want, hard

    return run


def _same(got, want):
    bad = np.nonzero(got.view(np.uint64) != want.view(np.uint64))[0]
    assert bad.size == 0, (bad.size, bad[:5], got[bad[:5]], want[bad[:5]])


def _mantissas(rng, n):
    return rng.integers(1 << 52, 1 << 53, n).tolist()


def hard_quotients(rng, n):
    """Pairs (a, b) of 53-bit integers whose quotient is within 2^-50 of its last place of a midpoint."""
    out = []
    while len(out) < n:
        b = int(rng.integers(1 << 52, 1 << 53)) | 1
        if rng.random() < 0.3:  # the divisors whose own reciprocal is hard
            b = (1 << 53) - (2 * int(rng.integers(0, 5000)) + 1)
        for k in (53, 54):
            inv = pow(b, -1, 1 << k)
            for d in (1, -1, 3, -3, 5, -5, 7, -7):
                m = -d * inv % (1 << k)
                if k == 53:
                    m += 1 << 53
                if m < 1 << 53:
                    continue
                a, rest = divmod(m * b + d, 1 << k)
                assert rest == 0 and m % 2 == 1
                if a >= 1 << 53:
                    if a % 2:
                        continue
                if a:
                    out.append((float(a), float(b)))
    return np.array(out[:n]).T


def hard_roots():
    """x whose square root is within 2^-39 of its last place of a midpoint (d / 2^56 and less)."""
    out = []
    for d in range(-40007, 40008, 8):
        s = 1
        for k in range(3, 57):
            if (s * s - d) % (1 << (k + 1)):
                s += 1 << (k - 1)
        for m in {r % (1 << 54) for r in (s, -s, s + (1 << 53), -s + (1 << 53))}:
            x, rest = divmod(m * m - d, 4)
            if m >= 1 << 53 and rest == 0 and x == int(float(x)):
                out.append(float(x))
    return np.array(out)


@pytest.mark.gpu
def test_quotients_beside_midpoints(check):
    a, b = hard_quotients(np.random.default_rng(1), 200000)
    q = a / b
    for ea, eb in ((0, 0), (-300, -500), (600, 500), (-800, 1), (300, -300), (-60, -60)):
        got, want, hard = check(1, np.ldexp(a, ea), np.ldexp(b, eb))
        _same(got, want)
        np.testing.assert_array_equal(want, np.ldexp(q, ea - eb))
        assert hard.mean() > 0.99  # all of these, but where q itself is already the nearest


@pytest.mark.gpu
def test_reciprocals_beside_midpoints(check):
    b = np.array([float((1 << 53) - k) for k in range(1, 40001)] + [float((1 << 52) + k) for k in range(40000)])
    for e in (0, -52, -700, 500):
        got, want, _ = check(0, b, np.ldexp(b, e))
        _same(got, want)


@pytest.mark.gpu
def test_roots_beside_midpoints(check):
    x = hard_roots()
    assert x.size > 2000
    for e in (0, -104, 200, -600):
        got, want, _ = check(2, np.ldexp(x, e), x)
        _same(got, want)


@pytest.mark.gpu
def test_random_operands(check):
    rng = np.random.default_rng(2)
    n = 4_000_000
    lead = lambda: 1.0 + rng.random(n)  # noqa: E731
    a, b = np.ldexp(lead(), rng.integers(-600, 600, n)), np.ldexp(lead(), rng.integers(-200, 200, n))
    for op in (0, 1, 2):
        got, want, hard = check(op, a, b)
        _same(got, want)
        assert hard.mean() < 1e-4  # the short form is the one taken
    # what lies outside sqrt_rn's range goes to sqrt()
    x = np.array([0.0, -0.0, -1.0, np.inf, np.nan, 5e-324, 2.2e-308, 1.7e308, 1e-250, 1e250])
    got, want, _ = check(2, x, x)
    np.testing.assert_array_equal(got, want)
