"""Fixed-point sums of products (csrc/sa_limb.cuh) on the host, through a shim.

Bound, with A the largest |a| and U the largest |u| of the sum, per product: |u| 2^-56 2A (an entry of a below a
quarter of A is rounded) and |a| 2^-57 2U, with the product of the two roundings; the result is rounded once
(2^-53).
"""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("limb") / "liblimb.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-o", out, os.path.join(HERE, "limb_shim.cpp")], check=True)
    l = C.CDLL(out)
    l.limb_dot.restype = C.c_double
    l.limb_dot.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int]
    return l


def dot(lib, a, u, eA=1, eU=1):
    a, u = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(u, dtype=np.float64)
    return lib.limb_dot(a.ctypes.data, u.ctypes.data, a.size, eA, eU)


def exact(a, u):
    return sum((Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, u)), Fraction(0))


@pytest.mark.parametrize("n", [1, 2, 45, 120])
@pytest.mark.parametrize("spread_a,spread_u", [(0, 0), (6, 4), (40, 0), (0, 70), (80, 80)])
def test_error_bound(lib, n, spread_a, spread_u):
    rng = np.random.default_rng(1000 * n + spread_a + spread_u)
    for scale in (0, -700, 500):
        for _ in range(20):
            a = rng.normal(size=n) * 2.0 ** (scale / 2 - rng.integers(0, spread_a + 1, n))
            u = rng.normal(size=n) * 2.0 ** (scale / 2 - rng.integers(0, spread_u + 1, n))
            A, U = Fraction(float(np.abs(a).max())), Fraction(float(np.abs(u).max()))
            want = exact(a, u)
            bound = sum(2 * A * abs(Fraction(float(y))) / 2**56 + 2 * U * abs(Fraction(float(x))) / 2**57
                        for x, y in zip(a, u)) + 4 * n * A * U / 2**113 + abs(want) / 2**53 + Fraction(5e-324)
            assert abs(Fraction(dot(lib, a, u)) - want) <= bound


def test_no_worse_than_fused_multiply_adds_on_operator_rows(lib):
    """Rows as the assembled operators have them (a dominant diagonal, off-diagonal entries of either sign): the largest
    error over the rows, relative to the sum of |a u|, is no larger than that of an FP64 multiply-add chain."""
    rng = np.random.default_rng(3)
    fixed, fma = 0.0, 0.0
    for _ in range(400):
        n = 3 * int(rng.integers(7, 16))
        a = rng.normal(size=n) * 0.2
        a[0] = 2.0
        u = rng.normal(size=n) * np.exp(rng.normal())
        want, size = exact(a, u), sum(abs(Fraction(float(x)) * Fraction(float(y))) for x, y in zip(a, u))
        acc = Fraction(0)
        for x, y in zip(a, u):
            acc = Fraction(float(acc + Fraction(float(x)) * Fraction(float(y))))      # one rounding per term
        eU = int(np.frexp(np.abs(u).max())[1]) + 1022 + 4        # the frame of a halo with 16 times larger entries
        fixed = max(fixed, float(abs(Fraction(dot(lib, a, u, 1, eU)) - want) / size))
        fma = max(fma, float(abs(acc - want) / size))
    assert fixed <= fma


def test_frames_edges_and_non_finite(lib):
    one = [1.0]
    assert dot(lib, one, one) == 1.0 and dot(lib, [-3.25], [0.75]) == -2.4375
    assert dot(lib, [0.0, 0.0], [1.0, 2.0]) == 0.0
    assert dot(lib, [1e300], [1e8]) == 1e308
    assert dot(lib, [1e300], [1e300]) == np.inf and dot(lib, [1e-300], [1e-300]) == 0.0
    assert dot(lib, [2.0 ** -500], [2.0 ** -570]) == 2.0 ** -1070       # subnormal result
    assert np.isnan(dot(lib, [np.nan, 1.0], [1.0, 1.0])) and np.isnan(dot(lib, [1.0, 1.0], [np.inf, 1.0]))
    n = lib.limb_max_terms()
    big = np.full(n, np.nextafter(2.0, 0.0))
    assert abs(dot(lib, big, -big) + 4.0 * n) < 1e-12 * n           # the largest sums do not overflow
