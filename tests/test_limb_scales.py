"""Column scales and longer digits of the fixed-point sums of products (csrc/sa_limb.cuh) on the host.

Bound: that of test_limb.py in the scaled entries a 2^s and u 2^-s, whose largest are A and U: per product |u| 2^-56 2A and
|a| 2^-57 2U, with the product of the two roundings; the result is rounded once (2^-53).  A row whose digits are g bits
longer rounds its entries 2^g times finer."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("scale") / "libscale.so")
    subprocess.run(["g++", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover=undefined", "-shared", "-fPIC", "-o", out,
                    os.path.join(HERE, "scale_shim.cpp"), "-static-libubsan"], check=True)
    l = C.CDLL(out)
    l.limb_scaled_dot.restype = C.c_double
    l.limb_scaled_dot.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_void_p]
    l.limb_above.restype = C.c_float
    l.limb_above.argtypes = [C.c_double, C.c_int]
    return l


def dot(lib, a, u, s, own=0, longer=0):
    a, u, s = (np.ascontiguousarray(x, dtype=t) for x, t in ((a, np.float64), (u, np.float64), (s, np.int32)))
    g = C.c_int()
    v = lib.limb_scaled_dot(a.ctypes.data, u.ctypes.data, s.ctypes.data, a.size, own, longer, C.byref(g))
    return (v, g.value) if longer else v


def check(got, g, av, uv, want):
    n = av.size
    A, U = Fraction(float(np.abs(av).max())), Fraction(float(np.abs(uv).max()))
    bound = sum(2 * A * abs(Fraction(float(y))) / 2**(56 + g) + 2 * U * abs(Fraction(float(x))) / 2**57
                for x, y in zip(av, uv)) + 4 * n * A * U / 2**113 + abs(want) / 2**53
    assert abs(Fraction(got) - want) <= bound


def exact(a, u):
    return sum((Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, u)), Fraction(0))


@pytest.mark.parametrize("n", [1, 2, 45, 80])
@pytest.mark.parametrize("spread", [0, 4, 30, 400])
def test_error_bound(lib, n, spread):
    """u of a column is 2^s of the others', its entry 2^-s, as in the rows where a stiff layer meets a soft one."""
    rng = np.random.default_rng(100 * n + spread)
    for _ in range(20):
        s = rng.integers(-spread, spread + 1, n)
        av, uv = rng.normal(size=n), rng.normal(size=n)
        a, u = np.ldexp(av, -s), np.ldexp(uv, s)
        check(dot(lib, a, u, s), 0, av, uv, exact(a, u))


def test_edges_and_non_finite(lib):
    for longer in (0, 1):
        d = lambda *x: dot(lib, *x, longer=1)[0] if longer else dot(lib, *x)
        for s in (-1022, -3, 0, 5, 1023):
            assert d([0.0], [1.0], [s]) == 0.0 and d([3.0], [0.0], [s]) == 0.0
            assert d([0.0, 0.0], [0.0, 0.0], [s, 0]) == 0.0
            assert d([-3.25], [0.75], [s]) == -2.4375
            assert d([0.0, 1.5], [0.0, 2.0 ** -40], [s, 0]) == 1.5 * 2.0 ** -40      # a zero does not set the frame
            for bad in (np.nan, np.inf, -np.inf):
                assert np.isnan(d([bad, 1.0], [1.0, 1.0], [s, 0]))
                assert np.isnan(d([1.0, 1.0], [1.0, bad], [0, s]))
        assert d([2.0 ** 900], [2.0 ** 900], [-100]) == np.inf
        assert d([2.0 ** 1000], [2.0 ** -1000], [-1000]) == 1.0
        assert d([2.0 ** -500], [2.0 ** -570], [400]) == 2.0 ** -1070
        assert d([1.0], [5e-324], [-1022]) == 5e-324


@pytest.mark.parametrize("n,least", [(21, 3), (45, 3), (80, 3)])
@pytest.mark.parametrize("own", [0, 9, -70])
def test_operator_rows_take_longer_digits(lib, n, least, own):
    """A dominant diagonal: the row's digits are `least` bits longer at least, and the matrix part of the bound that much
    smaller."""
    rng = np.random.default_rng(n)
    for _ in range(20):
        s = rng.integers(-20, 21, n)
        av, uv = rng.uniform(-0.1, 0.1, size=n), rng.normal(size=n)
        av[n // 2] = rng.uniform(1.0, 2.0)
        a, u = np.ldexp(av, -s - own), np.ldexp(uv, s)
        got, g = dot(lib, a, u, s, own, 1)
        assert g >= least
        check(got, g, np.ldexp(av, -own), uv, exact(a, u))


@pytest.mark.parametrize("big", [1.0, np.nextafter(2.0, 0.0), 1.86, 1.5])
@pytest.mark.parametrize("own", [0, 300])
def test_largest_sums_stay_in_range(lib, big, own):
    """Rows of n equal entries of one sign with the largest u: the digits are as long as the sums allow, and no longer."""
    for n in range(1, 81):
        a, u = np.full(n, big), np.full(n, np.nextafter(2.0, 0.0))
        for sign in (1.0, -1.0):
            got, g = dot(lib, sign * a, u, np.zeros(n, int), own, 1)
            assert abs(got - sign * n * big * u[0]) <= 1e-15 * n * big * 2
            assert own == 0 or g == 0                          # a sum out of FP32's range: no extra bits


def test_fp32_bounds(lib):
    for v in (1.0, -1.5, np.nextafter(2.0, 0.0), 3.1e-300, 7e300, 5e-324, 0.0):
        for s in (-1000, -40, 0, 40, 1000):
            want, got = abs(Fraction(v)) * (Fraction(2) ** s), lib.limb_above(v, s)
            assert got == np.inf or Fraction(float(got)) >= want
            if abs(v) >= 2.0 ** -1022 and Fraction(2) ** -120 < want < Fraction(2) ** 120:
                assert Fraction(float(got)) <= want * (1 + Fraction(2) ** -22)
