"""Fixed-point pair terms of the varifold objective (csrc/sa_pairfix.cuh) on the host, through a shim.

Bound, with the arguments as given doubles: root, exponential and product each lose at most 2^-56 of the value, the
direction product 2^-59 of its frame (each factor rounded to 2^-62, their low digits' product left out) and twice that
in its square, the last product 2^-60 of the frame before the kernel's own power of two is taken off: together below
2^-54 K_c K_d v + 2^-57 K_c + 2^-61, plus the shim's conversion to double, 2^-53 of the value.
"""
import ctypes as C
import os
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
getcontext().prec = 50


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pair") / "libpair.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-o", out, os.path.join(HERE, "pair_shim.cpp")], check=True)
    l = C.CDLL(out)
    l.pair_value.restype = C.c_double
    l.pair_value.argtypes = [C.c_int, C.c_int, C.c_double, C.c_void_p, C.c_void_p, C.c_double]
    l.pair_exp.restype = C.c_double
    l.pair_exp.argtypes = [C.c_double]
    l.pair_frame.argtypes = [C.c_double]
    return l


@pytest.mark.parametrize("ck", "MGC")
@pytest.mark.parametrize("dk", "BL")
def test_error_bound(lib, ck, dk):
    rng = np.random.default_rng(ord(ck) + ord(dk))
    lim = 63.0 if ck == "G" else 4000.0
    d2s = np.concatenate([[0.0, 5e-324, 1e-300, 1e-30, 0.25, np.nextafter(0.25, 0), 1.0, np.nextafter(1.0, 0), 4.0, lim,
                           np.nextafter(4096.0, 0), 4096.0, 1e5, 1e300], rng.uniform(0, 4, 300),
                          rng.uniform(0, lim, 300), 10.0 ** rng.uniform(-40, 3.5, 300)])
    worst = 0.0
    for d2 in d2s:
        u, w = rng.standard_normal(3), rng.standard_normal(3)
        u, w, v = u / np.linalg.norm(u), w / np.linalg.norm(w), rng.uniform(0, 1)
        if rng.uniform() < 0.2:
            w = u.copy()
        got = lib.pair_value(ord(ck), ord(dk), d2, u.ctypes.data, w.ctypes.data, v)
        q = Decimal(float(d2)) if ck != "C" else Decimal(1.0 + float(d2))
        r = q.sqrt()
        k = (1 + r) * (-r).exp() if ck == "M" else (-q).exp() if ck == "G" else 1 / q
        a = sum(Decimal(float(x)) * Decimal(float(y)) for x, y in zip(u, w))
        t = k * (a * a if dk == "B" else a) * Decimal(float(v))
        bound = float(abs(t)) * (2.0 ** -54 + 2.0 ** -53) + float(k) * 2.0 ** -57 + 2.0 ** -61
        err = abs(float(Decimal(got) - t))
        worst = max(worst, err / bound)
        assert err <= bound, (d2, got, float(t), err / bound)
    assert worst > 1e-3


def test_frames(lib):
    for n2, e in ((1.0, 0), (1.0 + 1e-15, 0), (1.0 - 1e-15, 0), (1.01, 1), (0.26, 0), (0.25, -1), (4.0, 1), (4.1, 2)):
        assert lib.pair_frame(n2) == e and n2 <= 4.0 ** e * (1 + 2.0 ** -38)


def test_exponential(lib):
    """e^-x as a double for 0 <= x < 64: x itself is cut to 57 bits, the table and the polynomial lose 2^-58, the
    conversion 2^-53: below 2^-52 together."""
    rng = np.random.default_rng(2)
    ln = np.log(2.0) / 256
    x = np.concatenate([rng.uniform(0, 64, 2000), np.arange(0, 23000, 37) * ln, [0.0, 1e-300, 1e-17, 63.999999]])
    for v in x:
        t = (-Decimal(float(v))).exp()
        assert abs(Decimal(lib.pair_exp(v)) / t - 1) < Decimal(2.0 ** -52), v
