"""Frames of the fixed-point products (csrc/sa_limb.cuh) on the host: the RKHS matrix's frame covers its diagonal 1 + eps
of either sign, and an entry above its frame has no digits."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("frame") / "libframe.so")
    subprocess.run(["g++", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover=undefined", "-shared", "-fPIC", "-o", out,
                    os.path.join(HERE, "frame_shim.cpp"), "-static-libubsan"], check=True)
    l = C.CDLL(out)
    l.unit_frame.argtypes = [C.c_double]
    l.digits_value.restype = C.c_double
    l.digits_value.argtypes = [C.c_double, C.c_int, C.c_int]
    return l


@pytest.mark.parametrize("eps", [0.0, 1e-10, 0.999, 1.0, 3.0, 1e9, -0.5, -1.0, -1.5, -2.999, -3.0, -5.0, -1e9])
def test_frame_covers_the_diagonal(lib, eps):
    e = lib.unit_frame(eps)
    for v in (1.0, 1.0 + eps):
        assert abs(v) < 2.0 ** (e - 1022)
        assert abs(lib.digits_value(v, e, 0) - v) <= 2.0 ** (e - 1078)           # half a unit of the digits
    assert 2.0 ** (e - 1023) <= max(1.0, abs(1.0 + eps))


@pytest.mark.parametrize("eps", [np.inf, -np.inf, np.nan])
def test_frame_of_a_diagonal_that_is_not_finite(lib, eps):
    assert lib.unit_frame(eps) == 2047


@pytest.mark.parametrize("vec", [0, 1])
@pytest.mark.parametrize("a", [2.0, -3.0, 1e300, np.inf, -np.inf, np.nan])
def test_no_digits_above_the_frame(lib, a, vec):
    assert lib.digits_value(a, 1023, vec) == 0.0
