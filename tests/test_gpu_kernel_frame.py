"""The RKHS matrix's frame on the GPU: entries that are not finite end the solve with SA_ERR_NONFINITE and DBL_MAX, as a
product in FP64 does, and entries beyond [-2, 2] are multiplied as any others.

Tolerance: the compared solves stop at the relative residual 1e-12; 1e-10 relative in positions and concentration, as in
the other comparisons of solver paths and with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def rel(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300))


@pytest.fixture(params=["persistent", "two-kernel", "matrix-free"])
def forward(request):
    """api.forward on each of the ways a K-PCG product runs."""
    from shape_atrophy_gb300 import api
    api.context(0)
    before = api.get_tuning()
    if request.param == "matrix-free":
        api.set_tuning(kernelMatrixFree=1)
    yield lambda spec: api.forward(dict(spec, cgKernel="two-kernel") if request.param == "two-kernel" else spec)
    api.set_tuning(**before)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("what", [dict(knlEps=np.nan), dict(knlEps=np.inf), dict(knlWidth=np.nan), dict(knlWidth=0.0),
                                  dict(knlWidth=1e-300, knlOrder=-1)])
def test_not_finite(forward, dim, what):
    from shape_atrophy_gb300 import _lib, problems
    spec = problems.demo_strip(21, 7, timeEnd=0.02) if dim == 2 else problems.frame_shell(level=0, lyrCntNum=3, timeEnd=0.02)
    got = forward(dict(spec, **what))
    assert got["info"]["status"] == _lib.SA_ERR_NONFINITE
    assert got["obj"][0] == np.finfo(np.float64).max


def test_diagonal_below_minus_two(forward):
    """A width so small that every k(i, j) underflows: K = (1 + eps) I and the velocity's system is ldm / (1 + eps) I + E,
    the same for (ldm, eps) = (1e4, -5) and (-1e4, 3)."""
    from shape_atrophy_gb300 import problems
    spec = dict(problems.demo_strip(21, 7, timeEnd=0.02), knlWidth=1e-4)
    a = forward(dict(spec, ldmWgt=1e4, knlEps=-5.0))
    b = forward(dict(spec, ldmWgt=-1e4, knlEps=3.0))
    assert a["info"]["status"] == 0 and b["info"]["status"] == 0
    move = b["lmkStk"][-1] - b["lmkStk"][0]
    assert np.abs(move).max() > 0.0
    assert rel(a["lmkStk"][-1] - a["lmkStk"][0], move) < TOL
    assert rel(a["tauMat"], b["tauMat"]) < TOL


@pytest.mark.parametrize("width,eps", [(-1.0, 1e4), (-0.1, 1e14)])
def test_width_that_is_not_positive(forward, width, eps):
    """k grows with the distance (order 0 in 3-D: exp(|d| / |w|)); eps keeps K positive definite for the oracle."""
    from shape_atrophy_gb300 import problems
    from oracle.oracle import Problem
    spec = dict(problems.frame_shell(level=1, lyrCntNum=3, timeEnd=0.02, knlOrder=0), knlWidth=width, knlEps=eps)
    want = Problem(spec).forward(spec["tauVarVec"], with_obj=True)
    got = forward(spec)
    assert want["status"] == 0 and got["info"]["status"] == 0
    assert rel(got["lmkStk"], want["lmkStk"]) < TOL
    assert rel(got["tauMat"], want["tauMat"]) < TOL
