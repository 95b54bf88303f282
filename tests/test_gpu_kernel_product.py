"""The fixed-point products with the RKHS matrix at the edges of their tiles (rows in blocks of 8, columns in tiles of 4,
a sixteenth of the tiles per warp), against the CPU oracle: FP64 throughout, CG tolerance 1e-12, bound 1e-10 as in the
other comparisons with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def rel(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300))


@pytest.mark.parametrize("ang,lyr", [(3, 2), (5, 3), (9, 7), (13, 5), (33, 4), (37, 17)])
def test_strips_of_every_remainder(ang, lyr):
    from shape_atrophy_gb300 import api, problems
    from oracle.oracle import Problem
    spec = problems.demo_strip(ang, lyr, timeEnd=0.02)
    want = Problem(spec).forward(spec["tauVarVec"], with_obj=True)
    got = api.forward(spec)
    assert got["info"]["status"] == want["status"]
    assert rel(got["lmkStk"], want["lmkStk"]) < TOL
    assert rel(got["tauMat"], want["tauMat"]) < TOL
    assert abs(got["obj"][0] - want["obj"]) <= TOL * abs(want["obj"])
    loop = api.forward(dict(spec, cgKernel="two-kernel"))
    assert rel(loop["lmkStk"], want["lmkStk"]) < TOL


def test_columns_in_several_chunks():
    """More nodes than one CTA's digits of r hold (10240 in 2D): the chunked product against the launch loop."""
    from shape_atrophy_gb300 import api, problems
    spec = problems.demo_strip(331, 32, timeEnd=0.01, cgTolVal=1e-9)      # 10592 nodes
    got = api.forward(spec, objective=False)
    loop = api.forward(dict(spec, cgKernel="two-kernel"), objective=False)
    assert got["info"]["status"] == 0 and loop["info"]["status"] == 0
    # both stop at the relative residual 1e-9
    assert rel(got["lmkStk"] - got["lmkStk"][0], loop["lmkStk"] - loop["lmkStk"][0]) < 1e-6
