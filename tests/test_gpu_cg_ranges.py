"""The fixed-point velocity CG at the ends of its ranges, against the two-kernel FP64 CG: 92 416 rows fill one chunk of 19
slices on each of 152 SMs, one more row takes several chunks per CTA; 95 000 rows lie between that and the sizes of the other
tests; and a node with 80 neighbours, whose rows the digit sums cannot take.

Tolerance as in the other comparisons of the solver paths: both stop at the relative residual 1e-12, 1e-10 relative in
positions and concentration."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def rel(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300))


def _compare(spec):
    from shape_atrophy_gb300 import api
    got = api.forward(spec, objective=False)
    want = api.forward(dict(spec, cgKernel="two-kernel"), objective=False)
    assert got["info"]["status"] == 0 and want["info"]["status"] == 0
    assert np.abs(want["lmkStk"][-1] - want["lmkStk"][0]).max() > 0.0
    assert rel(got["lmkStk"], want["lmkStk"]) < TOL
    assert rel(got["tauMat"], want["tauMat"]) < TOL
    assert abs(got["info"]["cgIterTotal"] - want["info"]["cgIterTotal"]) <= 0.02 * want["info"]["cgIterTotal"] + 4


@pytest.mark.parametrize("ang,rad", [(5776, 16), (5777, 16), (3801, 25)])
def test_one_chunk_to_several(ang, rad):
    from shape_atrophy_gb300 import problems
    _compare(problems.annulus_layered(angNum=ang, radNum=rad, steps=2, cgTolVal=1e-12, layers=3, native=True))


def wide_row():
    """A disc of 80 segments around its middle node, three rings; the middle and the first ring's first node are the bottom."""
    from shape_atrophy_gb300 import mesh
    n = 80
    th = 2.0 * np.pi * np.arange(n) / n
    nodes, tri = [np.zeros(2)], []
    for r in (0.5, 0.75, 1.0):
        nodes += [r * np.array([np.cos(t), np.sin(t)]) for t in th]
    for k in range(n):
        a, b = 1 + k, 1 + (k + 1) % n
        tri += [[0, a, b]]
        for ring in (0, n):
            tri += [[a + ring, a + ring + n, b + ring + n], [a + ring, b + ring + n, b + ring]]
    elm, lmk = np.array(tri).T.astype(np.int64), np.array(nodes).T.copy()
    N, E = lmk.shape[1], elm.shape[1]
    fvtx, ifo, _ = mesh._fem_pattern(elm, N, int(np.bincount(elm.reshape(-1), minlength=N).max()))
    btm = np.array([[0], [1]], dtype=np.int64)
    obj = dict(elmVtxMat=elm.astype(np.int32), vtxElmMat=mesh._adjacency(elm, N), tanVtxMat=np.zeros((4, E), np.int32),
               tsvVtxMat=np.zeros((4, E), np.int32), btmVtxMat=btm.astype(np.int32), vtxBtmMat=mesh._adjacency(btm, 2),
               femVtxMat=fvtx, femIfoMat=ifo, elmLyrVec=np.zeros(E, np.int32))
    assert int(np.bincount(np.asarray(fvtx)[0]).max()) == n + 1
    return dict(dim=2, elaType="isotropic", lmkIniMat=lmk, elmObj=obj, elmLyrVec=obj["elmLyrVec"],
                tauVarVec=np.array([0.6, 0.0, 1.0, 0.3]), tauPrmVec=np.array([0.0]), modVec=np.array([1.0, 0.5]),
                spdLyrVec=np.array([0.01]), ynkActPrmVec=np.array([0.5]), reaActPrmVec=np.array([2.0]), ldmWgt=0.0,
                knlOrder=1, knlWidth=0.1, knlEps=0.0, btmWgt=10.0, timeStp=0.01, timeNum=3, cgItrMax=20000,
                cgTolSqu=1e-24, rdItrMax=20000, rdTolSqu=1e-24)


def test_wide_row():
    _compare(wide_row())
