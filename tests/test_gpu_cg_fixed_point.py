"""The fixed-point persistent CG (csrc/sa_cgfix.cu) against the two-kernel FP64 CG at the edges of its ranges.

Both solve the same systems to the relative residual 1e-12, so a step's velocities differ by that times the operator's
condition; the bound, 1e-10 relative in positions and concentration, is the one the solver paths are held to against
the oracle.  Sizes: fewer rows than a warp, one row more than a slice, several warps per slice, one warp per slice,
slices that outgrow shared memory (tensor memory and streamed slots), several chunks per CTA (108 027 rows in 2-D, 122 886
in 3-D), and rows wide enough to be refused (FP64 kernels).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def rel(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300))


def _spec(kind, a, b):
    from shape_atrophy_gb300 import problems
    if kind == "annulus":
        return problems.annulus_layered(angNum=a, radNum=b, steps=3, cgTolVal=1e-12, layers=min(3, b - 1))
    return problems.shell_layered(level=a, lyrCntNum=b, steps=2, cgTolVal=1e-12, native=True)


@pytest.mark.parametrize("kind,a,b", [("annulus", 5, 4), ("annulus", 11, 3), ("annulus", 97, 13), ("annulus", 610, 8),
                                      ("annulus", 1201, 17), ("shell", 0, 2), ("shell", 1, 3), ("shell", 2, 4),
                                      ("shell", 3, 9), ("shell", 4, 5), ("shell", 4, 9), ("shell", 5, 6),
                                      ("annulus", 4001, 27), ("shell", 6, 3)])
def test_matches_two_kernel_cg(kind, a, b):
    from shape_atrophy_gb300 import api
    spec = _spec(kind, a, b)
    got = api.forward(spec, objective=False)
    want = api.forward(dict(spec, cgKernel="two-kernel"), objective=False)
    assert got["info"]["status"] == 0 and want["info"]["status"] == 0
    assert rel(got["lmkStk"], want["lmkStk"]) < TOL
    assert rel(got["tauMat"], want["tauMat"]) < TOL
    assert abs(got["info"]["cgIterTotal"] - want["info"]["cgIterTotal"]) <= 0.02 * want["info"]["cgIterTotal"] + 4
    again = api.forward(spec, objective=False)
    assert np.array_equal(again["lmkStk"], got["lmkStk"])          # the sums do not depend on the order of arrival


def test_many_columns_fall_back():
    """A node with more neighbours than a digit sum can take (a fan of 80 triangles around one node)."""
    from shape_atrophy_gb300 import api, mesh
    n = 80
    th = 2 * np.pi * np.arange(n) / n
    # ring layers 1 .. 3 around a hub: the hub is the bottom node 0
    obj, lmk = None, None
    tri, nodes = [], [np.zeros(2)]
    for r in (0.5, 1.0):
        nodes += [r * np.array([np.cos(t), np.sin(t)]) for t in th]
    for k in range(n):
        a, b = 1 + k, 1 + (k + 1) % n
        tri += [[0, a, b], [a, a + n, b + n], [a, b + n, b]]
    elm = np.array(tri).T.astype(np.int32)
    lmk = np.array(nodes).T.copy()
    N = lmk.shape[1]
    cnt = int(np.bincount(elm.reshape(-1), minlength=N).max())
    fvtx, ifo, _ = mesh._fem_pattern(elm.astype(np.int64), N, cnt)
    btm = np.array([[1 + k for k in range(n)], [1 + (k + 1) % n for k in range(n)]]).astype(np.int64) * 0
    btm = np.array([[0], [1]], dtype=np.int64)                     # bottom segment 0-1: nodes 0 and 1 come first
    E = elm.shape[1]
    obj = dict(elmVtxMat=elm, vtxElmMat=mesh._adjacency(elm.astype(np.int64), N), tanVtxMat=np.zeros((4, E), np.int32),
               tsvVtxMat=np.zeros((4, E), np.int32), btmVtxMat=btm.astype(np.int32),
               vtxBtmMat=mesh._adjacency(btm, 2), femVtxMat=fvtx, femIfoMat=ifo, elmLyrVec=np.zeros(E, np.int32))
    spec = dict(dim=2, elaType="isotropic", lmkIniMat=lmk, elmObj=obj, elmLyrVec=obj["elmLyrVec"],
                tauVarVec=np.array([0.6, 0.0, 1.0, 0.3]), tauPrmVec=np.array([0.0]), modVec=np.array([1.0, 0.5]),
                spdLyrVec=np.array([0.01]), ynkActPrmVec=np.array([0.5]), reaActPrmVec=np.array([2.0]), ldmWgt=0.0,
                knlOrder=1, knlWidth=0.1, knlEps=0.0, btmWgt=10.0, timeStp=0.01, timeNum=3, cgItrMax=20000,
                cgTolSqu=1e-24, rdItrMax=20000, rdTolSqu=1e-24)
    got = api.forward(spec, objective=False)
    want = api.forward(dict(spec, cgKernel="two-kernel"), objective=False)
    assert got["info"]["status"] == want["info"]["status"]
    if want["info"]["status"] == 0:
        assert rel(got["lmkStk"], want["lmkStk"]) < TOL
