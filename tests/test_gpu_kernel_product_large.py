"""The product with the RKHS matrix at sizes where a CTA converts r in several chunks (more than 10240 nodes in 2-D, 6826 in
3-D) and takes its rows in several passes, against numpy in FP64.

With no elasticity and no penalty the velocity's system is ldm K^-1 v = b, so one step moves the nodes by dt K b / ldm: b is
the load of the bump, formed here from the mesh, and K is evaluated here in row tiles.

Tolerance.  Relative to the row's sum of |K_ij b_j|: an entry of K is off by a few roundings of its argument and its
polynomial on either side, b by a few of its sum over the elements; 64 x 2^-53 covers them, the products' roundings and the
reading of the velocity from positions.  Beside it the digits' bounds (sa_limb.cuh): an entry of K is rounded at 2^-56 of twice
the largest, 1 + eps, an entry of the vector at 2^-57 of twice its largest; the vector is r = b in the one product of the
iteration.
"""
import numpy as np
import pytest
from scipy import special

pytestmark = pytest.mark.gpu

LOAD, STEP = 2.0 ** 20, 2.0 ** 10      # the displacement shows the velocity without the rounding of the positions


def _spec(dim, order):
    from shape_atrophy_gb300 import problems
    if dim == 2:
        spec = problems.annulus_layered(angNum=662, radNum=16, steps=1, cgTolVal=1e-12, layers=3)
    else:
        spec = problems.shell_layered(level=3, lyrCntNum=11, steps=1, cgTolVal=1e-12, native=True)
    return dict(spec, modVec=np.zeros(6), btmWgt=0.0, spdLyrVec=np.full(3, 1e-12), ynkActPrmVec=np.array([LOAD]),
                timeStp=STEP, ldmWgt=1.0, knlOrder=order, knlWidth=0.3, knlEps=1e-3)


def _load(spec):
    """-sum over the elements of mean(yank) volume grad(phi_i), and the sum of the terms' sizes"""
    x, elm, D = spec["lmkIniMat"].T, np.asarray(spec["elmObj"]["elmVtxMat"]).T.astype(int), spec["dim"]
    p = np.asarray(spec["tauVarVec"], float)
    tau = p[D] * np.exp(-((x - p[:D]) ** 2).sum(1) / (2.0 * p[D + 1] ** 2))
    X = x[elm]
    q = X[:, 1:] - X[:, :1]
    g = np.linalg.inv(q).transpose(0, 2, 1)                    # rows: gradients of phi_1 .. phi_D
    g = np.concatenate([-g.sum(1, keepdims=True), g], 1)
    vol = np.abs(np.linalg.det(q)) / (2.0 if D == 2 else 6.0)
    f = -(LOAD * tau[elm].mean(1) * vol)[:, None, None] * g
    b = np.zeros_like(x)
    np.add.at(b, elm.reshape(-1), f.reshape(-1, D))
    return b


def _rows(spec, i0, i1):
    x, D, order = spec["lmkIniMat"].T, spec["dim"], spec["knlOrder"]
    d2 = sum((x[i0:i1, None, d] - x[None, :, d]) ** 2 for d in range(D))
    w = spec["knlWidth"]
    if order == -1:
        K = np.exp(-d2 / (w * w))
    elif D == 2:                                               # order 3
        r = np.sqrt(d2) / w
        s = np.where(r > 0.0, r, 1.0)
        f0, f1 = s * s * special.k0(s), s * special.k1(s)
        K = np.where(r > 0.0, ((24.0 + s * s) * f0 + 8.0 * (6.0 + s * s) * f1) / 48.0, 1.0)
    else:                                                      # order 2
        r = np.sqrt(d2) / w
        K = (3.0 + r * (3.0 + r)) / 3.0 * np.exp(-r)
    K[np.arange(i1 - i0), np.arange(i0, i1)] += spec["knlEps"]
    return K


@pytest.mark.parametrize("dim,order", [(2, -1), (2, 3), (3, -1), (3, 2)])
def test_one_step_without_elasticity(dim, order):
    from shape_atrophy_gb300 import api
    spec = _spec(dim, order)
    b = _load(spec)
    N = b.shape[0]
    assert N > (10240 if dim == 2 else 6826)
    want, bound = np.empty_like(b), np.empty_like(b)
    top, total = np.abs(b).max(0), np.abs(b).sum(0)
    for i in range(0, N, 512):
        K = _rows(spec, i, min(N, i + 512))
        want[i:i + 512] = K @ b
        bound[i:i + 512] = 64.0 * 2.0 ** -53 * (np.abs(K) @ np.abs(b)) + 2.0 ** -55 * (1.0 + spec["knlEps"]) * total \
            + 2.0 ** -56 * np.abs(K).sum(1)[:, None] * top.max()
    api.context(0)
    before = api.get_tuning()
    runs = []
    try:
        for kernel, free in (("auto", 0), ("two-kernel", 0), ("auto", 1)):
            api.set_tuning(kernelMatrixFree=free)
            runs.append(api.forward(dict(spec, cgKernel=kernel), objective=False))
    finally:
        api.set_tuning(**before)
    for r in runs:
        assert r["info"]["status"] == 0 and r["info"]["cgIterTotal"] == 1
        v = (r["lmkStk"][1] - r["lmkStk"][0]).T / STEP
        assert (np.abs(v - want) <= bound).all()
    np.testing.assert_array_equal(runs[0]["lmkStk"], runs[2]["lmkStk"])
