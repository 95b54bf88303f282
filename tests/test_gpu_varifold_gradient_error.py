"""How far the FP64 varifold gradient is from sums in extended precision.

1. Nodes on a grid of 2^-20: centres and their differences are exact in FP64 wherever the shape lies, so the gradient of a
   curve moved by whole numbers keeps its bits.
2. A width whose square leaves the range of FP64 gives what a width far below every distance gives.
3. Against sums in numpy's long double (64 bits and more), relative in the 2-norm, root mean square over eight shapes: at
   most 1.5 times the error of the same pair terms in numpy's FP64.  Two FP64 evaluations that differ in the order of their
   sums differ by less than that over so many shapes; the bound leaves no room for a term that cancels (2 to 2.8 times)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _elements(x, vtx):
    X = x[:, vtx]
    if x.shape[0] == 2:
        e = X[:, 1] - X[:, 0]
        v = np.sqrt((e * e).sum(0))
        return (X[:, 0] + X[:, 1]) / 2, e / v, v
    a, b = X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]
    n = np.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])
    size = np.sqrt((n * n).sum(0))
    return (X[:, 0] + X[:, 1] + X[:, 2]) / 3, n / size, size / 2


def _gradient(x, vtx, target, vfd, T):
    """Node gradient of the objective in the number type T, pair by pair (2D_frame/varifold.cu:359-498)."""
    ck, cw, dk, dw = vfd
    x, target, cw, dw = x.astype(T), [np.asarray(t).astype(T) for t in target], T(cw), T(dw)
    c, u, v = own = _elements(x, vtx)
    D = x.shape[0]
    gc, gu, gv = np.zeros_like(c), np.zeros_like(c), np.zeros_like(v)
    for (cb, ub, vb), f in ((own, T(2)), (target, T(-2))):
        df = c[:, :, None] - cb[:, None, :]
        q = (df * df).sum(0) / (cw * cw)
        ang = (u[:, :, None] * ub[:, None, :]).sum(0)
        if ck == "G":
            k = np.exp(-q)
            c1 = -2 * k
        elif ck == "C":
            k = 1 / (1 + q)
            c1 = -2 * k * k
        else:
            r = np.sqrt(q)
            e = np.exp(-r)
            k, c1 = (1 + r) * e, -e
        if dk == "B":
            m, d1 = ang * ang, 2 * ang
        elif dk == "L":
            m, d1 = ang, np.ones_like(ang)
        elif dk == "O":
            m = np.exp(2 * (ang - 1) / (dw * dw))
            d1 = 2 * m / (dw * dw)
        else:
            m = np.exp(2 * (ang * ang - 1) / (dw * dw))
            d1 = 4 * ang * m / (dw * dw)
        gv += f * (k * m * vb).sum(1)
        gc += f * v * ((c1 * m * vb / (cw * cw))[None] * df).sum(2)
        # the part of u_j across u_i, per pair; times v_i / |e_i| or v_i / |n_i| below
        gu += f * ((k * d1 * vb)[None] * (ub[:, None, :] - ang[None] * u[:, :, None])).sum(2)
    g = np.zeros_like(x)
    if D == 2:
        ge = gu + gv * u
        parts = ((0, -ge + gc / 2), (1, ge + gc / 2))
    else:
        gn = (gu + gv * u) / 2
        X = x[:, vtx]
        a, b = X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]
        cross = lambda p, q: np.stack([p[1] * q[2] - p[2] * q[1], p[2] * q[0] - p[0] * q[2], p[0] * q[1] - p[1] * q[0]])
        ga, gb = cross(b, gn), cross(gn, a)
        parts = ((0, -ga - gb + gc / 3), (1, ga + gc / 3), (2, gb + gc / 3))
    for s, gs in parts:
        for d in range(D):
            np.add.at(g[d], vtx[s], gs[d])
    return g


def _shape(k, rng):
    from shape_atrophy_gb300 import api, mesh
    if k % 2 == 0:
        n = 60 + 9 * k
        obj = api.build_element_object_2d(n, 4, [1, 4], periodic=True)
        lmk = mesh.annulus_nodes(n, 4, 0.6, 1.0)
    else:
        surf, _, _, _, _, obj = mesh.shell_element_object(2, 3)
        lmk = mesh.shell_nodes(surf, 3, 0.7, 1.0)
    obj["vfdIfoMat"] = mesh.vfd_gradient_table(obj["vfdVtxMat"], lmk.shape[1])
    return obj, lmk + 0.003 * rng.normal(size=lmk.shape)


@pytest.mark.parametrize("cen", ["G", "C", "M"])
@pytest.mark.parametrize("direction", ["B", "L", "O", "U"])
def test_moving_a_curve_keeps_the_bits(cen, direction):
    from shape_atrophy_gb300 import api, mesh
    rng = np.random.default_rng(3)
    obj, lmk = _shape(0, rng)
    lmk = np.rint(lmk * 2.0 ** 20) / 2.0 ** 20
    moved = lmk + np.array([[4096.0], [-1024.0]])
    tgt = lmk + np.rint(0.02 * 2.0 ** 20 * np.sin(3 * lmk[::-1])) / 2.0 ** 20
    out = []
    for x, t in ((lmk, tgt), (moved, tgt + np.array([[4096.0], [-1024.0]]))):
        spec = dict(dim=2, elmObj=obj, lmkIniMat=x, tgt=mesh.varifold_target(t, obj["vfdVtxMat"]),
                    vfd=(cen, 0.13, direction, 0.7))
        out.append(api.varifold(spec, x, grad=True)[1])
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("cen", ["G", "C", "M"])
@pytest.mark.parametrize("direction,width", [("B", 1.0), ("L", 1.0), ("O", 0.8), ("O", 0.3), ("U", 0.8), ("U", 0.3)])
def test_error_against_extended_precision(cen, direction, width):
    from shape_atrophy_gb300 import api, mesh
    rng = np.random.default_rng(5)
    here, plain = [], []
    for k in range(8):
        obj, lmk = _shape(k, rng)
        vtx = np.asarray(obj["vfdVtxMat"]).astype(int)
        tgt = mesh.varifold_target(lmk + 0.02 * np.sin(3 * lmk[::-1]), obj["vfdVtxMat"])
        vfd = (cen, float(rng.uniform(0.05, 0.3)), direction, width)
        got = api.varifold(dict(dim=lmk.shape[0], elmObj=obj, lmkIniMat=lmk, tgt=tgt, vfd=vfd), lmk, grad=True)[1]
        want = _gradient(lmk, vtx, tgt, vfd, np.longdouble)
        err = lambda g: float(np.sqrt(((g - want) ** 2).sum() / (want ** 2).sum()))
        here.append(err(got))
        plain.append(err(_gradient(lmk, vtx, tgt, vfd, np.float64)))
    here, plain = (float(np.sqrt(np.mean(np.square(e)))) for e in (here, plain))
    print(f"{cen} x {direction} {width}: {here:.2e}, FP64 in numpy {plain:.2e}")
    assert here <= 1.5 * plain


@pytest.mark.parametrize("cen", ["G", "M"])
@pytest.mark.parametrize("k", [0, 1])
def test_width_below_every_distance(cen, k):
    """Only an element's pair with itself counts, whatever the width."""
    from shape_atrophy_gb300 import api, mesh
    obj, lmk = _shape(k, np.random.default_rng(3))
    spec = dict(dim=lmk.shape[0], elmObj=obj, lmkIniMat=lmk,
                tgt=mesh.varifold_target(lmk + 0.02 * np.sin(3 * lmk[::-1]), obj["vfdVtxMat"]))
    out = [api.varifold(dict(spec, vfd=(cen, w, "B", 1.0)), lmk, grad=True) for w in (1e-5, 1e-200)]
    assert np.abs(out[0][1]).max() > 0.0
    assert out[0][0] == out[1][0]
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("cen", ["G", "C", "M"])
def test_a_target_centre_that_is_not_a_number(cen):
    from shape_atrophy_gb300 import api, mesh
    obj, lmk = _shape(0, np.random.default_rng(3))
    tgt = [np.array(t, copy=True) for t in mesh.varifold_target(lmk + 0.01, obj["vfdVtxMat"])]
    tgt[0][0, 3] = np.nan
    spec = dict(dim=2, elmObj=obj, lmkIniMat=lmk, tgt=tuple(tgt), vfd=(cen, 0.1, "B", 1.0))
    value, grad = api.varifold(spec, lmk, grad=True)
    assert np.isnan(value) and np.isnan(grad).any() and np.isnan(api.varifold(spec, lmk))
