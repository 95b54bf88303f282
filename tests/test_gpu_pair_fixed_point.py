"""Fixed-point pair sums of the varifold objective (csrc/sa_varifold.cu k_vfd_rows_fix) against a plain FP64 evaluation.

Bound, relative to the sum of the absolute values of the terms: the plain evaluation rounds each term a few times
(distance, exponential, products: below 16 x 2^-53 with the exponent's own rounding at r <= 8, where the terms matter), the
kernel less; the sums add 2^-53 per 128 columns here and nothing there (fsum).  1e-14 covers both.  Sizes: fewer
elements than a warp, both sides of the 128-element tile, more and fewer columns than rows.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spec(dim, size):
    from shape_atrophy_gb300 import problems
    if dim == 2:
        return problems.annulus_layered(angNum=size, radNum=4, steps=1, cgTolVal=1e-8, layers=3)
    return problems.shell_layered(level=size, lyrCntNum=2, steps=1, cgTolVal=1e-8)


def _plain(S, T, vfd):
    ck, cw, dk, dw = vfd
    d2 = ((S[0][:, :, None] - T[0][:, None, :]) ** 2).sum(0) / cw ** 2
    r = np.sqrt(d2)
    kc = (1 + r) * np.exp(-r) if ck == "M" else np.exp(-d2) if ck == "G" else 1.0 / (1.0 + d2)
    ang = np.einsum("di,dj->ij", S[1], T[1])
    kd = {"B": lambda a: a * a, "L": lambda a: a, "O": lambda a: np.exp(2.0 * (a - 1.0) / dw ** 2),
          "U": lambda a: np.exp(2.0 * (a * a - 1.0) / dw ** 2)}[dk](ang)
    return (kc * kd * S[2][:, None] * T[2][None, :]).reshape(-1)


def _check(spec, lmk, tgt, vfd):
    from shape_atrophy_gb300 import api, mesh
    S = mesh.varifold_target(lmk, spec["elmObj"]["vfdVtxMat"])
    terms = np.concatenate([_plain(S, S, vfd), -2.0 * _plain(S, tgt, vfd), _plain(tgt, tgt, vfd)])
    got = api.varifold(dict(spec, tgt=tgt, vfd=vfd), lmk)
    assert abs(got - math.fsum(terms)) <= 1e-14 * np.abs(terms).sum()


@pytest.mark.parametrize("dim,size", [(2, 5), (2, 127), (2, 128), (2, 129), (2, 700), (3, 0), (3, 2), (3, 3)])
@pytest.mark.parametrize("ck,dk,w", [("M", "B", 0.3), ("M", "L", 0.02), ("G", "B", 0.5), ("G", "L", 5.0), ("M", "B", 1e-3),
                                     ("C", "O", 0.15), ("C", "U", 0.02), ("M", "O", 0.3), ("G", "U", 0.2), ("C", "B", 2.0)])
def test_matches_plain_evaluation(dim, size, ck, dk, w):
    from shape_atrophy_gb300 import mesh
    spec = _spec(dim, size)
    lmk, vtx = spec["lmkIniMat"], spec["elmObj"]["vfdVtxMat"]
    tgt = mesh.varifold_target(lmk + mesh.smooth_displacement(lmk, 0.05, 3), vtx)
    n = tgt[2].size
    for cut in (n, max(1, n // 3), 1):                       # as many target elements as rows, and fewer
        _check(spec, lmk, tuple(np.ascontiguousarray(a[..., :cut]) for a in tgt), (ck, w, dk, 0.8))
    more = tuple(np.ascontiguousarray(np.concatenate([a, a[..., : n // 2 + 1]], axis=-1)) for a in tgt)
    _check(spec, lmk, more, (ck, w, dk, 0.8))


@pytest.mark.parametrize("dk", "BLOU")
def test_targets_of_other_lengths(dk):
    """Target directions that are no unit vectors, volumes over many decades, zero and negative ones."""
    from shape_atrophy_gb300 import mesh
    rng = np.random.default_rng(4)
    spec = _spec(3, 2)
    lmk = spec["lmkIniMat"]
    cen, uni, vol = mesh.varifold_target(lmk, spec["elmObj"]["vfdVtxMat"])
    for su, sv in ((3.7, 1.0), (1e-9, 1e6), (1e12 if dk in "BL" else 1.5, 1e-20)):
        v = vol * sv * 10.0 ** rng.uniform(-12, 0, vol.size)
        v[::7], v[3::11] = 0.0, -v[3::11]
        u = uni * su * rng.uniform(0.1, 1.0, vol.size)
        u[:, 5] = 0.0
        _check(spec, lmk, (cen + 0.01, u, v), ("M", 0.4, dk, 1.6))


@pytest.mark.parametrize("k", range(3))
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_that_are_not_finite(k, bad):
    from shape_atrophy_gb300 import api, mesh
    spec = _spec(3, 1)
    tgt = [a.copy() for a in mesh.varifold_target(spec["lmkIniMat"], spec["elmObj"]["vfdVtxMat"])]
    tgt[k].reshape(-1)[7] = bad
    assert np.isnan(api.varifold(dict(spec, tgt=tuple(tgt), vfd=("M", 0.4, "B", 1.0)), spec["lmkIniMat"]))


@pytest.mark.parametrize("ck", "MGC")
@pytest.mark.parametrize("dk", "BLOU")
@pytest.mark.parametrize("w,size", [(0.3, 129), (5e-3, 40)])
def test_gradient_matches_complex_step(ck, dk, w, size):
    """Gradient rows, whose kernel values are formed in fixed point (in FP64 beyond 64 widths), along a random direction
    against the complex step of a plain evaluation, exact to rounding; 1e-12 of the sum of the absolute products."""
    from shape_atrophy_gb300 import api, mesh
    rng = np.random.default_rng(size)
    spec = _spec(2, size)
    lmk, vtx = spec["lmkIniMat"], spec["elmObj"]["vfdVtxMat"]
    tgt = mesh.varifold_target(lmk + mesh.smooth_displacement(lmk, 0.03, 5), vtx)
    vfd = (ck, w, dk, 0.8)
    p = rng.standard_normal(lmk.shape)
    x = lmk + 1e-30j * p
    q0, q1 = x[:, vtx[0]], x[:, vtx[1]]
    d = q1 - q0
    v = np.sqrt((d * d).sum(0))
    S = (0.5 * (q0 + q1), d / v, v)
    d2 = ((S[0][:, :, None] - S[0][:, None, :]) ** 2).sum(0)
    if ck == "M":                                            # no complex root of the diagonal's zero
        S = tuple(S)
        i = np.arange(v.size)
        r2 = d2 / w ** 2
        r2[i, i] = 1.0
        r = np.sqrt(r2)
        k = (1 + r) * np.exp(-r)
        k[i, i] = 1.0
        a = np.einsum("di,dj->ij", S[1], S[1])
        kd = {"B": a * a, "L": a, "O": np.exp(2 * (a - 1) / 0.64), "U": np.exp(2 * (a * a - 1) / 0.64)}[dk]
        own = (k * kd * v[:, None] * v[None, :]).sum()
    else:
        own = _plain(S, S, vfd).sum()
    want = float((own - 2.0 * _plain(S, tgt, vfd).sum()).imag * 1e30)
    _, g = api.varifold(dict(spec, tgt=tgt, vfd=vfd), lmk, grad=True)
    assert abs((g * p).sum() - want) <= 1e-12 * np.abs(g * p).sum()
