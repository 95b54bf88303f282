"""The fixed-point velocity CG where neighbouring materials differ by orders of magnitude, against FP64 kernels.

One step from rest with materials 1 : c : 1.  Rounding is multiplied by about c there, so the yardstick is measured: the
two-kernel CG and the persistent kernel with vectors in global memory are both FP64 and differ by one sample d of it,
relative in the 2-norm.  The fixed-point solve is held to 4 d from the first, and to its iteration count within a fifth
(the FP64 kernels' counts differ by up to a tenth).  Sizes: the resident, the streamed and the several-chunk form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spec(kind, a, b, contrast):
    from shape_atrophy_gb300 import problems
    if kind == "annulus":
        spec = problems.annulus_layered(angNum=a, radNum=b, steps=1, cgTolVal=1e-13, layers=3)
    else:
        spec = problems.shell_layered(level=a, lyrCntNum=b, steps=1, cgTolVal=1e-13, native=True)
    lam = np.array([1.0, contrast, 1.0])
    # a large load and step: the displacement shows the velocity without the rounding of the positions
    return dict(spec, modVec=np.column_stack([lam, lam / 2]).reshape(-1), spdLyrVec=np.full(3, 1e-12),
                ynkActPrmVec=np.array([0.5 * 2.0 ** 20]), timeStp=2.0 ** 10, cgItrMax=60000)


@pytest.mark.parametrize("contrast", [1e6, 1e8])
@pytest.mark.parametrize("kind,a,b", [("annulus", 128, 13), ("shell", 3, 7), ("shell", 4, 9), ("shell", 6, 3)])
def test_contrast(kind, a, b, contrast):
    from shape_atrophy_gb300 import api
    spec = _spec(kind, a, b, contrast)
    runs = [api.forward(dict(spec, cgKernel=k), objective=False) for k in ("auto", "two-kernel", "persistent-global")]
    assert all(r["info"]["status"] == 0 for r in runs)
    v = [r["lmkStk"][1] - r["lmkStk"][0] for r in runs]
    its = [r["info"]["cgIterTotal"] for r in runs]
    err, d = (np.sqrt(((x - v[1]) ** 2).sum() / (v[1] ** 2).sum()) for x in (v[0], v[2]))
    print(f"{kind} {a} {b} contrast {contrast:g}: fixed point {err:.2e}, FP64 {d:.2e}, iterations {its}")
    assert err <= 4.0 * d
    assert abs(its[0] - its[1]) <= 0.2 * its[1]
