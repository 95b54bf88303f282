"""Which CG kernel a layered FP64 call launches, by mesh size and row width, over a CUDA runtime without a GPU."""
import pytest

import fake_cuda

RUN = """
from shape_atrophy_gb300 import api, problems
import test_gpu_cg_ranges as t
def mark(n):
    with open(__import__("os").environ["FAKE_CUDART_LOG"], "a") as f:
        f.write("- " + n + chr(10))
def annulus(a, b):
    return problems.annulus_layered(angNum=a, radNum=b, steps=1, layers=3, native=True)
for name, spec in (("small", annulus(97, 13)), ("92416", annulus(5776, 16)), ("92432", annulus(5777, 16)), ("wide", t.wide_row())):
    mark(name)
    assert api.forward(spec, objective=False)["info"]["status"] == 0
mark("two-kernel")
api.forward(dict(annulus(97, 13), cgKernel="two-kernel", cgItrMax=5, rdItrMax=5), objective=False)
mark("global")
api.forward(dict(annulus(97, 13), cgKernel="persistent-global"), objective=False)
"""


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    r, lines = fake_cuda.run(RUN, tmp_path_factory.mktemp("cudart"))
    assert r.returncode == 0, r.stderr[-2000:]
    out, now = {}, None
    for device, kernel in lines:
        if device == "-":
            now = out.setdefault(kernel, [])
        else:
            now.append(kernel)
    return out


# mangled names: the velocity's kernels have the block size 2, the reaction-diffusion ones 1
FIX, MANY, FP64 = "k_cg_fixILi2E", "k_cg_fix_manyILi2E", "k_cg_persistILi2E"


@pytest.mark.parametrize("call,runs", [("small", FIX), ("92416", FIX), ("92432", MANY), ("wide", FP64),
                                       ("two-kernel", "k_cg_spmvILi2E"), ("global", "k_cg_persist_gILi2E")])
def test_choice(kernels, call, runs):
    assert any(runs in k for k in kernels[call])
    for other in (FIX, MANY, FP64):
        assert other == runs or not any(other in k for k in kernels[call])
