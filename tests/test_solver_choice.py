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

MEMORY = """
import ctypes, os
from shape_atrophy_gb300 import api, problems
rt = ctypes.CDLL("libcudart.so.13")
rt.fake_cudart_most.restype = ctypes.c_size_t
def mark(n):
    with open(os.environ["FAKE_CUDART_LOG"], "a") as f:
        f.write("- " + n + chr(10))
spec = problems.shell_layered(level=3, lyrCntNum=5, steps=1, native=True)
other = dict(spec, cgKernel="persistent-global")
api.forward(other)
rt.fake_cudart_most()
api.forward(other)
need = rt.fake_cudart_most()                 # without a plan
for extra in range(0, 3 << 20, 1 << 14):
    ctypes.CDLL(None).setenv(b"FAKE_CUDART_MEMORY", str(need + extra).encode(), 1)
    mark("memory" if extra == 0 else "more")
    assert api.forward(spec)["info"]["status"] == 0, extra
ctypes.CDLL(None).unsetenv(b"FAKE_CUDART_MEMORY")
mark("plenty")
assert api.forward(spec)["info"]["status"] == 0
"""


def _by_mark(lines):
    out, now = {}, None
    for device, kernel in lines:
        if device == "-":
            now = out.setdefault(kernel, [])
        elif now is not None:
            now.append(kernel)
    return out


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    r, lines = fake_cuda.run(RUN, tmp_path_factory.mktemp("cudart"))
    assert r.returncode == 0, r.stderr[-2000:]
    return _by_mark(lines)


# mangled names: the velocity's kernels have the block size 2, the reaction-diffusion ones 1
FIX, MANY, FP64 = "k_cg_fixILi2E", "k_cg_fix_manyILi2E", "k_cg_persistILi2E"


@pytest.mark.parametrize("call,runs", [("small", FIX), ("92416", FIX), ("92432", MANY), ("wide", FP64),
                                       ("two-kernel", "k_cg_spmvILi2E"), ("global", "k_cg_persist_gILi2E")])
def test_choice(kernels, call, runs):
    assert any(runs in k for k in kernels[call])
    for other in (FIX, MANY, FP64):
        assert other == runs or not any(other in k for k in kernels[call])


def test_memory_for_the_call_but_not_for_a_plan(tmp_path):
    """With the memory that a call without a plan needs, and from there up to the plan's own: every call runs, the first in FP64
    kernels."""
    r, lines = fake_cuda.run(MEMORY, tmp_path)
    assert r.returncode == 0, r.stderr[-2000:]
    calls = _by_mark(lines)
    assert any("k_cg_persistILi3E" in k for k in calls["memory"]) and not any("k_cg_fix" in k for k in calls["memory"])
    assert any("k_cg_fixILi3E" in k for k in calls["more"])
    assert any("k_cg_fixILi3E" in k for k in calls["plenty"])
