"""One process, two devices: the host code runs over a CUDA runtime without a GPU (fake_cudart.cpp), the same calls first on
device 0, then on device 1.  Limits that a kernel has per device (dynamic shared memory) are raised on both: no launch is
refused, and both devices run the same kernels."""
import pytest

import fake_cuda

RUN = """
from shape_atrophy_gb300 import _lib, api, problems
frame = problems.demo_strip(101, 31, timeEnd=0.01)
layered = problems.annulus_layered(steps=1)
shell = problems.shell_layered(level=5, lyrCntNum=9, steps=1, native=True)
for device in (0, 1):
    for spec, precision in ((frame, "fp64"), (layered, "fp64"), (layered, "mixed"), (dict(layered, ldmWgt=1e-2), "fp64"), (shell, "fp64")):
        r = api.forward(spec, objective=False, precision=precision, device=device)
        # kernels that do nothing leave mixed precision's outer residual where it is
        assert r["info"]["status"] == (0 if precision == "fp64" else _lib.SA_ERR_NOT_CONVERGED), r["info"]
    api.forward(dict(layered, cgKernel="persistent-global"), objective=False, device=device)
"""


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    return fake_cuda.run(RUN, tmp_path_factory.mktemp("cudart"))


def test_calls_succeed_on_both_devices(launches):
    r, lines = launches
    assert not [l for l in lines if "refused" in l[1]]
    assert r.returncode == 0, r.stderr[-2000:]


def test_both_devices_run_the_same_kernels(launches):
    _, lines = launches
    first, second = ([k for d, k in lines if d == dev] for dev in "01")
    assert any("k_kpcg_persist" in k for k in first) and any("k_cg_fix" in k for k in first)
    assert first == second
