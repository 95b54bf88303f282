"""One process, two devices: the host code runs over a CUDA runtime without a GPU (fake_cudart.cpp), the same calls first on
device 0, then on device 1.  Limits that a kernel has per device (dynamic shared memory) are raised on both: no launch is
refused, and both devices run the same kernels."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = "/usr/local/cuda/include"

RUN = """
import sys
sys.path.insert(0, {root!r})
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
    if not os.path.exists(os.path.join(CUDA, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    from shape_atrophy_gb300 import build
    build.build()
    out = tmp_path_factory.mktemp("cudart")
    with open(out / "versions", "w") as f:
        f.write("libcudart.so.13 { global: *; };\n")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CUDA, "-Wl,-soname,libcudart.so.13",
                    f"-Wl,--version-script={out}/versions", "-o", str(out / "libcudart.so.13"),
                    os.path.join(HERE, "fake_cudart.cpp")], check=True)
    log = out / "log"
    env = dict(os.environ, LD_LIBRARY_PATH=str(out), FAKE_CUDART_LOG=str(log))
    r = subprocess.run([sys.executable, "-c", RUN.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=600)
    lines = [l.split(" ", 1) for l in log.read_text().splitlines()] if log.exists() else []
    return r, lines


def test_calls_succeed_on_both_devices(launches):
    r, lines = launches
    assert not [l for l in lines if "refused" in l[1]]
    assert r.returncode == 0, r.stderr[-2000:]


def test_both_devices_run_the_same_kernels(launches):
    _, lines = launches
    first, second = ([k for d, k in lines if d == dev] for dev in "01")
    assert any("k_kpcg_persist" in k for k in first) and any("k_cg_fix" in k for k in first)
    assert first == second
