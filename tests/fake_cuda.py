"""Runs Python code over the built library with a CUDA runtime that has no GPU (fake_cudart.cpp): for CPU tests of the host
code.  Kernels do nothing, so results are zeros; the launches are what is looked at."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = "/usr/local/cuda/include"


def run(code, folder):
    """(the finished process, its launches as [device, kernel] pairs of texts)"""
    if not os.path.exists(os.path.join(CUDA, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    from shape_atrophy_gb300 import build
    build.build()
    with open(folder / "versions", "w") as f:
        f.write("libcudart.so.13 { global: *; };\n")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CUDA, "-Wl,-soname,libcudart.so.13",
                    f"-Wl,--version-script={folder}/versions", "-o", str(folder / "libcudart.so.13"),
                    os.path.join(HERE, "fake_cudart.cpp")], check=True)
    log = folder / "log"
    env = dict(os.environ, LD_LIBRARY_PATH=str(folder), FAKE_CUDART_LOG=str(log), PYTHONPATH=f"{ROOT}:{HERE}")
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    lines = [l.split(" ", 1) for l in log.read_text().splitlines()] if log.exists() else []
    return r, lines
