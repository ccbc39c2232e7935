"""CPU: the library's host code over a CUDA runtime that runs nothing
(tests/fake_cuda.h, tests/host_checks.cpp): sizes of scratch buffers, what a
failing call leaves behind, budgets and plans, without a GPU."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "host_checks.cpp")
NAMES = re.findall(r'^\s+\{"(\w+)", \w+\},$', open(SRC).read(), re.M)


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    gxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not gxx or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no g++ or CUDA headers")
    out = str(tmp_path_factory.mktemp("host") / "host_checks")
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"), "-I",
                           os.path.join(ROOT, "skylens-stream-rs_gb300", "csrc"), "-I", inc, "-o", out, SRC, "-lpthread"])
    return out


@pytest.mark.parametrize("name", NAMES)
def test_host(exe, name):
    r = subprocess.run([exe, name], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
