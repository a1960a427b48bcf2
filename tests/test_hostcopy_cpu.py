"""CPU: the staged host -> device copies (hostcopy.cu) on a stand-in for the CUDA runtime that carries every
asynchronous copy out as late as the runtime may (tests/hostcopy/)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

HERE = os.path.join(ROOT, "tests", "hostcopy")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    out = str(tmp_path_factory.mktemp("hostcopy") / "driver")
    cuda = os.path.join(PKG, "csrc", "cuda")
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-include", "math.h", "-I", include, "-I", os.path.join(ROOT, "include"), "-I", cuda, "-I", HERE, "-o", out,
                    "-x", "c++", os.path.join(cuda, "hostcopy.cu"), os.path.join(HERE, "fake_runtime.cpp"), os.path.join(HERE, "main.cpp"),
                    "-lpthread"], check=True)
    return out


@pytest.mark.parametrize("scenario", ["sizes", "panels", "threads", "capture", "capture_elsewhere", "failed_copy", "other_device"])
def test_staged_copies(driver, scenario):
    r = subprocess.run([driver, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
