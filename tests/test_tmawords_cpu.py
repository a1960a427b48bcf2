"""CPU: the words through which kernels report a bulk copy that did not arrive are set up once per handle, whole, whichever threads
come first (mem.cu on a stand-in for the CUDA runtime, tests/tmawords/)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

HERE = os.path.join(ROOT, "tests", "tmawords")


def test_words_of_a_handle_for_several_threads(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    out, cuda = str(tmp_path / "driver"), os.path.join(PKG, "csrc", "cuda")
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-include", "math.h", "-D__cvta_generic_to_shared(p)=(size_t)(p)", "-I", include,
                    "-I", os.path.join(ROOT, "include"), "-I", cuda, "-o", out,
                    "-x", "c++", os.path.join(cuda, "mem.cu"), os.path.join(HERE, "main.cpp"), "-lpthread"], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
