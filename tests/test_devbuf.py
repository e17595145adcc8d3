"""Device buffers follow the current GPU (as_devbuf.h, checked against a fake runtime)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def cuda_include():
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def test_buffers_follow_the_device(tmp_path):
    if not os.path.exists(os.path.join(cuda_include(), "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    exe = str(tmp_path / "devbuf_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "analogsat_b200", "csrc"),
                    "-I", cuda_include(), os.path.join(ROOT, "tests", "cpp", "devbuf_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "devbuf ok" in r.stdout, r.stderr
