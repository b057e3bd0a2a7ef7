"""The threaded copies of large host arrays (koral-zig_b200/csrc/kc_host_copy.cuh) on
the host, against a stand-in for the runtime calls whose copies run as late as the
waits allow (host_copy_check.cpp): sizes around the staged minimum and its chunks,
page-locked arrays, several threads, the area given back and made again, device resets,
failing copies, helper threads that cannot be made."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _cuda_include():
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def test_threaded_host_copies(tmp_path):
    inc = _cuda_include()
    if not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    exe = tmp_path / "host_copy_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", inc, "-o", str(exe),
                    os.path.join(HERE, "host_copy_check.cpp")], check=True)
    for _ in range(3):
        r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0 and r.stdout.split() == ["0"], r.stdout + r.stderr
