"""Staged copies from the device against a faked runtime: the bytes arrive at
every size, and errors are neither lost nor left behind."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "moldy_b200", "csrc")


def test_staged_copies_and_their_errors(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not gxx or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime_api.h")):
        pytest.skip("no host compiler or CUDA headers")
    exe = str(tmp_path / "copystage")
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", os.path.join(cuda, "include"), os.path.join(HERE, "fake_cudart.cpp"),
                    os.path.join(CSRC, "copystage.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
