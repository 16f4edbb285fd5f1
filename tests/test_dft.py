"""The small DFTs of the FP64 FFT (csrc/dft.cuh, compiled here for the host with g++) against the sums
that define them, radices 2 .. 16, FP64 and FP32 (tests/dft_check.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def test_small_dfts_match_their_definition(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no g++ or CUDA headers")
    exe = str(tmp_path / "dft_check")
    subprocess.check_call([gxx, "-std=c++17", "-O2", "-I", CUDA, "-I", os.path.join(ROOT, "bacterial-droplet_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "dft_check.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
