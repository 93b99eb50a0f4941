"""Launchers in a process with more than one CUDA context (a second device, or
the same one after a reset): the compiled launchers against a fake runtime, on
the CPU."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "dm-sim_gb300")
UNITS = ["kernels.cu", "kernels_real.cu", "kernels_k1.cu", "kernels_mono.cu", "tensor.cu", "tensor64.cu", "tensor32.cu"]


def test_launchers_in_every_context(tmp_path):
    sys.path.insert(0, PKG)
    try:
        import build as engine_build  # the engine's own objects, compiled if stale
    finally:
        sys.path.remove(PKG)
    gxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if gxx is None or not os.path.exists(nvcc):
        pytest.skip("no compiler")
    engine_build.build()
    exe = str(tmp_path / "context_check")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", engine_build.CSRC, "-I", engine_build.INCLUDE,
                    "-I", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "cpp", "context_check.cpp")] +
                   [os.path.join(engine_build.BUILD, u + ".o") for u in UNITS] + ["-lpthread", "-o", exe],
                   check=True, capture_output=True, text=True, timeout=600)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout[:3000] + out.stderr
