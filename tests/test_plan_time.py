"""What an upload pays for planning half-range passes, on the CPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dm-sim_gb300", "csrc")


def test_half_range_planning_time(tmp_path):
    """No more than six times the additions of the search alone (measured: 1.1;
    10 when each step worked the passes' times out again)."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "plan_time_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "plan_time_check.cpp"), os.path.join(CSRC, "plan.cpp"),
                    os.path.join(CSRC, "gates.cpp"), "-o", exe], check=True, capture_output=True, text=True,
                   timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
