"""The run-time transform plans of pfc_b200/csrc/fft_rt.cuh, checked on the CPU:
tests/host/fft_rt_check.cu compiles their host-and-device code for the host and
checks, for every even 7-smooth length from 8 to 8192 in both precisions, which
lengths have a plan, every address and division the passes use, and the
transform they compute."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc is not installed")
def test_run_time_plans_on_host(tmp_path):
    exe = tmp_path / "fft_rt_check"
    subprocess.run([NVCC, "-std=c++17", "-O1", "-o", str(exe), os.path.join(HERE, "host", "fft_rt_check.cu")],
                   check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
    assert out.stdout.strip().splitlines()[-1].endswith(" 0 failures"), out.stdout
