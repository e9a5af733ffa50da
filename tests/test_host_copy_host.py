"""The pinned chunks of pfc_b200/csrc/host_copy.cu, checked on the CPU over a stand-in
for the CUDA runtime (tests/host/host_copy_check.cpp): callers that move their fields
once pin nothing, others once, and the last one gives the chunks back."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc is not installed")
def test_pinned_chunks_on_host(tmp_path):
    exe = tmp_path / "host_copy_check"
    subprocess.run([NVCC, "-std=c++17", "-O1", "-cudart", "none", "-x", "c++", "-o", str(exe),
                    os.path.join(HERE, "host", "host_copy_check.cpp"), "-lpthread"],
                   check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
    assert out.stdout.strip().splitlines()[-1] == "0 failures", out.stdout
