"""The exact form's wave speed over the whole range of the format, on the CPU
(host code compiled by nvcc; no GPU needed)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not available")
def test_wave_speed_is_the_references_at_any_magnitude(tmp_path):
    exe = str(tmp_path / "wave_speed_check")
    subprocess.run([NVCC, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler",
                    "-ffp-contract=off", f"-I{os.path.join(os.path.dirname(HERE), 'sddc_b200', 'csrc')}",
                    os.path.join(HERE, "native", "wave_speed_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
