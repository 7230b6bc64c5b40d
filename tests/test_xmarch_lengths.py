"""The marching x-line pass at the splits of 256, 288, 432, 512 and 576 points, and its FP64 layout with both
exchanges in one place, on the CPU: the checks of tests/xmarch_check.cu (test_xmarch_plan.py) and that
every cell either exchange touches lies in front of the history."""
import os
import subprocess

import pytest

from test_fft_prune import _nvcc

HERE = os.path.dirname(os.path.abspath(__file__))


def test_more_lengths(tmp_path):
    nvcc = _nvcc()
    if not nvcc:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "xmarch_lengths_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Wno-deprecated-gpu-targets", "-o", exe,
                    os.path.join(HERE, "xmarch_lengths_check.cu")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    lines = r.stdout.strip().splitlines()
    assert lines[-1] == "OK"
    assert sum(ln.startswith("roles ") for ln in lines) == 5 * 2 and sum(ln.startswith("shared ") for ln in lines) == 6
