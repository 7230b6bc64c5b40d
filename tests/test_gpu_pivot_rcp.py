"""The reciprocal that the column solves take of their pivots lies within one unit in the last place of 1/x,
which is what its comment says: tests/pivot_rcp_check.cu compares a thousand million normal values of either
sign, from 2^-1000 to 2^999, the neighbours of powers of two among them."""
import os
import subprocess

import pytest

from test_fft_prune import _nvcc

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_within_an_ulp(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nvcc = _nvcc()
    if not nvcc:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "pivot_rcp_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "pivot_rcp_check.cu")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
