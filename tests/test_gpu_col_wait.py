"""The waits of the column solves (k_col_solve) for their transfers, when they run out: a group of warps
leaves as one, the fields stay as they were, and the calls that synchronise say so until a new state is
uploaded."""
import os
import subprocess

import numpy as np
import pytest

from test_fft_prune import _nvcc

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def test_group_leaves_as_one(torch_cuda, tmp_path):
    nvcc = _nvcc()
    if not nvcc:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "col_wait_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "col_wait_check.cu")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout + r.stderr


@pytest.mark.parametrize("kw", [dict(), dict(flag_ctpress=0, qxt=2.0), dict(ngal2=96, band_vface=4, ngal1_mid=18, ngal2_mid=64)])
def test_wait_that_runs_out_is_reported(torch_cuda, monkeypatch, kw):
    from cfd_b200.capi import CfdError
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from cfd_b200.ensemble import Ensemble
    monkeypatch.setenv("CFD_SOLVE_TRIES", "0")
    s = build_channel(tiny(**{**dict(ngal1=24, ngal2=18, ny=29, cyl_diameter=0.0, posth=0.0, seed=2), **kw}))
    g = Channel(s)
    g.upload_state()
    before = g.download_state()
    g.step(1)
    for call in (g.synchronize, g.scalars, g.divergence_max, lambda: g.step(1), lambda: g.rhs0(1),
                 lambda: g.download("u1"), lambda: Ensemble([g]).step(1)):
        with pytest.raises(CfdError, match="column solves"):
            call()
    g.upload_state()  # a new state: the fields are defined again
    after = g.download_state()
    for k in before:
        np.testing.assert_array_equal(after[k], before[k])
    for stage in ("solve_uvw", "solve_p"):  # the stage calls' forms of the kernel
        getattr(g, stage)(1)
        with pytest.raises(CfdError, match="column solves"):
            g.synchronize()
        g.upload_state()
    e = Ensemble([g])
    e.step(1)
    with pytest.raises(CfdError, match="column solves"):
        e.synchronize()
    e.close()
    g.close()
