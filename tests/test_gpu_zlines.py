"""Every number of z lines a CTA that cfd_tuning takes, on the x-line path without a register x transform and
in three bands, at the z lengths whose FP64 kernels hold the most registers: the context steps, and the
nonlinear term of u lies within 1e-11 relative L2 of the oracle's (1e-4 FP32-mixed: products of FP32 fields times
ik, 3e-5 off at any length)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [dict(ngal1=12, ngal2=n, ny=9) for n in (432, 486, 512, 576, 648, 768)] + \
        [dict(ngal1=24, ngal2=768, ny=17, band_vface=4, ngal1_mid=16, ngal2_mid=384)]


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("zlines", [4, 8, 16])
@pytest.mark.parametrize("kw", CASES)
def test_zlines(kw, zlines):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(posth=0.0, cyl_diameter=0.0, seed=zlines, **kw))
    o = OracleChannel(s)
    o.upload_state()
    o.nonlinear(1)
    for precision in ("fp64", "mixed"):
        g = Channel(s, precision=precision, tuning=dict(xline_path=2, zlines=zlines))
        g.upload_state()
        g.nonlinear(1)
        assert rel(g.download("nu1"), o.download("nu1")) < (1e-11 if precision == "fp64" else 1e-4)
        g.step(1)
        g.synchronize()
        g.close()
