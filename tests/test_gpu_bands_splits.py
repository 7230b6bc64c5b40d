"""Three-band channels with cylinders at the z lengths whose one-band default is the transposed split
(192 and 768 points) and with that split asked for: the forcing's z passes run the plain split there, and
their launches have its shared memory.  Against the FP64 oracle, the bounds of the other three-band tests:
1e-11 relative L2 stage by stage in FP64, 1e-5 on u, v, w after two FP32-mixed steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STAGES = ("rhs0", "nonlinear", "solve_uvw", "meanflow", "solve_p", "vcorr")
FIELDS = ("u1", "u2", "u3", "p", "du1", "du2", "du3", "nu1", "nu2", "nu3")
CASES = [(dict(ngal1=48, ngal2=192, ny=29, band_vface=5, ngal1_mid=24, ngal2_mid=96), None),
         (dict(ngal1=96, ngal2=768, ny=17, band_vface=4, ngal1_mid=48, ngal2_mid=64, cyl_diameter=0.1, cyl_spacing=0.5), None),
         (dict(ngal1=48, ngal2=96, ny=29, band_vface=5, ngal1_mid=24, ngal2_mid=64), dict(zsplit=2, zlines=16))]


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("kw,tuning", CASES)
def test_forced_bands(kw, tuning):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(**{"cyl_diameter": 0.3, "cyl_spacing": 1.5, "seed": 9, **kw}))
    assert s.ibu.n > 0 and s.ibv.n > 0
    g, o = Channel(s, precision="fp64", tuning=tuning), OracleChannel(s)
    assert g.tuning()["zsplit"] == 1
    g.upload_state()
    o.upload_state()
    for krk in (1, 2):
        for stage in STAGES:
            getattr(g, stage)(krk)
            getattr(o, stage)(krk)
            for k in FIELDS:
                e = rel(g.download(k), o.download(k))
                assert e < 1e-11, (krk, stage, k, e)
    g.close()
    o = OracleChannel(s)
    o.upload_state()
    o.step(2)
    ref = o.download_state()
    m = Channel(s, precision="mixed", tuning=tuning)
    m.upload_state()
    m.step(2)
    st = m.download_state()
    for k in ("u1", "u2", "u3"):
        assert rel(st[k], ref[k]) < 1e-5, (k, rel(st[k], ref[k]))
    m.close()
