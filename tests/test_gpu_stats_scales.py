"""The statistics of quantities of very different size: w and p nine decades below u and v.  A quantity's
rounding is relative to itself, so each sum lies within 1e-12 (some 1e5 terms of a few rounding errors each)
of the size its own factors give it, against the oracle; the CFL terms within 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng1,ng2,ny,dnx,dnz", [(12, 18, 17, 12, 18), (64, 36, 17, 8, 9), (384, 48, 9, 96, 12), (192, 162, 30, 8, 27),
                                                (768, 16, 9, 3, 4)])
def test_small_and_large(ng1, ng2, ny, dnx, dnz):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(ngal1=ng1, ngal2=ng2, ny=ny, cyl_diameter=0.0, seed=ng1))
    g, o = Channel(s), OracleChannel(s)
    o.upload_state()
    o.step(1)
    st = o.download_state()
    st["u3"], st["p"] = 1e-9 * st["u3"], 1e-9 * st["p"]
    for c in (g, o):
        c.upload_state(st)
        c.stats_configure(0, dnx, dnz, spectra=False)
        c.stats_accumulate()
    a, b = g.stats_read(), o.stats_read()
    n = ng1 * ng2
    for tail, m in (("", n), ("C", n / (dnx * dnz))):  # points of a plane, points folded onto one of the tile
        top = {k: np.abs(b[k + "2m" + tail]).max() for k in ("U", "V", "W", "P", "wx")}
        size = {k + "2m": v for k, v in top.items()}
        size.update({k + "m": np.sqrt(v * m) for k, v in top.items()})
        size.update({k + "m": np.sqrt(top[k[0]] * top[k[1]]) for k in ("UV", "UW", "VW")})
        for k, v in size.items():
            assert np.abs(a[k + tail] - b[k + tail]).max() <= 1e-12 * v, (k + tail, v)
    np.testing.assert_allclose(g.cfl()[1], o.cfl()[1], rtol=1e-12)
    g.close()
