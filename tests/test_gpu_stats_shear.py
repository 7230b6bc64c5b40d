"""omega_x where w hardly changes from plane to plane (1e-6 of itself over the channel): the difference is
taken from the state, not from transforms that have rounded w already, so the sums of omega_x lie within 1e-12
of their size (some 1e5 terms of a few rounding errors each) of the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng1,ng2,ny,dnx,dnz", [(12, 18, 17, 12, 18), (64, 36, 17, 8, 9), (192, 162, 30, 8, 27)])
def test_omega_x_of_a_weak_shear(ng1, ng2, ny, dnx, dnz):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(ngal1=ng1, ngal2=ng2, ny=ny, cyl_diameter=0.0, seed=ng1))
    cfg, y = s.cfg, s.grid.yu
    rng = np.random.default_rng(ng1)
    a = (rng.standard_normal((cfg.n2, cfg.nkx)) + 1j * rng.standard_normal((cfg.n2, cfg.nkx))) / (1.0 + np.arange(cfg.nkx) ** 2)
    a[:, 0] = 0
    a[0, 0] = 1.0
    st = s.state()
    st = {"u1": st["u1"], "u2": np.zeros_like(st["u2"]), "p": st["p"], "u3": a.reshape(-1, 1) * (1 + 1e-6 * np.sin(y))}
    g, o = Channel(s), OracleChannel(s)
    for c in (g, o):
        c.upload_state(st)
        c.stats_configure(0, dnx, dnz, spectra=False)
        c.stats_accumulate()
    x, ref = g.stats_read(), o.stats_read()
    for tail, m in (("", ng1 * ng2), ("C", ng1 * ng2 / (dnx * dnz))):
        top = np.abs(ref["wx2m" + tail]).max()
        assert np.abs(x["wx2m" + tail] - ref["wx2m" + tail]).max() <= 1e-12 * top
        assert np.abs(x["wxm" + tail] - ref["wxm" + tail]).max() <= 1e-12 * np.sqrt(top * m)
    g.close()
