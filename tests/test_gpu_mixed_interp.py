"""FP32-mixed contexts interpolate u, v, w in y in FP64 unless both lengths are among the named six: u
alternates from plane to plane so that its values at the faces are 1e-4 of those at the centres, and the
products uv of the v planes are those of the small values.  FP32 interpolation leaves them 1e-4 of the large
ones' rounding, 6e-4, off; interpolated in FP64 and rounded once they keep the 1e-5 relative L2 of the
FP32-mixed path against the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# neither length named, one that marches on request, x named, z named
@pytest.mark.parametrize("ng1,ng2", [(36, 54), (256, 18), (384, 54), (54, 192), (18, 648)])
def test_interpolation_keeps_fp64(ng1, ng2):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(ngal1=ng1, ngal2=ng2, ny=17, posth=0.0, cyl_diameter=0.0, seed=ng1))
    g, cfg = s.grid, s.cfg
    rng = np.random.default_rng(ng2)

    def amp():
        a = rng.standard_normal((cfg.n2, cfg.nkx)) + 1j * rng.standard_normal((cfg.n2, cfg.nkx))
        a /= 1.0 + np.arange(cfg.nkx) ** 2
        a[:, 0] = 0
        a[cfg.n2 // 2] = 0
        return a.reshape(-1, 1)

    fa = (g.yv - g.yu[:-1]) / (g.yu[1:] - g.yu[:-1])
    b = np.ones(g.nyu)
    for j in range(g.nyv):
        b[j + 1] = -b[j] * (1 - fa[j]) / fa[j]  # nothing is left at the face
    b /= np.abs(b).max()
    st = {"u1": amp() * (b + 1e-4 * np.cos(g.yu)), "u2": 1e-4 * amp() * (1 - g.yv ** 2),
          "u3": np.zeros((cfg.ncol, g.nyu), complex), "p": np.zeros((cfg.ncol, g.nyp), complex)}
    o, m = OracleChannel(s), Channel(s, precision="mixed")
    for c in (o, m):
        c.upload_state(st)
        c.nonlinear(1)
    a, ref = m.download("nu2"), o.download("nu2")
    m.close()
    assert np.linalg.norm(a - ref) < 1e-5 * np.linalg.norm(ref)
