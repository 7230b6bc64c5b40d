"""The forcing in row groups gives the same bits every time: groups of an odd number of rows, whose last
row shares a forward transform with a line that holds no row, while z row 0 is forced by a group of its
own.  The fields of equal substeps are compared bit for bit."""
import numpy as np
import pytest

from test_gpu_ib_groups import points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ng1", [48, 384])
def test_odd_groups_repeat(precision, ng1):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    s = build_channel(tiny(ngal1=ng1, ngal2=108, ny=17, cyl_diameter=0.3, cyl_spacing=0.9, seed=3))
    s.ibu, s.ibv = points(np.random.default_rng(1), s, s.ibu, "seven"), points(np.random.default_rng(1), s, s.ibv, "seven")
    assert (s.ibu.idx[:, 1] == 1).any() and (s.ibv.idx[:, 1] == 1).any()  # z row 0 is forced
    g = Channel(s, precision=precision)
    first = None
    for _ in range(12):
        g.upload_state()
        for stage in ("rhs0", "nonlinear", "solve_uvw"):
            getattr(g, stage)(1)
        got = {k: g.download(k) for k in ("du1", "du2", "du3")}
        first = first or got
        for k in got:
            np.testing.assert_array_equal(got[k], first[k])
    g.close()
