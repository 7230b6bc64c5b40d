"""cfd_tuning.rhs_chunk over the range that the library chooses from: what cfd_get_tuning reports can be asked
for, one plane per thread included, on a small and on an ordinary grid, with the same fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng1,ng2,ny", [(24, 18, 17), (96, 96, 33)])
def test_every_chunk(ng1, ng2, ny):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    s = build_channel(tiny(ngal1=ng1, ngal2=ng2, ny=ny, cyl_diameter=0.0, seed=3))
    ref = None
    for chunk in (0, 1, 2, 3, 7, 64):
        g = Channel(s, tuning=dict(rhs_chunk=chunk))
        assert chunk == 0 or g.tuning()["rhs_chunk"] == chunk
        h = Channel(s, tuning=g.tuning())
        assert h.tuning() == g.tuning()
        h.close()
        g.upload_state()
        g.rhs0(1)
        g.nonlinear(1)
        g.solve_uvw(1)
        got = {k: g.download(k) for k in ("du1", "du2", "du3", "nu1", "nu2", "nu3")}
        g.close()
        ref = ref or got
        for k in got:
            np.testing.assert_array_equal(got[k], ref[k])  # a plane's value does not depend on its chunk
