"""cfd_tuning.xline_rows on the FP32-mixed x pass of lengths that are not among the named six: every number of
rows runs, is reported, and gives the same fields bit for bit (a row's transform does not depend on its
neighbours), also where the rows do not divide Ngal2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng1,ng2", [(36, 54), (648, 18), (192, 54)])
def test_rows(ng1, ng2):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    s = build_channel(tiny(ngal1=ng1, ngal2=ng2, ny=9, posth=0.0, cyl_diameter=0.0, seed=ng1))
    ref = None
    for rows in (0, 2, 4, 8):
        g = Channel(s, precision="mixed", tuning=dict(xline_rows=rows))
        t = g.tuning()
        assert t["xline_path"] == 1 and t["xline_rows"] == (rows or 4)
        g.upload_state()
        g.rhs0(1)
        g.nonlinear(1)
        got = {k: g.download(k) for k in ("nu1", "nu2", "nu3")}
        g.close()
        ref = ref or got
        for k in got:
            np.testing.assert_array_equal(got[k], ref[k])
