"""Forced planes whose x length has the two-step transform and whose z length has not: the z rows
left out of the x round trip lose Im of the kx = 0 entry like the others (the inverse real
transform ignores it, rft_buff.f:78-80).  FP64 against the oracle, 1e-11 relative L2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("ng1,ng2", [(64, 48), (128, 36), (64, 972)])
def test_unforced_rows_are_real(ng1, ng2):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(ngal1=ng1, ngal2=ng2, ny=17, cyl_diameter=0.3, cyl_spacing=0.9, seed=ng1))
    g, o = Channel(s), OracleChannel(s)
    g.upload_state()
    o.upload_state()
    for stage in ("rhs0", "nonlinear", "solve_uvw"):
        getattr(g, stage)(1)
        getattr(o, stage)(1)
    for k in ("du1", "du2", "du3", "u1", "u2", "u3"):
        assert rel(g.download(k), o.download(k)) < 1e-11, k
    g.close()
