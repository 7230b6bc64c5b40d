"""cfd_rft's forward transform keeps its lines apart: neighbours twelve decades apart in size each within
1e-13 of numpy relative to themselves (log2(N) rounding errors of 1e-16), a zero line exactly zero, a NaN or
an infinity in its own line alone.  At every first step the two-step forms have, with line counts that fill
no CTA and pairs on 16 or only on 8 bytes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [12, 16, 18, 24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384, 432, 486, 512,
           576, 648, 768]


@pytest.mark.parametrize("pad", [2, 3])
@pytest.mark.parametrize("ng1", LENGTHS)
def test_lines_of_different_size(ng1, pad):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    g = Channel(build_channel(tiny(ngal1=ng1, ngal2=16, ny=9, posth=0.0, cyl_diameter=0.0), with_fields=False))
    rng = np.random.default_rng(ng1)
    m, h = 45, ng1 // 2 + 1
    scale = np.array([1.0, 1e-12, 1e6, 0.0, 1e-6, 1.0])[np.arange(m) % 6]
    x = rng.standard_normal((m, ng1 + pad)) * scale[:, None]
    x[8, 3] = np.nan
    x[20, ng1 - 1] = np.inf
    buf = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    g._chk(g.lib.cfd_rft(g.ctx, C.c_void_p(buf.data_ptr()), ng1 + pad, m, -1), "rft")
    g.synchronize()
    y = buf.cpu().numpy()
    g.close()
    got = np.ascontiguousarray(y[:, :2 * h]).view(complex)
    for r in range(m):
        if r in (8, 20):
            assert not np.isfinite(got[r]).any()
            continue
        ref = np.fft.rfft(x[r, :ng1]) / ng1
        if scale[r] == 0.0:
            assert not got[r].any()
        else:
            assert np.linalg.norm(got[r] - ref) < 1e-13 * np.linalg.norm(ref), r
    assert not got[:, 0].imag[np.isfinite(got[:, 0].real)].any() and not got[np.isfinite(got[:, -1].real), -1].imag.any()
    assert (y[:, 2 * h:] == x[:, 2 * h:]).all()
