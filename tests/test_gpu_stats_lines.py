"""The statistics pass and the CFL query on rows and lines (k_st_z, k_st_x) where their chunks and
tiles change: chunks of a few planes (a tile as wide as the channel on long rows), the narrowest
tile, several chunks, rows that no CTA divides evenly.  Against the oracle: sums within 1e-12 of the
largest of their kind (some 1e5 terms of a few rounding errors each), the CFL terms within 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng1,ng2,ny,dnx,dnz", [(12, 18, 17, 12, 18), (54, 36, 17, 1, 1), (768, 384, 9, 768, 384),
                                                (192, 162, 60, 8, 27), (24, 648, 9, 3, 4)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sums_and_cfl(ng1, ng2, ny, dnx, dnz, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(ngal1=ng1, ngal2=ng2, ny=ny, cyl_diameter=0.0, seed=ng1))
    g, o = Channel(s, precision=precision), OracleChannel(s)
    o.upload_state()
    o.step(1)
    g.upload_state(o.download_state())
    for c in (g, o):
        c.stats_configure(0, dnx, dnz, spectra=False)
        c.stats_accumulate()
        c.stats_accumulate()
    a, b = g.stats_read(), o.stats_read()
    for k in b:
        if k == "istat":
            assert a[k] == b[k] == 2
        else:
            top = max(np.abs(b[k]).max(initial=0.0), np.abs(b["U2m" + k[len(k.rstrip("C")):]]).max(initial=0.0))
            assert np.abs(a[k] - b[k]).max(initial=0.0) <= 1e-12 * top, k
    (da, ta), (db, tb) = g.cfl(), o.cfl()
    np.testing.assert_allclose(da, db, rtol=1e-12)
    np.testing.assert_allclose(ta, tb, rtol=1e-12)
    g.close()


@pytest.mark.parametrize("off,pad", [(0, 2), (1, 2), (0, 3), (1, 5)])
@pytest.mark.parametrize("ng1,ng2,m", [(12, 18, 1), (54, 36, 7), (384, 192, 33), (768, 648, 2)])
def test_line_transforms(ng1, ng2, m, off, pad):
    """cfd_rft and cfd_cft on lines whose pairs lie on 16 or only on 8 bytes, and line counts that
    fill no CTA: within 1e-13 of numpy relative L2 (log2(N) rounding errors of 1e-16)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ctypes as C
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    g = Channel(build_channel(tiny(ngal1=ng1, ngal2=ng2, ny=9, posth=0.0, cyl_diameter=0.0), with_fields=False))
    rng = np.random.default_rng(m)

    def rel(a, b):
        return np.linalg.norm(a - b) / np.linalg.norm(b)

    def call(f, x, *args):
        buf = torch.zeros(off + x.size, dtype=torch.float64, device="cuda")
        buf[off:] = torch.from_numpy(x).cuda().ravel()
        torch.cuda.synchronize()
        g._chk(f(g.ctx, C.c_void_p(buf.data_ptr() + 8 * off), *args), "transform")
        g.synchronize()
        return buf[off:].cpu().numpy().reshape(x.shape)

    x = rng.standard_normal((m, ng1 + pad))
    h = ng1 // 2 + 1
    y = call(g.lib.cfd_rft, x, ng1 + pad, m, -1)
    ref = np.fft.rfft(x[:, :ng1], axis=1) / ng1
    assert rel(y[:, :2 * h:2] + 1j * y[:, 1:2 * h:2], ref) < 1e-13
    assert (y[:, 2 * h:] == x[:, 2 * h:]).all()
    sp = x[:, :2 * h:2] + 1j * x[:, 1:2 * h:2]
    y = call(g.lib.cfd_rft, x, ng1 + pad, m, 1)
    assert rel(y[:, :ng1], np.fft.irfft(sp, n=ng1, axis=1) * ng1) < 1e-13
    # complex lines down the rows: element stride 2 m + pad - 2, line stride 2
    ise = 2 * m + pad - 2
    x = rng.standard_normal((ng2, ise))
    z = x[:, :2 * m:2] + 1j * x[:, 1:2 * m:2]
    for iopt, ref in ((-1, np.fft.fft(z, axis=0) / ng2), (1, np.fft.ifft(z, axis=0) * ng2)):
        y = call(g.lib.cfd_cft, x, ise, 2, m, iopt)
        assert rel(y[:, :2 * m:2] + 1j * y[:, 1:2 * m:2], ref) < 1e-13
        assert (y[:, 2 * m:] == x[:, 2 * m:]).all()
    g.close()
