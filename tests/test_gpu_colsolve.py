"""The warp-per-column solves (k_col_solve) at the heights where their partition changes: rows
that fill every lane, one row more, the rows per lane that solve u and w one at a time, a
column too tall for them (the sweeps run), a column count no group size divides, and groups of
eight columns.  Against the FP64 oracle: each stage to 1e-11 and two fused steps to 1e-10
relative L2, the bounds of the other FP64 parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# ny + 1 planes: 32 M of them for M = 1, 3, 11, 15, 19, 23, one more, and the least
HEIGHTS = [9, 31, 32, 95, 351, 352, 479, 607, 735, 736]


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("group", ["4", "8"])
@pytest.mark.parametrize("ny", HEIGHTS)
def test_column_solves(torch_cuda, monkeypatch, ny, group):
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    monkeypatch.setenv("CFD_SOLVE_GROUP", group)
    # 50 columns; constant flow rate, so that the mean mode follows the fused solve
    s = build_channel(tiny(ngal1=12, ngal2=16, ny=ny, posth=0.0, cyl_diameter=0.0, flag_ctpress=0, qxt=2.0, seed=ny))
    g, o = Channel(s), OracleChannel(s)
    g.upload_state()
    o.upload_state()
    for krk in (1, 2):
        for stage in ("rhs0", "nonlinear", "solve_uvw", "meanflow", "solve_p", "vcorr"):
            getattr(g, stage)(krk)
            getattr(o, stage)(krk)
            # psi of the second substep is a small difference of pressures: solved in extended
            # precision it lies 1e-11 from the oracle's sequential sweep, so p stands for it
            for k in ("u1", "u2", "u3", "p") + (("psi",) if krk == 1 else ()):
                e = rel(g.download(k), o.download(k))
                assert e < 1e-11, (krk, stage, k, e)
    g.step(2)
    o.step(2)
    a, b = g.download_state(), o.download_state()
    for k in a:
        assert rel(a[k], b[k]) < 1e-10, (k, rel(a[k], b[k]))
    assert g.scalars()["mpgx"] == pytest.approx(o.scalars()["mpgx"], rel=1e-10)
    g.close()


@pytest.mark.parametrize("ny", [95, 352])
def test_segment_solves(torch_cuda, ny):
    """The same for a three-band channel, whose short columns are two segments with identity
    rows between them."""
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(ngal1=16, ngal2=96, ny=ny, posth=0.0, cyl_diameter=0.0, seed=ny, band_vface=ny // 5,
                           ngal1_mid=12, ngal2_mid=64))
    g, o = Channel(s), OracleChannel(s)
    g.upload_state()
    o.upload_state()
    for stage in ("rhs0", "nonlinear", "solve_uvw", "meanflow", "solve_p", "vcorr"):
        getattr(g, stage)(1)
        getattr(o, stage)(1)
        for k in ("u1", "u2", "u3", "p", "psi", "div", "du1", "du2", "du3"):
            a, b = g.download(k), o.download(k)
            if k != "div" or stage == "solve_p":
                assert rel(a, b) < 1e-11, (stage, k, rel(a, b))
    g.step(2)
    o.step(2)
    a, b = g.download_state(), o.download_state()
    for k in a:
        assert rel(a[k], b[k]) < 1e-10, (k, rel(a[k], b[k]))
    g.close()
