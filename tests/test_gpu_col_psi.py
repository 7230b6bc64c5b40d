"""psi of every substep against its own tridiagonal system (LU_buildP) solved in extended precision: no
further from it than twice a sequential elimination of the same system in FP64, the reference's own form,
plus a few units of rounding (psi of later substeps is a small difference of pressures, so a comparison
with another run's psi says little)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
RKA = (4 / 15, 1 / 15, 1 / 6)


def thomas(a, b, c, r):
    cp, x = np.zeros_like(b), r.copy()
    cp[0], x[0] = c[0] / b[0], r[0] / b[0]
    for j in range(1, len(b)):
        m = 1 / (b[j] - a[j] * cp[j - 1])
        cp[j], x[j] = c[j] * m, (r[j] - a[j] * x[j - 1]) * m
    for j in range(len(b) - 2, -1, -1):
        x[j] -= cp[j] * x[j + 1]
    return x


@pytest.mark.parametrize("ny", [9, 31, 95, 351, 479, 607, 735])
def test_psi(ny):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    s = build_channel(tiny(ngal1=12, ngal2=16, ny=ny, posth=0.0, cyl_diameter=0.0, seed=ny))
    g, cfg = s.grid, s.cfg
    col = np.arange(cfg.ncol)
    q = col // cfg.nkx
    ch = Channel(s)
    ch.upload_state()

    def system(real, krk, div):
        kx, kz = (cfg.alp * (col % cfg.nkx)).astype(real), (cfg.bet * np.where(q < cfg.n2 // 2, q, q - cfg.n2)).astype(real)
        du, dv = g.dthdyu.astype(real)[1:-1], g.dthdyv.astype(real)
        lo, hi = du * dv[:-1], du * dv[1:]
        lo[0] = hi[-1] = 0
        a, c = lo[:, None] + 0 * kx, hi[:, None] + 0 * kx
        b = (-kx * kx - kz * kz) - lo[:, None] - hi[:, None]
        i = 1 - g.ju0
        b[0, 0], c[0, 0] = 1 / (real(g.yu[i + 1]) - real(g.yu[i])) ** 2, 0
        r = div / (real(s.dt) * 2 * real(RKA[krk - 1]))
        r[0, 0] = 0
        return thomas(a, b, c, r)

    for krk in (1, 2, 3):
        for stage in ("rhs0", "nonlinear", "solve_uvw", "meanflow", "solve_p"):
            getattr(ch, stage)(krk)
        div, psi = ch.download("div").T, ch.download("psi").T
        x = system(np.longdouble, krk, div.astype(np.clongdouble))
        n = np.linalg.norm(x.astype(complex))
        err = float(np.sqrt((np.abs(psi - x) ** 2).sum())) / n
        seq = float(np.sqrt((np.abs(system(np.float64, krk, div) - x) ** 2).sum())) / n
        assert err <= 2 * seq + 4 * 2.0 ** -52, (krk, err, seq)
        ch.vcorr(krk)
    ch.close()
