"""Each entry of a column solve, not only its norm: a right-hand side in one row, whose solution falls by some
orders from row to row, against the tridiagonal system solved in extended precision.  An entry is a product of
one factor a row, each with some twelve roundings (coefficients, pivot, couplings): relative error below
12 n 2^-53 on n rows, down to 1e-250."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def thomas(a, b, c, r):
    n = r.shape[0]
    cp, x = np.zeros(n, np.longdouble), r.astype(np.longdouble)
    cp[0], x[0] = c[0] / b[0], x[0] / b[0]
    for j in range(1, n):
        m = b[j] - a[j] * cp[j - 1]
        cp[j], x[j] = c[j] / m, (x[j] - a[j] * x[j - 1]) / m
    for j in range(n - 2, -1, -1):
        x[j] -= cp[j] * x[j + 1]
    return x


@pytest.mark.parametrize("at", [0.02, 0.5, 0.97])
@pytest.mark.parametrize("ny", [9, 31, 95, 257, 480, 610, 735])
def test_entries(ny, at):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from cfd_b200.grid import grid_weights
    s = build_channel(tiny(ngal1=12, ngal2=16, ny=ny, posth=0.0, cyl_diameter=0.0, seed=ny))
    g, cfg, L = s.grid, s.cfg, np.longdouble
    s.dt = float(2e-3 * np.diff(g.yv).min() ** 2 * cfg.re_b)  # couplings of a few 1e-3
    st = {k: np.zeros_like(v) for k, v in s.state().items()}
    row = max(1, min(g.nyu - 2, int(at * g.nyu)))
    st["u1"][:, row], st["u3"][:, row] = 1.0, 1j
    st["u2"][:, max(1, min(g.nyv - 2, row))] = 1.0
    ch = Channel(s)
    ch.upload_state(st)
    for k, n in (("du1", g.nyu), ("du2", g.nyv), ("du3", g.nyu)):
        ch.upload(k, np.zeros((cfg.ncol, n), complex))
    ch.solve_uvw(1)
    beta = L(4) / 15 * L(s.dt) / L(cfg.re_b)
    gwb, gwt = grid_weights(g)[:2]
    seen = 0
    for col in (0, 5, cfg.ncol // 2 + 3):
        i, q = col % cfg.nkx, col // cfg.nkx
        kz = cfg.bet * (q if q < cfg.n2 // 2 else q - cfg.n2)
        k2 = -L(cfg.alp * i) ** 2 - L(kz) ** 2
        for k, w, e0, e1 in (("u1", g.dyu2i, gwb, gwt), ("u2", g.dyv2i, 0.0, 0.0)):
            w = np.asarray(w).reshape(-1, 3).astype(L)
            a, b, c = -beta * w[:, 0], 1 - beta * (w[:, 1] + k2), -beta * w[:, 2]
            a[0], b[0], c[0], a[-1], b[-1], c[-1] = 0, 1, e0, e1, 1, 0
            x, y = thomas(a, b, c, st[k][col].real)[1:-1], ch.download(k)[col][1:-1]
            big = np.abs(x) > 1e-250
            assert np.abs(y[big].imag).max() == 0.0
            err = np.abs(y[big].real - x[big]) / np.abs(x[big])
            assert err.max() <= 12 * len(b) * 2.0 ** -53, (k, col, int(err.argmax()), float(err.max()))
            seen += int((np.abs(x[big]) < 1e-30).sum())
    assert ny < 20 or seen > 0
    ch.close()
