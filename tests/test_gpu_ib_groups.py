"""The forcing in groups of z rows (k_ib_zin, k_ib_force_x, k_ib_zout) and the point lists that keep it
from running: stencils that tie single rows, pairs, seven rows, more rows than a group of eight
holds, a stencil in another plane, repeated targets.  Against the FP64 oracle, right-hand sides and
velocities to 1e-11 relative L2 (the stage bound of the other parity tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def points(rng, s, lst, which):
    """A list on the planes of lst: targets (i, k, j), stencils by kind."""
    ng1, ng2 = s.cfg.ngal1, s.cfg.ngal2
    j = np.unique(lst.idx[:, 2])
    n = 400
    i, k, jj = rng.integers(1, ng1 + 1, n), rng.integers(1, ng2 + 1, n), rng.choice(j, n)
    if which == "single":
        k2 = k3 = k
    elif which == "pair":
        k2, k3 = (k - 1) // 2 * 2 + 1, (k - 1) // 2 * 2 + 2
    elif which == "seven":
        k2 = k3 = np.minimum((k - 1) // 7 * 7 + 1 + (k % 7), ng2)
    elif which == "fourteen":
        k2 = k3 = np.minimum((k - 1) // 14 * 14 + 1 + (k % 14), ng2)
    else:  # one component of every row
        k2, k3 = k % ng2 + 1, k
    j2 = np.where(rng.random(n) < 0.5, jj, j[0]) if which == "plane" else jj
    idx = np.stack([i, k, jj, rng.integers(1, ng1 + 1, n), k2, j2, rng.integers(1, ng1 + 1, n), k3, jj], 1)
    idx = np.concatenate([idx, idx[:40]])  # repeated targets
    w = np.stack([rng.choice([0.0, 1.0], n + 40), rng.uniform(-1, 1, n + 40), rng.uniform(-1, 1, n + 40)], 1)
    o = np.lexsort((idx[:, 0], idx[:, 1], idx[:, 2]))
    return type(lst)(np.ascontiguousarray(idx[o], dtype=np.int32), np.ascontiguousarray(w[o]), lst.jlo, lst.jhi)


@pytest.mark.parametrize("groups", ["1", "0"])
@pytest.mark.parametrize("which", ["single", "pair", "seven", "fourteen", "all", "plane"])
def test_point_lists(monkeypatch, which, groups):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    monkeypatch.setenv("CFD_IB_GROUPS", groups)
    s = build_channel(tiny(ngal1=48, ngal2=54, ny=17, cyl_diameter=0.3, cyl_spacing=0.9, seed=3))
    rng = np.random.default_rng(7)
    s.ibu, s.ibv = points(rng, s, s.ibu, which), points(rng, s, s.ibv, which)
    g, o = Channel(s), OracleChannel(s)
    g.upload_state()
    o.upload_state()
    for upload in (False, True):  # with the nonlinear pass's transforms of the velocities, and without
        for stage in ("rhs0", "nonlinear", "solve_uvw"):
            if upload and stage == "solve_uvw":
                g.upload("u1", g.download("u1"))
            getattr(g, stage)(1)
            getattr(o, stage)(1)
        for k in ("du1", "du2", "du3", "u1", "u2", "u3"):
            assert rel(g.download(k), o.download(k)) < 1e-11, (upload, k)
    g.close()


def test_contexts_with_other_group_sizes():
    """A kernel's shared-memory limit holds for every context that launches it: groups of eight rows
    (58 KB at 384 points) still run after a context of six (45 KB) is made."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    sets = []
    for which in ("seven", "single"):
        s = build_channel(tiny(ngal1=384, ngal2=54, ny=17, cyl_diameter=0.3, cyl_spacing=0.9, seed=3))
        s.ibu, s.ibv = points(np.random.default_rng(7), s, s.ibu, which), points(np.random.default_rng(8), s, s.ibv, which)
        sets.append(s)

    def substep(ch):
        ch.upload_state()
        ch.rk_substep(1)
        return ch.download("u1")

    a = Channel(sets[0])
    before = substep(a)
    b = Channel(sets[1])
    substep(b)
    np.testing.assert_array_equal(substep(a), before)


@pytest.mark.parametrize("change", ["none", "weight", "stencil", "missing"])
def test_repeated_planes(change):
    """Planes that list the same points share them on the device; one point that differs on a plane in
    the middle ends that.  Against the oracle to 1e-11, as above."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cfd_b200.channel import Channel, build_channel
    from cfd_b200.config import tiny
    from oracle.oracle import OracleChannel
    s = build_channel(tiny(ngal1=48, ngal2=54, ny=17, cyl_diameter=0.3, cyl_spacing=0.9, seed=3))
    lists = []
    for lst in (s.ibu, s.ibv):
        base = points(np.random.default_rng(5), s, lst, "pair")
        one = base.idx[:, 2] == base.idx[0, 2]
        idx, w = [], []
        planes = np.unique(lst.idx[:, 2])
        for n, j in enumerate(planes):
            a, b = base.idx[one].copy(), base.w[one].copy()
            a[:, [2, 5, 8]] = j
            if n == len(planes) // 2:
                if change == "weight":
                    b[len(b) // 2, 1] += 0.5
                elif change == "stencil":
                    a[-1, 3] = a[-1, 3] % s.cfg.ngal1 + 1
                elif change == "missing":
                    a, b = a[:-1], b[:-1]
            idx.append(a)
            w.append(b)
        lists.append(type(lst)(np.ascontiguousarray(np.concatenate(idx), dtype=np.int32),
                               np.ascontiguousarray(np.concatenate(w)), lst.jlo, lst.jhi))
    s.ibu, s.ibv = lists
    g, o = Channel(s), OracleChannel(s)
    g.upload_state()
    o.upload_state()
    for stage in ("rhs0", "nonlinear", "solve_uvw"):
        getattr(g, stage)(1)
        getattr(o, stage)(1)
    for k in ("du1", "du2", "du3", "u1", "u2", "u3"):
        assert rel(g.download(k), o.download(k)) < 1e-11, k
    g.close()
