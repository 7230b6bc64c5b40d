"""Performance cases of the channel-DNS hot path, called the way a user's program calls it.

A case is one pass through public entry points on a state that already lives on the GPU:

=========  ==============================================================================
kind       one pass
=========  ==============================================================================
step       ``Channel.step(steps)``: the main loop of a run, replayed as a CUDA graph
stages     one RK3 step through the per-stage entry points a Fortran driver binds
stats      a statistics call and the CFL query on the current state, and the sums read back
planes     the plane transforms: fill, to physical space, a product, back to modes
ensemble   ``Ensemble.step(steps)``: independent uneven channels advanced together
bands      ``Channel.step(steps)`` of a channel with three y-bands of x/z resolution
=========  ==============================================================================

FP32-mixed runs hand their fields over in single precision, the accuracy they carry; FP64
runs hand over the state itself.  ``exact`` restates the same passes in FP64 with torch.
"""
import ctypes as C
import math

import numpy as np
import torch

from cfd_b200.bands import long_columns
from cfd_b200.channel import Channel, build_channel, field_planes
from cfd_b200.config import ENSEMBLE_GROUPS, PRESETS, ChannelConfig, ensemble_configs
from cfd_b200.ensemble import Ensemble

DEV = "cuda:0"

# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------


def _preset(name, **kw):
    c = PRESETS[name]
    return dict(ng1=c.ngal1, ng2=c.ngal2, ny=c.ny, re_tau=c.re_tau, posth=c.posth, dia=c.cyl_diameter,
                spacing=c.cyl_spacing, **kw)


def _groups(groups):
    return ",".join("%dx%dx%dx%d" % (n, ng, ny, rt) for n, ng, ny, rt in groups)


def listed():
    return [
        # the smallest run: a parity-test channel, where launches and latency are all there is
        dict(name="step_tiny_fp64", kind="step", precision="fp64", steps=1, ng1=24, ng2=18, ny=17, re_tau=180.0,
             posth=0.12, dia=0.5, spacing=2.0),
        # the CPU-sized workload (Re_tau 180) in the reference's own precision
        dict(name="step_re180_fp64", kind="step", precision="fp64", steps=1, **_preset("re180")),
        # an ordinary channel at lengths that are no named workload's, without roughness
        dict(name="step_ragged_mixed", kind="step", precision="mixed", steps=1, ng1=144, ng2=108, ny=131, re_tau=300.0,
             posth=0.0, dia=0.0, spacing=0.0),
        # the FP64 workload compared field by field with the CPU run (Re_tau 395)
        dict(name="step_re395_fp64", kind="step", precision="fp64", steps=1, **_preset("re395")),
        # the headline workload (Re_tau 550) in FP64 and FP32-mixed
        dict(name="step_re550_fp64", kind="step", precision="fp64", steps=1, **_preset("re550")),
        dict(name="step_re550_mixed", kind="step", precision="mixed", steps=2, **_preset("re550")),
        # the largest channel (Re_tau 1000), FP32-mixed
        dict(name="step_re1000_mixed", kind="step", precision="mixed", steps=1, **_preset("re1000")),
        # a driver that keeps the reference's call sequence, stage by stage, at constant flow rate
        dict(name="stages_re395_fp64", kind="stages", precision="fp64", **_preset("re395")),
        # the statistics call of every nstat-th step with the canopy's conditional sums, and dtc_calc
        dict(name="stats_re550_mixed", kind="stats", precision="mixed", spectra=False, cond=True, **_preset("re550")),
        # the transform entry points on planes a driver fills itself
        dict(name="planes_192", kind="planes", precision="fp64", nplanes=193, ng1=192, ng2=192, ny=33, re_tau=180.0,
             posth=0.0, dia=0.0, spacing=0.0),
        # the batched ensemble of 16 uneven channels
        dict(name="ensemble_16_mixed", kind="ensemble", precision="mixed", steps=2, groups=_groups(ENSEMBLE_GROUPS)),
        # finer x/z resolution in the wall bands than in the middle, as the reference's input.in has it
        dict(name="bands_re180_fp64", kind="bands", precision="fp64", steps=1, ng1=128, ng2=128, ny=97, re_tau=180.0,
             posth=0.10, dia=0.05, spacing=0.20, ng1_mid=64, ng2_mid=64, band_vface=16),
    ]


# even lengths 2^a 3^b, the ones the transforms take, and those of three-band z planes
LENGTHS = [12, 16, 18, 24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384, 432, 486, 512,
           576, 648, 768]
TWO_STEP = [64, 96, 128, 192, 384]


def _near(rng, x, lengths=LENGTHS):
    """A length near x, one of the nearest three."""
    return rng.choice(sorted(lengths, key=lambda n: abs(math.log(n / x)))[:3])


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["stages", "stats", "stats", "planes", "planes", "ensemble", "bands"])
    precision = rng.choice(["fp64", "mixed"])
    # points of the channel, over the logarithm of the range
    pts = math.exp(rng.uniform(math.log(8e3), math.log(6e7 if kind == "step" else 2e7)))
    ny = max(9, int((pts * rng.uniform(0.2, 1.0)) ** (1 / 3)) + rng.randrange(0, 8))
    side = math.sqrt(pts / ny)
    asp = rng.uniform(0.7, 1.4)
    ng1, ng2 = _near(rng, side * asp), _near(rng, side / asp)
    rough = rng.random() < 0.7
    dia = rng.choice([0.03, 0.04, 0.05, 0.06]) if rough else 0.0
    c = dict(kind=kind, precision=precision, ng1=ng1, ng2=ng2, ny=ny, re_tau=float(rng.choice([180, 300, 395, 550])),
             posth=rng.choice([0.04, 0.06, 0.08]) if rough else 0.0, dia=dia, spacing=4.0 * dia)
    if kind in ("step", "bands"):
        c["steps"] = rng.choice([1, 1, 2])
    if kind == "stats":
        c["spectra"] = pts < 1e6 and rng.random() < 0.5
        c["cond"] = rough
    if kind == "planes":
        c.update(precision="fp64", ny=33, posth=0.0, dia=0.0, spacing=0.0, nplanes=max(1, int(pts / (ng1 * ng2))))
    if kind == "bands":
        z = _near(rng, min(side / asp, 192), TWO_STEP[1:4])
        c["ng2"], c["ng2_mid"] = z, rng.choice([n for n in TWO_STEP if n < z])
        c["ng1"] = min(c["ng1"], 256)
        c["ng1_mid"] = rng.choice([n for n in LENGTHS if c["ng1"] / 3 <= n <= c["ng1"]])
        c["ny"] = min(max(ny, 29), 129)
        c["band_vface"] = max(4, c["ny"] // 6)
    if kind == "ensemble":
        n = rng.randrange(2, 7)
        sizes = [rng.choice([24, 36, 48, 64, 72, 96, 128]) for _ in range(n)]
        c = dict(kind=kind, precision=precision, steps=rng.choice([1, 2]),
                 groups=_groups([(1, g, g + 1 + rng.randrange(0, 12), 180) for g in sizes]))
    return c


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------


def _config(case):
    kw = {}
    if case["kind"] == "bands":
        kw = dict(ngal1_mid=case["ng1_mid"], ngal2_mid=case["ng2_mid"], band_vface=case["band_vface"])
    if case["kind"] == "stages":
        kw = dict(flag_ctpress=0, qxt=2.0)
    return ChannelConfig(ngal1=case["ng1"], ngal2=case["ng2"], ny=case["ny"], re_tau=case["re_tau"], posth=case["posth"],
                         cyl_diameter=case["dia"], cyl_spacing=case["spacing"], precision=case["precision"],
                         dyq=10.0 if case["ny"] > 48 else 3.0, **kw)


_SETUPS = {}


def _setup_of(cfg):
    """Grid, point lists and time step of a configuration (host set-up, once per grid)."""
    key = repr(cfg)
    if key not in _SETUPS:
        s = build_channel(cfg, with_fields=False)
        # a fixed step well inside the advective and viscous limits of a developed flow
        kx, kz = cfg.alp * cfg.n1 / 2, cfg.bet * cfg.n2 / 2
        dy = float(np.diff(s.grid.yv).min())
        s.dt = min(0.15 / (2.0 * kx), 0.15 / (0.5 * kz), 2.0 * cfg.re_b / (kx * kx + kz * kz + 4.0 / dy ** 2), 0.02)
        while len(_SETUPS) >= 32:
            _SETUPS.pop(next(iter(_SETUPS)))
        _SETUPS[key] = s
    return _SETUPS[key]


def _weights(g):
    """Ghost-point weights (gridweighting, gridweighting_interp) of the two walls."""
    yu, yv = g.yu, g.yv
    return (-(yv[0] - yu[0]) / (yv[0] - yu[1]), (yu[-1] - yv[-1]) / (yv[-1] - yu[-2]),
            (yu[0] - yu[1]) / (yv[0] - yu[1]), (yu[-1] - yu[-2]) / (yv[-1] - yu[-2]))


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=DEV)


def _waves(cfg):
    i = torch.arange(cfg.nkx, device=DEV)
    q = torch.arange(cfg.n2, device=DEV)
    qs = torch.where(q < cfg.n2 // 2, q, q - cfg.n2)
    kx = (cfg.alp * i.double()).repeat(cfg.n2)
    kz = (cfg.bet * qs.double()).repeat_interleave(cfg.nkx)
    return kx, kz


def _fields(setup, seed):
    """A parabolic mean flow over the whole depth, the canopies included, with a broadband,
    discretely divergence-free perturbation of 10 % rms: random v and wall-normal vorticity
    with a decaying spectrum, u and w from them."""
    cfg, g = setup.cfg, setup.grid
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    nkx, n2, ncol = cfg.nkx, cfg.n2, cfg.ncol
    kx, kz = _waves(cfg)
    k2 = kx * kx + kz * kz
    shape = (1.0 + ((kx / cfg.alp) ** 2 + (kz / cfg.bet) ** 2) / 16.0) ** -1.2
    if cfg.band_vface > 0:
        shape = shape * _t(long_columns(cfg).astype(np.float64))

    def amp():
        a = torch.randn(3, n2, nkx, 2, generator=gen, device=DEV, dtype=torch.float64)
        a = torch.view_as_complex(a)
        a[:, n2 // 2] = 0  # the kz = -N2/2 row
        h = a[:, 1:n2 // 2, 0]
        a[:, n2 // 2 + 1:, 0] = torch.flip(h, (1,)).conj()  # a real field's kx = 0 column
        return a.reshape(3, ncol) * shape

    top = float(g.yv[-1])

    def profile(a, y):
        y = y / top
        env = torch.clamp(1 - y * y, min=0.0)
        b = torch.stack([torch.ones_like(y), y, torch.cos(3 * math.pi * y)]) * env ** 2
        return b.t().to(a.dtype) @ a

    yu, yv = _t(g.yu), _t(g.yv)
    v = profile(amp(), yv)
    eta = profile(amp(), yu)
    v[:, 0] = 0
    eta[:, 0] = 0
    ik2 = torch.where(k2 > 0, 1.0 / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))
    dv = torch.zeros_like(eta)
    dv[1:-1] = _t(g.dthdyu)[1:-1, None] * (v[1:] - v[:-1])
    u = 1j * kx * ik2 * dv - 1j * kz * eta * torch.sqrt(ik2)
    w = 1j * kz * ik2 * dv + 1j * kx * eta * torch.sqrt(ik2)
    del dv, eta
    fac = torch.where(kx > 0, 2.0, 1.0)
    e = sum((torch.view_as_real(f).square().sum(-1) * fac).sum() / f.shape[0] for f in (u, v, w))
    s = cfg.perturbation / torch.sqrt(e / 3.0)
    u *= s
    v *= s
    w *= s
    u[:, 0] = (1.5 * torch.clamp(1 - (yu / top) ** 2, min=0.0)).to(u.dtype)
    gwb, gwt = _weights(g)[:2]
    for f in (u, w):
        f[0] = -gwb * f[1]
        f[-1] = -gwt * f[-2]
    return u, v, w


class _Memory:
    """A field of a channel on the device, [plane][column], as torch sees it."""

    def __init__(self, ch, name):
        self.owner = ch
        self.__cuda_array_interface__ = {"shape": (field_planes(ch.setup, name), ch.cfg.ncol), "typestr": "<c16",
                                         "data": (ch.device_ptr(name), False), "version": 3}


def _view(ch, name):
    t = torch.as_tensor(_Memory(ch, name), device=DEV)
    t.owner = ch  # the channel's memory lives as long as a tensor on it does
    return t


def _mean_modes(setup, seed, v, w):
    """For the statistics alone: a pressure, and mean modes of v and w, so that every sum is a
    sum of something."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) + 1)
    cfg, g = setup.cfg, setup.grid
    kx, kz = _waves(cfg)
    shape = (1.0 + ((kx / cfg.alp) ** 2 + (kz / cfg.bet) ** 2) / 16.0) ** -1.2
    a = torch.view_as_complex(torch.randn(2, cfg.ncol, 2, generator=gen, device=DEV, dtype=torch.float64)) * shape * 0.01
    y = _t(g.yu)[1:-1].to(a.dtype)[:, None]
    p = a[0] + a[1] * y
    p[:, 0] = 0.02 + 0.01 * _t(g.yu)[1:-1] ** 2
    v[:, 0] = 0.01 * (1 + _t(g.yv))
    w[:, 0] = 0.03 * (2 + _t(g.yu))
    return p


def _channel(cfg, seed, stats=False):
    setup = _setup_of(cfg)
    ch = Channel(setup)
    f = {n: _view(ch, n) for n in ("u1", "u2", "u3", "p")}
    u, v, w = _fields(setup, seed)
    f["p"].zero_()
    if stats:
        f["p"].copy_(_mean_modes(setup, seed, v, w))
    for n, x in (("u1", u), ("u2", v), ("u3", w)):
        f[n].copy_(x)
    torch.cuda.synchronize()
    return ch, f


def _planes(case, seed):
    """Spectral planes in the reference's layout xPL(Ngal1+2, Ngal2), retained modes filled."""
    cfg = _config(case)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    x = torch.zeros(case["nplanes"], cfg.ngal2, cfg.ngal1 // 2 + 1, 2, dtype=torch.float64, device=DEV)
    h = cfg.n2 // 2
    for rows in (slice(0, h), slice(cfg.ngal2 - h, cfg.ngal2)):
        x[:, rows, :cfg.nkx] = torch.randn(case["nplanes"], h, cfg.nkx, 2, generator=gen, device=DEV, dtype=torch.float64)
    x[:, :, 1:] /= torch.arange(1, x.shape[2], device=DEV, dtype=torch.float64)[:, None]
    x[:, :, 0, 1] = 0
    return x.reshape(case["nplanes"], cfg.ngal2, cfg.ngal1 + 2)


def _members(case):
    groups = tuple(tuple(float(v) if k == 3 else int(v) for k, v in enumerate(g.split("x")))
                   for g in case["groups"].split(","))
    return ensemble_configs(precision=case["precision"], groups=groups)


def _tile(setup):
    """The lattice tile of the conditional sums and the last v plane of the bottom canopy."""
    from cfd_b200.geometry import lattice_params
    _, _, dnx, dnz = lattice_params(setup.cfg)[:4]
    return 0, dnx, dnz


def prepare(case, seed):
    kind = case["kind"]
    stream = torch.cuda.Stream(DEV)
    if kind == "ensemble":
        pairs = [_channel(cfg, seed + 1000 * k) for k, cfg in enumerate(_members(case))]
        ens = Ensemble([ch for ch, _ in pairs])
        return dict(case=case, ens=ens, stream=torch.cuda.ExternalStream(ens.stream(), device=DEV), members=pairs)
    if kind == "planes":
        setup = _setup_of(_config(case))
        ch = Channel(setup)
        ch.set_stream(stream.cuda_stream)
        spec = _planes(case, seed)
        torch.cuda.synchronize()
        return dict(case=case, ch=ch, stream=stream, spec=spec, buf=torch.empty_like(spec), prod=torch.empty_like(spec))
    ch, f = _channel(_config(case), seed, kind == "stats")
    ch.set_stream(stream.cuda_stream)
    if kind == "stages":
        f["psi"] = _view(ch, "psi")
    if kind == "stats":
        if case["cond"]:
            ch.stats_configure(*_tile(ch.setup), spectra=case["spectra"])
        else:
            ch.stats_configure(-10 ** 6, 1, 1, spectra=case["spectra"])
    return dict(case=case, ch=ch, stream=stream, f=f)


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------


def _hand_over(case, f):
    if case["precision"] == "mixed":
        return {n: x.to(torch.complex64) for n, x in f.items()}
    return dict(f)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "bands"):
        state["ch"].step(case["steps"])
        with torch.cuda.stream(state["stream"]):
            return _hand_over(case, state["f"])
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        with torch.cuda.stream(state["stream"]):
            return [_hand_over(case, f) for _, f in state["members"]]
    ch = state["ch"]
    if kind == "stages":
        for krk in (1, 2, 3):
            ch.rhs0(krk)
            ch.nonlinear(krk)
            ch.solve_uvw(krk)
            ch.meanflow(krk)
            ch.solve_p(krk)
            ch.vcorr(krk)
        with torch.cuda.stream(state["stream"]):
            return _hand_over(case, state["f"])
    if kind == "stats":
        ch.stats_reset()
        ch.stats_accumulate()
        out = ch.stats_read()
        if case["spectra"]:
            out.update(ch.spectra_read())
        out["dtc"], out["terms"] = ch.cfl()
        return out
    with torch.cuda.stream(state["stream"]):
        buf, prod, n = state["buf"], state["prod"], case["nplanes"]
        buf.copy_(state["spec"])
        ch._chk(ch.lib.cfd_four_to_phys(ch.ctx, C.c_void_p(buf.data_ptr()), n, 1), "four_to_phys")
        torch.mul(buf, buf, out=prod)
        ch._chk(ch.lib.cfd_phys_to_four(ch.ctx, C.c_void_p(prod.data_ptr()), n), "phys_to_four")
        return {"phys": buf, "product": prod}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------


def _fft_flops(n, lines):
    return 5.0 * n * math.log2(n) * lines


def _step_work(cfg, steps):
    """State and advective history read and written once per RK substep; the transforms of
    3 fields and 6 products on every plane, and some 160 operations per mode and plane."""
    setup = _setup_of(cfg)
    g = setup.grid
    hist = 8 if cfg.precision == "mixed" else 16
    pl = 2 * g.nyu + g.nyv
    by = 3 * cfg.ncol * 2 * ((pl + g.nyp) * 16 + pl * hist)
    lines = pl + 4 * g.nyu + 2 * g.nyv
    fl = 3 * lines * (_fft_flops(cfg.ngal2, cfg.nkx) + 0.5 * _fft_flops(cfg.ngal1, cfg.ngal2)) + 3 * 160.0 * cfg.ncol * g.nyu
    return steps * by, steps * fl


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        w = [_step_work(cfg, case["steps"]) for cfg in _members(case)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    cfg = _config(case)
    if kind in ("step", "bands", "stages"):
        by, fl = _step_work(cfg, case.get("steps", 1))
        return {"bytes": by, "flops": fl}
    if kind == "stats":
        g = _setup_of(cfg).grid
        pl = 2 * g.nyu + g.nyv + g.nyp
        lines = 3 * g.nyu + 3 * g.nyv + g.nyp
        return {"bytes": 2 * 16 * cfg.ncol * pl,
                "flops": lines * (_fft_flops(cfg.ngal2, cfg.nkx) + 0.5 * _fft_flops(cfg.ngal1, cfg.ngal2))}
    n = case["nplanes"]
    return {"bytes": 8 * n * cfg.ngal2 * (cfg.ngal1 + 2) * 6,
            "flops": 2 * n * (_fft_flops(cfg.ngal2, cfg.nkx) + 0.5 * _fft_flops(cfg.ngal1, cfg.ngal2))}


# ------------------------------------------------------------------------------------------
# the same passes in FP64, plainly
# ------------------------------------------------------------------------------------------

RKA = (4 / 15, 1 / 15, 1 / 6)
RKG = (8 / 15, 5 / 12, 3 / 4)
RKC = (0.0, -17 / 60, -5 / 12)
RKD = (8 / 15, 2 / 15, 1 / 3)


class _Plain:
    """One RK3 step of the channel on [plane][column] arrays."""

    def __init__(self, setup, u, v, w):
        self.s, self.cfg, self.g = setup, setup.cfg, setup.grid
        cfg, g = self.cfg, self.g
        self.u1, self.u2, self.u3 = u, v, w
        z = lambda n: torch.zeros(n, cfg.ncol, dtype=torch.complex128, device=DEV)  # noqa: E731
        self.p, self.psi, self.div = z(g.nyp), z(g.nyp), z(g.nyp)
        self.nu = [z(g.nyu), z(g.nyv), z(g.nyu)]
        self.kx, self.kz = _waves(cfg)
        self.k2 = -(self.kx ** 2) - (self.kz ** 2)
        self.gwb, self.gwt, self.gwib, self.gwit = _weights(g)
        self.du, self.dv = _t(g.dthdyu)[:, None], _t(g.dthdyv)[:, None]
        self.cu, self.cv = _t(g.dyu2i), _t(g.dyv2i)
        yu, yv = _t(g.yu), _t(g.yv)
        self.fa = ((yv - yu[:-1]) / (yu[1:] - yu[:-1]))[:, None]
        self.fb = ((yu[1:] - yv) / (yu[1:] - yu[:-1]))[:, None]
        self.ca = ((yu[1:-1] - yv[:-1]) / (yv[1:] - yv[:-1]))[:, None]
        self.cb = ((yv[1:] - yu[1:-1]) / (yv[1:] - yv[:-1]))[:, None]
        self.dyv = yv[1:] - yv[:-1]
        self.mpgx = cfg.mpgx
        self.ib = [self._points(setup.ibu, g.ju0, g.nyu), self._points(setup.ibv, g.jv0, g.nyv)]
        self.chunk = max(1, int(2e7 / (cfg.ngal1 * cfg.ngal2)))

    def phys(self, f):
        cfg = self.cfg
        h, n = cfg.n2 // 2, f.shape[0]
        full = torch.zeros(n, cfg.ngal2, cfg.ngal1 // 2 + 1, dtype=torch.complex128, device=DEV)
        f = f.reshape(n, cfg.n2, cfg.nkx)
        full[:, :h, :cfg.nkx] = f[:, :h]
        full[:, cfg.ngal2 - h:, :cfg.nkx] = f[:, h:]
        zc = torch.fft.ifft(full, dim=1) * cfg.ngal2
        zc[:, :, 0] = zc[:, :, 0].real.to(zc.dtype)  # the real transform ignores Im of kx = 0
        return torch.fft.irfft(zc, n=cfg.ngal1, dim=2) * cfg.ngal1

    def spec(self, x):
        cfg = self.cfg
        h = cfg.n2 // 2
        r = torch.fft.rfft(x, dim=2)[:, :, :cfg.nkx] / cfg.ngal1
        z = torch.fft.fft(r, dim=1) / cfg.ngal2
        return torch.cat([z[:, :h], z[:, cfg.ngal2 - h:]], 1).reshape(x.shape[0], cfg.ncol)

    def _points(self, lst, j0, n):
        planes = []
        for s in range(2):
            for j in range(max(lst.jlo[s], j0 + 1), min(lst.jhi[s], j0 + n - 2) + 1):
                if j not in planes:
                    planes.append(j)
        if not planes:
            return None
        slot = np.zeros(n, np.int64)
        slot[np.array(planes) - j0] = np.arange(len(planes))
        idx = lst.idx.astype(np.int64)
        flat = lambda k: (slot[idx[:, k + 2] - j0] * self.cfg.ngal2 + idx[:, k + 1] - 1) * self.cfg.ngal1 + idx[:, k] - 1  # noqa: E731
        t = flat(0)
        # the points of a run of equal targets apply one after another, in list order
        start = np.r_[True, t[1:] != t[:-1]] if lst.n else np.zeros(0, bool)
        turn = np.arange(lst.n) - np.maximum.accumulate(np.where(start, np.arange(lst.n), 0)) if lst.n else np.zeros(0, int)
        rounds = [np.nonzero(turn == k)[0] for k in range(int(turn.max()) + 1 if lst.n else 0)]
        f2, f3 = flat(3), flat(6)
        return ([j - j0 for j in planes],
                [(_t(t[r]), _t(f2[r]), _t(f3[r]), _t(lst.w[r])) for r in rounds])

    def _force(self, u, r, ib):
        if ib is None:
            return
        planes, rounds = ib
        U, R = self.phys(u[planes]), self.phys(r[planes])
        shape = R.shape
        U, R = U.reshape(-1), R.reshape(-1)
        for t, f2, f3, w in rounds:
            R[t] = w[:, 0] * (w[:, 1] * U[f2] + w[:, 2] * U[f3] - U[t] + R[t])
        r[planes] = self.spec(R.reshape(shape))

    @staticmethod
    def _thomas(a1, a2, a3, r):
        """LU and substitution over all columns; a*: one row of coefficients per plane."""
        n = r.shape[0]
        x, cs = r.clone(), []
        d = 1.0 / a2(0)
        x[0] *= d
        for j in range(1, n):
            c = a3(j - 1) * d
            cs.append(c)
            d = 1.0 / (a2(j) - a1(j) * c)
            x[j] = (x[j] - a1(j) * x[j - 1]) * d
        for j in range(n - 2, -1, -1):
            x[j] -= cs[j] * x[j + 1]
        return x

    def vcentre(self):
        v = torch.empty(self.g.nyu, self.cfg.ncol, dtype=torch.complex128, device=DEV)
        v[1:-1] = self.ca * self.u2[1:] + self.cb * self.u2[:-1]
        v[0] = self.gwib * (self.u2[0] - v[1]) + v[1]
        v[-1] = self.gwit * (self.u2[-1] - v[-2]) + v[-2]
        return v

    def nonlinear(self):
        g, cfg = self.g, self.cfg
        zr = slice(cfg.n2 // 2 * cfg.nkx, (cfg.n2 // 2 + 1) * cfg.nkx)
        ikx, ikz = 1j * self.kx, 1j * self.kz
        vc = self.vcentre()
        vv = torch.empty_like(vc)
        nu1, nu3 = torch.empty_like(vc), torch.empty_like(vc)
        for a in range(0, g.nyu, self.chunk):
            b = min(a + self.chunk, g.nyu)
            U, V, W = self.phys(self.u1[a:b]), self.phys(vc[a:b]), self.phys(self.u3[a:b])
            uu, uw, ww = self.spec(U * U), self.spec(U * W), self.spec(W * W)
            vv[a:b] = self.spec(V * V)
            nu1[a:b] = ikx * uu + ikz * uw
            nu3[a:b] = ikx * uw + ikz * ww
        uv, vw = torch.empty_like(self.u2), torch.empty_like(self.u2)
        for a in range(0, g.nyv, self.chunk):
            b = min(a + self.chunk, g.nyv)
            f = lambda s: self.fa[a:b] * s[a + 1:b + 1] + self.fb[a:b] * s[a:b]  # noqa: E731
            U, V, W = self.phys(f(self.u1)), self.phys(self.u2[a:b]), self.phys(f(self.u3))
            uv[a:b], vw[a:b] = self.spec(U * V), self.spec(W * V)
        nu2 = ikx * uv + ikz * vw
        for x in (nu1, nu2, nu3):
            x[:, zr] = 0
        nu1[1:-1] += self.du[1:-1] * (uv[1:] - uv[:-1])
        nu3[1:-1] += self.du[1:-1] * (vw[1:] - vw[:-1])
        nu2[1:-1] += self.dv[1:-1] * (vv[2:-1] - vv[1:-2])
        return [nu1, nu2, nu3]

    def substep(self, k):
        g, s = self.g, self.s
        dt, re = s.dt, self.cfg.re_b
        beta, c = RKA[k] * dt / re, self.cu
        new = self.nonlinear()
        lap = lambda u, c: c[1:-1, 0:1] * u[:-2] + (self.k2 + c[1:-1, 1:2]) * u[1:-1] + c[1:-1, 2:3] * u[2:]  # noqa: E731
        grad = [1j * self.kx * self.p, self.dv[1:-1] * (self.p[1:] - self.p[:-1]), 1j * self.kz * self.p]
        rhs = []
        for f, (u, c) in enumerate(((self.u1, self.cu), (self.u2, self.cv), (self.u3, self.cu))):
            r = RKA[k] / re * lap(u, c) - RKC[k] * self.nu[f][1:-1] - RKD[k] * grad[f]
            if f == 0:
                r[:, 0] -= RKD[k] * self.mpgx
            r = u[1:-1] + dt * (r - RKG[k] * new[f][1:-1])
            full = torch.zeros_like(u)
            full[1:-1] = r
            rhs.append(full)
        self.nu = new
        del grad, r, full
        for f, (u, ib) in enumerate(((self.u1, self.ib[0]), (self.u2, self.ib[1]), (self.u3, self.ib[0]))):
            self._force(u, rhs[f], ib)
        for f, (c, e0, e1) in enumerate(((self.cu, self.gwb, self.gwt), (self.cv, 0.0, 0.0), (self.cu, self.gwb, self.gwt))):
            n = rhs[f].shape[0]
            a1 = lambda j: e1 if j == n - 1 else -beta * c[j, 0]  # noqa: E731
            a2 = lambda j: torch.ones_like(self.kx) if j in (0, n - 1) else 1 - beta * (c[j, 1] + self.k2)  # noqa: E731
            a3 = lambda j: e0 if j == 0 else -beta * c[j, 2]  # noqa: E731
            rhs[f] = self._thomas(a1, a2, a3, rhs[f])
        self.u1, self.u2, self.u3 = rhs
        if self.cfg.flag_ctpress == 0:
            self.meanflow(k)
        self.divergence()
        dtab = dt * 2 * RKA[k]
        r = self.div / dtab
        r[0, 0] = 0
        n = g.nyp
        du, dvm, dvp = self.du[1:-1, 0], self.dv[:-1, 0], self.dv[1:, 0]
        first = torch.zeros_like(self.kx)
        first[0] = 1

        def a2(j):
            lo, hi = (du[j] * dvm[j] if j > 0 else 0.0), (du[j] * dvp[j] if j < n - 1 else 0.0)
            a = self.k2 - lo - hi
            return torch.where(first > 0, 1.0 / (self.g.u(2) - self.g.u(1)) ** 2, a) if j == 0 else a
        self.psi = self._thomas(lambda j: du[j] * dvm[j], a2, lambda j: du[j] * dvp[j] * (1 - first if j == 0 else 1), r)
        self.p = self.p + self.psi
        self.u1[1:-1] -= dtab * 1j * self.kx * self.psi
        self.u3[1:-1] -= dtab * 1j * self.kz * self.psi
        self.u2[1:-1] -= dtab * self.dv[1:-1] * (self.psi[1:] - self.psi[:-1])
        for u in (self.u1, self.u3):
            u[0] = -self.gwb * u[1]
            u[-1] = -self.gwt * u[-2]
        self.u2[0] = 0
        self.u2[-1] = 0

    def divergence(self):
        self.div = 1j * self.kx * self.u1[1:-1] + 1j * self.kz * self.u3[1:-1] + self.du[1:-1] * (self.u2[1:] - self.u2[:-1])

    def meanflow(self, k):
        g, dt = self.g, self.s.dt
        d, nn = g.dny, g.ny - 2
        beta, n = RKA[k] * dt / self.cfg.re_b, g.ny + 1
        c = g.dyu2i
        a1 = lambda j: self.gwt if j == n - 1 else -beta * c[j + d, 0]  # noqa: E731
        a2 = lambda j: torch.ones(1, device=DEV, dtype=torch.float64) if j in (0, n - 1) else \
            torch.full((1,), 1 - beta * c[j + d, 1], device=DEV, dtype=torch.float64)  # noqa: E731
        a3 = lambda j: self.gwb if j == 0 else -beta * c[j + d, 2]  # noqa: E731
        r = torch.full((n, 1), -RKD[k] * dt, dtype=torch.float64, device=DEV)
        r[0] = r[-1] = 0
        x = self._thomas(a1, a2, a3, r)[:, 0]
        h = self.dyv[d:d + nn + 1]
        q = lambda y: (h * y).sum()  # noqa: E731
        gg = (self.cfg.qxt - q(self.u1[d + 1:d + nn + 2, 0].real)) / q(x[1:nn + 2])
        self.mpgx += float(gg)
        self.u1[d:d + n, 0] += gg * x

    def step(self):
        for k in range(3):
            self.substep(k)

    def state(self):
        return {"u1": self.u1, "u2": self.u2, "u3": self.u3, "p": self.p}

    def stats(self, jband, dnx, dnz):
        """stats() on zeroed sums, the conditional sums folded onto one tile, and dtc_calc."""
        g, cfg = self.g, self.cfg
        cond = jband >= g.jv0
        nb = (jband + 2 - g.ju0, jband + 1 - g.jv0, jband + 1 - g.jp0) if cond else (0, 0, 0)
        if not cond:
            dnx = dnz = 0
        dz = 1j * self.kz * self.u2
        dz[:, cfg.n2 // 2 * cfg.nkx:(cfg.n2 // 2 + 1) * cfg.nkx] = 0
        wi = self.fa * self.u3[1:] + self.fb * self.u3[:-1]
        wx = self.dv * (self.u3[1:] - self.u3[:-1]) - dz
        out, top = {"istat": 1}, []
        vc = self.vcentre()
        for names, fields, k in ((("Um", "U2m", "Wm", "W2m", "UVm", "UWm"), (self.u1, self.u3, vc), 0),
                                 (("Vm", "V2m", "wxm", "wx2m", "VWm"), (self.u2, wi, wx), 1), (("Pm", "P2m"), (self.p,), 2)):
            ny = fields[0].shape[0]
            sums = torch.zeros(len(names), ny, dtype=torch.float64, device=DEV)
            fold = torch.zeros(len(names), nb[k], dnz, dnx, dtype=torch.float64, device=DEV)
            big = [0.0, 0.0]
            for a in range(ny):
                x = [self.phys(f[a:a + 1])[0] for f in fields]
                for side, j1 in ((1.0, a), (-1.0, ny - 1 - a)):
                    if side < 0 and j1 >= nb[k]:
                        continue
                    if k == 0:
                        q = (x[0], x[0] * x[0], x[1], x[1] * x[1], x[0] * x[2] * side, x[0] * x[1])
                    elif k == 1:
                        q = (x[0] * side, x[0] * x[0], x[2], x[2] * x[2], x[0] * side * x[1])
                    else:
                        q = (x[0], x[0] * x[0])
                    if side > 0:
                        for i, y in enumerate(q):
                            sums[i, a] = (y[:cfg.n2, :cfg.n1] if k == 1 and i in (2, 3) else y).sum()
                    if j1 < nb[k]:
                        for i, y in enumerate(q):
                            fold[i, j1] += y.reshape(cfg.ngal2 // dnz, dnz, cfg.ngal1 // dnx, dnx).sum((0, 2))
                if k == 0:
                    big = [max(b, float(y.abs().max())) for b, y in zip(big, x)]
                elif k == 1 and 0 < a < ny - 1:
                    big[0] = max(big[0], float(x[0].abs().max()) * g.dthdyv[a])
            for i, n in enumerate(names):
                out[n], out[n + "C"] = sums[i], fold[i]
            top += big
        t = [1 / (cfg.alp * (cfg.n1 // 2) * top[0]), 1 / (cfg.bet * (cfg.n2 // 2) * top[1]), 1 / max(1e-6, top[2])]
        out["dtc"], out["terms"] = min(t[0], t[1]), np.array(t)
        return out

    def spectra(self):
        sq = lambda f: torch.view_as_real(f).square().sum(-1).t()  # noqa: E731
        vc = self.vcentre()
        return {"spU": sq(self.u1), "spV": sq(self.u2), "spW": sq(self.u3),
                "spUV": (self.u1.real * vc.real + self.u1.imag * vc.imag).t(), "spP": sq(self.p)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "bands":
        return None
    if kind == "ensemble":
        out = []
        for k, cfg in enumerate(_members(case)):
            setup = _setup_of(cfg)
            c = _Plain(setup, *_fields(setup, seed + 1000 * k))
            for _ in range(case["steps"]):
                c.step()
            out.append(c.state())
        return out
    if kind == "planes":
        cfg = _config(case)
        x = torch.view_as_complex(_planes(case, seed).reshape(case["nplanes"], cfg.ngal2, cfg.ngal1 // 2 + 1, 2))
        # the z transform covers the modes 0..N1/2 of a plane; the others are zero here
        z = torch.fft.ifft(x, dim=1) * cfg.ngal2
        z[:, :, 0] = z[:, :, 0].real.to(z.dtype)
        phys = torch.nn.functional.pad(torch.fft.irfft(z, n=cfg.ngal1, dim=2) * cfg.ngal1, (0, 2))
        r = torch.fft.rfft(phys[:, :, :cfg.ngal1] ** 2, dim=2) / cfg.ngal1
        r[:, :, :cfg.nkx] = torch.fft.fft(r[:, :, :cfg.nkx], dim=1) / cfg.ngal2
        return {"phys": phys, "product": torch.view_as_real(r).reshape(phys.shape)}
    setup = _setup_of(_config(case))
    u, v, w = _fields(setup, seed)
    p = _mean_modes(setup, seed, v, w) if kind == "stats" else None
    c = _Plain(setup, u, v, w)
    if kind == "stats":
        c.p = p
        out = c.stats(*(_tile(setup) if case["cond"] else (-10 ** 6, 1, 1)))
        if case["spectra"]:
            out.update(c.spectra())
        return out
    for _ in range(case.get("steps", 1)):
        c.step()
    out = c.state()
    if kind == "stages":
        out["psi"] = c.psi
    return out
