"""Performance cases of the large step and its routines on one GPU.

A case is a dict of plain values.  Its "kind" names the public entry point that
is called: a whole large step (Context.step with graph replay, or an ensemble
step), one routine of the step as a host program calls it (advs, advuvw, sound),
one of solve1's tendencies (diff2, turbsmag), the statistics package, or one
training step of the learned closure.  States live on the GPU, as in a program
that keeps its model there.  All inputs are made from the seed: soundings and
grids of cm1_b200.cases, smooth velocity, pressure and scalar perturbations of a
few wavelengths with both signs, and small-scale noise on theta.
"""
import ctypes as C
import functools
import math
import random

import numpy as np
import torch

from cm1_b200 import binding
from cm1_b200.abi import Config
from cm1_b200.cases import ENSEMBLE_SIZES, WORKLOADS, Layout, make_case, stat_opts
from cm1_b200.learned import N_PARAMS, init_params

DEV = "cuda"
P00, RD, CP, RV = 1.0e5, 287.04, 1005.7, 461.5


def listed():
    return [
        # the smallest whole step in use: a dry warm bubble, 5th-order advection;
        # launches and latency count here
        dict(name="step_bubble_64", kind="step", workload="dry_bubble", ni=64, nj=64, nk=40, bc=1, npt=0, weno=0, nsound=6),
        # the repository's benchmark configuration: moist, open-radiative, five tracers
        dict(name="step_supercell_256", kind="step", workload="supercell", ni=256, nj=256, nk=80, bc=2, npt=5, weno=1, nsound=8),
        # a large-eddy domain, dry and periodic with two tracers: the largest single step
        dict(name="step_cbl_512", kind="step", workload="cbl", ni=512, nj=512, nk=128, bc=1, npt=2, weno=1, nsound=6),
        # warm-rain microphysics on an odd-sized domain
        dict(name="step_kessler_odd", kind="step", workload="kessler", ni=203, nj=150, nk=61, bc=2, npt=0, weno=1, nsound=8),
        # an uneven ensemble of small domains advanced together
        dict(name="ensemble_12", kind="ensemble", members=12, sizes=7, weno=1),
        # one positive-definite scalar through the drop-in advection routine
        dict(name="advs_pdef_odd", kind="advs", ni=251, nj=187, nk=79, bc=2, weno=1, pdef=1, pdefweno=1),
        # the three momentum tendencies through the drop-in routine
        dict(name="advuvw_256", kind="advuvw", ni=256, nj=256, nk=80, bc=1),
        # the acoustic substeps of the final stage through the drop-in routine
        dict(name="sound_384x250", kind="sound", ni=384, nj=250, nk=64, bc=1, nsound=6),
        # subgrid turbulence tendencies of a large-eddy simulation
        dict(name="turbsmag_256", kind="turbsmag", ni=256, nj=256, nk=128, npt=2, tconfig=2, bcturbs=1, bbc=1, tbc=1),
        # fixed-viscosity diffusion of momentum, theta and three tracers
        dict(name="diff2_256", kind="diff2", ni=256, nj=256, nk=80, npt=3, bbc=1, tbc=1),
        # every statistic of a moist run
        dict(name="stats_256", kind="stats", ni=256, nj=256, nk=80, npt=5),
        # one optimiser step of the learned closure at its training batch size
        dict(name="train_65536", kind="train", n=65536, act="relu"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, most, nk_lo=24, nk_hi=128):
    """Horizontal extents and levels, spread over the logarithm, at most `most` cells."""
    while True:
        ni, nj, nk = _log(rng, 40, 700), _log(rng, 40, 700), _log(rng, nk_lo, nk_hi)
        if 6.0e4 <= ni * nj * nk <= most:
            return dict(ni=ni, nj=nj, nk=nk)


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["ensemble", "advs", "advuvw", "sound", "turbsmag", "diff2", "stats", "train"])
    if kind == "step":
        wl = rng.choice(["dry_bubble", "supercell", "cbl", "kessler"])
        npt = {"dry_bubble": 0, "supercell": rng.randint(0, 5), "cbl": rng.randint(0, 3), "kessler": rng.randint(0, 1)}[wl]
        return dict(kind=kind, workload=wl, bc=rng.choice([1, 2]) if wl != "cbl" else 1, npt=npt, weno=rng.choice([0, 1, 2]),
                    nsound=rng.choice([6, 8, 10]), **_grid(rng, 6.0e6 if wl in ("supercell", "kessler") else 2.0e7))
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(3, 14), sizes=rng.randint(0, 10 ** 6), weno=rng.choice([0, 1]))
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 2000, 400000), act=rng.choice(["relu", "gelu"]))
    g = _grid(rng, 1.0e7)
    if kind == "advs":
        return dict(kind=kind, bc=rng.choice([1, 2]), weno=rng.choice([0, 1]), pdef=rng.choice([0, 1]), pdefweno=rng.choice([0, 1]), **g)
    if kind == "advuvw":
        return dict(kind=kind, bc=rng.choice([1, 2]), **g)
    if kind == "sound":
        return dict(kind=kind, bc=rng.choice([1, 2]), nsound=rng.choice([6, 8, 10]), **g)
    if kind == "turbsmag":
        return dict(kind=kind, npt=rng.randint(0, 3), tconfig=rng.choice([1, 2]), bcturbs=rng.choice([1, 2]), bbc=rng.choice([1, 2]), tbc=rng.choice([1, 2]), **g)
    if kind == "diff2":
        return dict(kind=kind, npt=rng.randint(0, 4), bbc=rng.choice([1, 2]), tbc=rng.choice([1, 2]), **g)
    return dict(kind="stats", npt=rng.randint(0, 5), **g)


# ---------------------------------------------------------------- grids and states
@functools.lru_cache(maxsize=24)
def _columns(workload, nk, bc, npt, weno, nsound):
    """The configuration and the vertical profiles of a workload (from an 8 x 8 domain)."""
    return make_case(workload, ni=8, nj=8, nk=nk, bc=bc, npt=npt, advwenos=weno, nsound=nsound)


@functools.lru_cache(maxsize=3)
def _host_grid(workload, ni, nj, nk, bc, npt, weno, nsound):
    """(cfg, grid arrays, Layout) of a workload at ni x nj: cm1g_init's host arguments."""
    col = _columns(workload, nk, bc, npt, weno, nsound)
    lay = Layout(ni, nj, nk)
    cfg = Config.from_buffer_copy(bytes(col.cfg))
    cfg.ni, cfg.nj = ni, nj
    shape = {"mf": 4, "rmf": 4, "u0": 2, "v0": 3}
    grid = {}
    for n, a in col.grid.items():
        if a.ndim == 3:
            grid[n] = np.ascontiguousarray(np.broadcast_to(a[:, :1, :1], lay.shape(shape.get(n, 1))))
        elif a.ndim == 1:
            grid[n] = np.ones({"u": lay.NI, "v": lay.NJ}[n.lstrip("r")[0]] + (n[-1] == "f"), np.float32)
    op = bc != 1
    for n in ("dtu0", "dtv0"):
        grid[n] = np.zeros((lay.NJ, lay.NI), np.float32)
    grid["dtu0"][lay.jx(1):lay.jx(nj) + 1, lay.ix(1 + op):lay.ix(ni + 1 - op) + 1] = 1.0
    grid["dtv0"][lay.jx(1 + op):lay.jx(nj + 1 - op) + 1, lay.ix(1):lay.ix(ni) + 1] = 1.0
    return cfg, grid, lay


class _Maker:
    """Seeded fields of one grid on the GPU, halos filled."""

    def __init__(self, lay, bc, seed):
        self.lay, self.periodic = lay, bc == 1
        self.rng = random.Random(seed)
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(seed)

    def _points(self, stag):
        lay = self.lay
        op = not self.periodic
        return lay.ni + (op and stag == 2), lay.nj + (op and stag == 3), lay.nk + (stag == 4)

    def halo(self, a, stag):
        """The full array of a field given at its physical points: lateral halos by wrap
        or by copy of the edge, the levels below and above by copy (w: zero)."""
        lay = self.lay
        nz, ny, nx = lay.shape(stag)
        ix, iy = torch.arange(nx, device=DEV) - 3, torch.arange(ny, device=DEV) - 3
        ix = ix % a.shape[2] if self.periodic else ix.clamp(0, a.shape[2] - 1)
        iy = iy % a.shape[1] if self.periodic else iy.clamp(0, a.shape[1] - 1)
        out = torch.zeros((nz, ny, nx), device=DEV)
        out[1:1 + a.shape[0]] = a[:, iy][:, :, ix]
        if stag == 4:
            out[1] = 0.0
            out[lay.nk + 1] = 0.0
        else:
            out[0], out[lay.nk + 1] = out[1], out[lay.nk]
        return out

    def smooth(self, stag, amp, modes=4):
        """A sum of a few waves with both signs, zero at the bottom and top for w."""
        nx, ny, nz = self._points(stag)
        x = torch.arange(nx, device=DEV) / self.lay.ni
        y = torch.arange(ny, device=DEV) / self.lay.nj
        z = (torch.arange(nz, device=DEV) + (0.0 if stag == 4 else 0.5)) / self.lay.nk
        out = torch.zeros((nz, ny, nx), device=DEV)
        for _ in range(modes):
            r = self.rng
            fx = torch.sin(2 * math.pi * (r.randint(1, 4) * x + r.random()))
            fy = torch.sin(2 * math.pi * (r.randint(1, 4) * y + r.random()))
            fz = torch.sin(math.pi * r.randint(1, 3) * z) if stag == 4 else torch.cos(math.pi * r.randint(1, 3) * z)
            out += (amp * r.uniform(0.4, 1.0) / modes ** 0.5) * fz[:, None, None] * fy[None, :, None] * fx[None, None, :]
        return out

    def noise(self, stag, amp):
        nx, ny, nz = self._points(stag)
        return amp * (2.0 * torch.rand((nz, ny, nx), device=DEV, generator=self.gen) - 1.0)


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _state(case, seed, cfg, grid, lay):
    """The prognostic state of a workload in the middle of a run (t and t+dt arrays equal)."""
    mk = _Maker(lay, case["bc"], seed)
    nk = lay.nk
    col = lambda n: _t(grid[n][:, 0, 0])[:, None, None]          # noqa: E731
    wind = {"dry_bubble": 3.0, "supercell": 4.0, "kessler": 4.0, "cbl": 1.0}[case["workload"]]
    st = {}
    st["ua"] = col("u0") + mk.halo(mk.smooth(2, wind) + mk.noise(2, 0.05 * wind), 2)
    st["va"] = col("v0") + mk.halo(mk.smooth(3, wind) + mk.noise(3, 0.05 * wind), 3)
    st["wa"] = mk.halo(mk.smooth(4, 0.4 * wind), 4)
    st["tha"] = mk.halo(mk.smooth(1, 0.5) + mk.noise(1, 0.05), 1)
    st["ppi"] = mk.halo(mk.smooth(1, 2.0e-5), 1)
    if cfg.imoist:
        qv = col("qv0")[1:nk + 1] * (1.0 + mk.smooth(1, 0.05))
        q = [mk.halo(qv, 1)]
        for amp in (1.5e-3, 1.0e-3)[:cfg.numq - 1]:              # cloud and rain with clear air between
            q.append(mk.halo((mk.smooth(1, 2.0 * amp) - 0.5 * amp).clamp_min(0.0), 1))
        st["qa"] = torch.stack(q)
    else:
        st["qa"] = torch.zeros((0,) + lay.shape(1), device=DEV)
    npt = cfg.npt if cfg.iptra else 0
    pt = [mk.halo((mk.smooth(1, 2.0e-3) - 2.0e-4).clamp_min(0.0), 1) for _ in range(npt)]
    st["pta"] = torch.stack(pt) if pt else torch.zeros((0,) + lay.shape(1), device=DEV)
    for a, b in (("ua", "u3d"), ("va", "v3d"), ("wa", "w3d"), ("tha", "th3d"), ("ppi", "pp3d"), ("qa", "q3d"), ("pta", "pt3d")):
        st[b] = st[a].clone()
    st["ppx"] = st["ppi"].clone()
    for a, b in (("ua", "uten1"), ("va", "vten1"), ("wa", "wten1"), ("tha", "thten1"), ("ppi", "ppten"), ("qa", "qten"), ("pta", "ptten")):
        st[b] = torch.zeros_like(st[a])
    pi = (col("pi0") + st["pp3d"]).double()
    st["prs"] = (P00 * pi ** (CP / RD)).float()
    qv = st["q3d"][0].double().clamp_min(0.0) if cfg.imoist else 0.0
    st["rho"] = (st["prs"].double() / ((col("th0") + st["th3d"]).double() * pi * (RD + qv * RV))).float()
    for n in ("radbcw", "radbce"):
        st[n] = torch.zeros((lay.NK, lay.NJ), device=DEV)
    for n in ("radbcs", "radbcn"):
        st[n] = torch.zeros((lay.NK, lay.NI), device=DEV)
    if cfg.ptype == 1:
        st["rain"], st["prate"] = (torch.zeros((lay.NJ, lay.NI), device=DEV) for _ in range(2))
    return {k: v.contiguous() for k, v in st.items()}


def _key(case):
    return (case["workload"], case["ni"], case["nj"], case["nk"], case["bc"], case["npt"], case["weno"], case["nsound"])


def _as_workload(case):
    """A routine's case with the workload its grid, sounding and state come from."""
    more = {"advs": dict(workload="dry_bubble", npt=0, nsound=6),
            "advuvw": dict(workload="dry_bubble", npt=0, weno=0, nsound=6),
            "sound": dict(workload="dry_bubble", npt=0, weno=0),
            "turbsmag": dict(workload="cbl", bc=1, weno=1, nsound=6),
            "diff2": dict(workload="cbl", bc=1, weno=1, nsound=6),
            "stats": dict(workload="supercell", bc=2, weno=1, nsound=8)}
    return {**case, **more.get(case["kind"], {})}


def _member_cases(case):
    r = random.Random(case["sizes"])
    return [dict(kind="step", workload="dry_bubble", ni=r.choice(ENSEMBLE_SIZES), nj=r.choice(ENSEMBLE_SIZES), nk=r.choice((40, 60, 80)),
                 bc=1, npt=0, weno=case["weno"], nsound=6) for _ in range(case["members"])]


def _domain(case, seed):
    cfg, grid, lay = _host_grid(*_key(case))
    return binding.Context(cfg, grid), _state(case, seed, cfg, grid, lay), lay, cfg, grid


def _surface_weights(dz):
    """Extrapolation of three half levels to the surface (and, mirrored, to the top)."""
    z = [0.5 * dz, 1.5 * dz, 2.5 * dz]
    return [math.prod((0.0 - z[m]) / (z[q] - z[m]) for m in range(3) if m != q) for q in range(3)]


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _prepare_train(case, seed)
    if kind == "ensemble":
        parts = [(c,) + _domain(c, seed + 31 * q)[:3] for q, c in enumerate(_member_cases(case))]
        ctxs, states = [p[1] for p in parts], [p[2] for p in parts]
        mass = [float(s["rho"][p[3].interior(1)].double().sum()) for p, s in zip(parts, states)]
        return dict(kind=kind, ens=binding.Ensemble(ctxs), ctxs=ctxs, states=states, dt=[WORKLOADS["dry_bubble"]["dt"]] * len(parts), mass=mass)
    case = _as_workload(case)
    ctx, st, lay, cfg, grid = _domain(case, seed)
    s = dict(kind=kind, ctx=ctx, lay=lay, dt=WORKLOADS[case["workload"]]["dt"], case=case)
    mk = _Maker(lay, case["bc"], seed + 7)
    if kind == "step":
        s.update(st=st, mass1=float(st["rho"][lay.interior(1)].double().sum()))
    elif kind == "advs":
        rho0, rf0 = _t(grid["rho0"][:, :1, :1]), _t(np.concatenate([grid["rf0"][:, :1, :1], grid["rf0"][-1:, :1, :1]]))
        s.update(rru=rho0 * st["ua"], rrv=rho0 * st["va"], rrw=rf0 * st["wa"], divx=mk.halo(mk.smooth(1, 1.0e-3), 1))
        q = (mk.smooth(1, 2.0e-3) - 3.0e-4).clamp_min(0.0) if case["pdef"] or case["pdefweno"] else mk.smooth(1, 2.0) + mk.noise(1, 0.05)
        s["s0"] = mk.halo(q, 1)
        s["s"] = mk.halo(q * (1.0 + mk.smooth(1, 0.05)), 1)
        s["sten"] = mk.halo(mk.smooth(1, 1.0e-6), 1)
        s["weps"] = 1.0e-20 if case["pdef"] or case["pdefweno"] else 1.0e-17
    elif kind == "advuvw":
        s.update(u=st["ua"], v=st["va"], w=st["wa"], ut=mk.halo(mk.smooth(2, 1e-3), 2), vt=mk.halo(mk.smooth(3, 1e-3), 3), wt=mk.halo(mk.smooth(4, 1e-3), 4))
    elif kind == "sound":
        a = {n: st[n] for n in ("radbcw", "radbce", "radbcs", "radbcn", "ua", "u3d", "va", "v3d", "wa", "w3d", "ppi", "pp3d")}
        a["ppx"] = mk.halo(mk.smooth(1, 1.0e-6), 1)
        a["rru"], a["rrv"], a["rrw"] = (torch.zeros_like(st[n]) for n in ("ua", "va", "wa"))
        a["uten"], a["vten"], a["wten"] = (mk.halo(mk.smooth(q, 5.0e-3), q) for q in (2, 3, 4))
        a["ppten"] = mk.halo(mk.smooth(1, 1.0e-9), 1)
        pi0, th0 = _t(grid["pi0"][:, :1, :1]), _t(grid["th0"][:, :1, :1])
        a["piadv"] = pi0 + st["pp3d"]
        a["thv"] = th0 + st["th3d"]
        a["ppterm"] = a["piadv"] * (RD / (CP - RD))
        s["a"] = {n: v.contiguous() for n, v in a.items()}
    elif kind in ("turbsmag", "diff2"):
        s.update(st=st, cg=_surface_weights(cfg.dz), csm=0.18, kdiff2=75.0)
        s["ten"] = {n: mk.halo(mk.smooth(q, 1.0e-4), q) for n, q in (("uten1", 2), ("vten1", 3), ("wten1", 4), ("thten1", 1))}
        s["ten"]["ptten"] = torch.zeros_like(st["pta"])
        if kind == "turbsmag":
            s["kmh"], s["kmv"] = (torch.zeros(lay.shape(4), device=DEV) for _ in range(2))
    else:
        opts, keep = stat_opts(_columns(case["workload"], case["nk"], case["bc"], case["npt"], case["weno"], case["nsound"]))
        s.update(st=st, keep=keep, names=ctx.stat_setup(opts), bud=np.zeros(cfg.numq))
    return s


def _prepare_train(case, seed):
    n = case["n"]
    binding.check(binding.lib().cm1g_mlp_set_activation(1 if case["act"] == "gelu" else 0))
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    rand = lambda *shape: torch.rand(shape, device=DEV, generator=gen)          # noqa: E731
    randn = lambda *shape: torch.randn(shape, device=DEV, generator=gen)        # noqa: E731
    # stencils of a rough scalar, normalised by their mean and range as the closure's features are
    v = torch.cumsum(randn(n, 6), 1)
    scale = v.amax(1) - v.amin(1) + 1e-6
    mean = v.mean(1)
    x = torch.zeros(n, 8, device=DEV)
    x[:, :6] = (v - mean[:, None]) / scale[:, None]
    x[:, 6] = 0.5 * rand(n)
    c5 = torch.tensor([2, -13, 47, 27, -3, 0], device=DEV) / 60.0
    target = mean + scale * ((x[:, :6] * c5).sum(1) + 0.05 * randn(n))
    p = torch.from_numpy(init_params(seed % 1000)).to(DEV)
    z = lambda *shape: torch.zeros(shape, device=DEV)                           # noqa: E731
    m2 = (1e-3 * (0.5 + rand(N_PARAMS))) ** 2
    return dict(kind="train", n=n, x=x, m=mean, d=scale, target=target, w=0.5 + rand(n), p=p, m1=1e-4 * randn(N_PARAMS), m2=m2, g=z(N_PARAMS),
                y=z(n, 8), z1=z(n, 64), z2=z(n, 64), dy=z(n, 8), loss=torch.zeros(1, dtype=torch.float64, device=DEV), step=100)


# ---------------------------------------------------------------- run
STEP_OUT = ("u3d", "v3d", "w3d", "pp3d", "ppx", "th3d", "rho", "prs", "q3d", "pt3d", "rain", "prate")


def run(s):
    kind = s["kind"]
    if kind == "step":
        mass2, cfl = s["ctx"].step(s["st"], s["dt"], s["mass1"], use_graph=True)
        return dict({n: s["st"][n] for n in STEP_OUT if n in s["st"]}, mass2=mass2, cfl=cfl)
    if kind == "ensemble":
        mass2, cfl = s["ens"].step(s["states"], s["dt"], s["mass"])
        return dict(mass2=np.array(mass2), cfl=np.array(cfl), **{n: [m[n] for m in s["states"]] for n in ("u3d", "w3d", "pp3d", "th3d")})
    if kind == "advs":
        c = s["case"]
        s["ctx"].advs(3, c["weno"], s["divx"], s["rru"], s["rrv"], s["rrw"], s["s0"], s["s"], s["sten"], c["pdef"], c["pdefweno"], s["dt"], s["weps"])
        return s["sten"]
    if kind == "advuvw":
        s["ctx"].advuvw(3, s["u"], s["v"], s["w"], s["ut"], s["vt"], s["wt"])
        return dict(ut=s["ut"], vt=s["vt"], wt=s["wt"])
    if kind == "sound":
        a = s["a"]
        s["ctx"].sound(3, s["dt"], s["dt"], **a)
        return {n: a[n] for n in SOUND_OUT}
    if kind == "turbsmag":
        c, st, t = s["case"], s["st"], s["ten"]
        s["ctx"].turbsmag(s["csm"], c["tconfig"], c["bcturbs"], c["bbc"], c["tbc"], s["cg"], s["cg"], st["ua"], st["va"], st["wa"], st["rho"],
                          st["tha"], st["pta"] if c["npt"] else None, t["uten1"], t["vten1"], t["wten1"], t["thten1"],
                          t["ptten"] if c["npt"] else None, s["kmh"], s["kmv"])
        return dict(t, kmh=s["kmh"], kmv=s["kmv"])
    if kind == "diff2":
        c, st, t = s["case"], s["st"], s["ten"]
        s["ctx"].diff2(s["kdiff2"], 1, c["bbc"], c["tbc"], s["cg"], s["cg"], st["ua"], st["va"], st["wa"], st["rho"], st["tha"], None,
                       st["pta"] if c["npt"] else None, t["uten1"], t["vten1"], t["wten1"], t["thten1"], None, t["ptten"] if c["npt"] else None)
        return dict(t)
    if kind == "stats":
        st = s["st"]
        return s["ctx"].statpack(3600.0, s["dt"], *[st[n] for n in ("ua", "va", "wa", "ppi", "tha", "prs", "rho")], qa=st["qa"],
                                 pta=st["pta"] if s["case"]["npt"] else None, asq=s["bud"], bsq=s["bud"])
    # one step of learned.train: forward, loss and its gradient, backward, Adam
    lib, check, f = binding.lib(), binding.check, binding.ptr
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    n = s["n"]
    check(lib.cm1g_mlp_forward(f(s["p"]), n, f(s["x"]), f(s["y"]), None, f(s["z1"]), f(s["z2"]), stream))
    s["loss"].zero_()
    check(lib.cm1g_closure_loss(n, f(s["x"]), f(s["y"]), f(s["m"]), f(s["d"]), f(s["target"]), f(s["w"]), f(s["dy"]),
                                C.c_void_p(s["loss"].data_ptr()), stream))
    s["g"].zero_()
    check(lib.cm1g_mlp_backward(f(s["p"]), n, f(s["x"]), f(s["z1"]), f(s["z2"]), f(s["dy"]), f(s["g"]), stream))
    s["step"] += 1
    check(lib.cm1g_adam(N_PARAMS, f(s["p"]), f(s["g"]), f(s["m1"]), f(s["m2"]), s["step"], 1e-3, 1.0 / n, stream))
    return {k: s[k] for k in TRAIN_OUT}


SOUND_OUT = ("u3d", "v3d", "w3d", "pp3d", "ppx", "rru", "rrv", "rrw")
TRAIN_OUT = ("y", "z1", "z2", "dy", "g", "loss", "p", "m1", "m2")


# ---------------------------------------------------------------- work
def work(case):
    """Bytes of every input array read once and every output written once, and the
    arithmetic of the method (about 20 operations a 5th-order face, 60 a WENO5 face,
    90 a cell and acoustic substep)."""
    kind = case["kind"]
    if kind == "train":
        macs = 8 * 64 + 64 * 64 + 64 * 8
        return dict(bytes=4.0 * case["n"] * (8 + 4 + 2 * 8 + 2 * 128), flops=6.0 * macs * case["n"])
    if kind == "ensemble":
        parts = [work(m) for m in _member_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    cells = float(case["ni"] * case["nj"] * case["nk"])
    npt = case.get("npt", 0)
    if kind == "step":
        nq = {"supercell": 1, "kessler": 3}.get(case["workload"], 0)
        ns = case["nsound"]
        loops = round(ns / 3.0) + ns // 2 + ns
        weno_stages = {0: 0, 1: 3, 2: 1}[case["weno"]]
        faces = (1 + nq + npt) * 3 * (60 * weno_stages + 20 * (3 - weno_stages)) + 3 * 3 * 3 * 20
        return dict(bytes=4.0 * cells * (16 + 13 + 5 * (nq + npt)), flops=cells * (90 * loops + faces + 200))
    per = {"advs": (6 + 2 * case.get("pdef", 0) * 0.5, 200 if case.get("weno") else 80), "advuvw": (9, 220),
           "sound": (15 + 8, 90 * case.get("nsound", 6)), "turbsmag": (5 + 8 + 2 + 3 * npt, 200 + 40 * npt),
           "diff2": (5 + 8 + 3 * npt, 150 + 30 * npt), "stats": (8 + npt, 300)}[kind]
    return dict(bytes=4.0 * cells * per[0], flops=cells * per[1])


# ---------------------------------------------------------------- exact
# The routines restated in 64 bits with plain tensor operations.  Whole steps and
# the statistics list have no such short form here: their outputs are compared with
# each other between builds.
def exact(case, seed):
    f = {"advs": _exact_advs, "advuvw": _exact_advuvw, "sound": _exact_sound, "turbsmag": _exact_turbsmag, "diff2": _exact_diff2,
         "train": _exact_train}.get(case["kind"])
    if f is None or (case["kind"] in ("advuvw", "sound") and case["bc"] != 1):   # open boundaries: edge forms not restated
        return None
    if case["kind"] != "train":
        case = _as_workload(case)
        _, grid, lay = _host_grid(*_key(case))
        return f(case, prepare(case, seed), {n: _t(grid[n][:, 0, 0]).double() for n in grid if grid[n].ndim == 3}, lay)
    return f(case, prepare(case, seed))


def _flx3(a, b, c):
    return (-a + 5 * b + 2 * c) / 6


def _flx5(a, b, c, d, e):
    return (2 * a - 13 * b + 47 * c + 27 * d - 3 * e) / 60


def _weno5(a, b, c, d, e, eps):
    b1 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b2 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b3 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    tau = (b1 - b3).abs()
    w1, w2, w3 = (g * (1 + (tau / (q + eps)).clamp_max(1e30) ** 2) for g, q in ((0.1, b1), (0.6, b2), (0.3, b3)))
    return (w1 * (2 * a - 7 * b + 11 * c) / 6 + w2 * (-b + 5 * c + 2 * d) / 6 + w3 * (2 * c + 5 * d - e) / 6) / (w1 + w2 + w3)


def _upstrpd(a, b, c, eps):
    d = b - a
    r = (c - b) / (torch.copysign(torch.full_like(d, eps), d) + d)
    return b + torch.minimum(r, torch.clamp_max(1 / 6 + r / 3, 1.0)).clamp_min(0.0) * d


def _faces(r, a, weno, pdef, eps):
    """Face fluxes from the mass flux r and the six values a[0..5] across each face."""
    up = r >= 0
    v = [torch.where(up, a[q], a[5 - q]) for q in range(5)]
    if not weno:
        return r * _flx5(*v)
    out = r * _weno5(*v, eps)
    return torch.where(torch.stack(v).abs().amax(0) > eps, out, 0.0) if pdef else out


def _pdef_fix(d, axis, lo, n):
    """Mass moved into the points lo .. lo+n-1 of `axis` to fill negative provisional masses."""
    v = lambda o: d.narrow(axis, lo + o, n)                     # noqa: E731
    pos = lambda t: t.clamp_min(0.0)                            # noqa: E731
    m, hit = torch.zeros_like(v(0)), torch.zeros_like(v(0), dtype=torch.bool)
    for c in (-1, 0, 1):                                        # the point that gives: below, itself, above
        have = pos(v(c - 1)) + pos(v(c + 1))
        on = (v(c) < 0) & (have > 1e-30)
        part = torch.maximum(v(c), -have) / have.clamp_min(1e-300)
        m += torch.where(on, -have * part if c == 0 else pos(v(0)) * part, 0.0)
        hit |= on if c == 0 else on & (v(0) > 1e-30)
    return m, hit


def _exact_advs(case, s, g, lay):
    ni, nj, nk, weno, pdef, eps = lay.ni, lay.nj, lay.nk, case["weno"], case["pdef"], s["weps"]
    dx, dz = float(s["ctx"].cfg.dx), float(s["ctx"].cfg.dz)
    K, J, I = slice(1, nk + 1), slice(3, 3 + nj), slice(3, 3 + ni)
    q, q0 = s["s"].double(), s["s0"].double()
    ru, rv, rw = s["rru"].double()[K, J, 3:4 + ni], s["rrv"].double()[K, 3:4 + nj, I], s["rrw"].double()[1:nk + 2, J, I]
    fx = _faces(ru, [q[K, J, d:d + ni + 1] for d in range(6)], weno, pdef, eps)
    fy = _faces(rv, [q[K, d:d + nj + 1, I] for d in range(6)], weno, pdef, eps)
    sc, col = q[K, J, I], q[:, J, I]
    fz = torch.zeros_like(rw)
    for kk in range(2, nk + 1):
        r = rw[kk - 1]
        A = lambda d: col[min(max(kk + d, 0), nk + 1)]          # noqa: E731
        lin = g["c1"][kk] * A(-1) + g["c2"][kk] * A(0)
        five = lambda: _faces(r, [A(d) for d in range(-3, 3)], weno, weno and case["pdefweno"], eps)   # noqa: E731,B023
        low_up = (lambda a, b, c: _upstrpd(a, b, c, eps)) if weno else _flx3
        if kk == 2:
            fz[kk - 1] = r * torch.where(r >= 0, lin, low_up(A(1), A(0), A(-1)))
        elif kk == nk:
            fz[kk - 1] = r * torch.where(r >= 0, low_up(A(-2), A(-1), A(0)), lin)
        elif kk == 3:
            fz[kk - 1] = torch.where(r >= 0, r * low_up(A(-2), A(-1), A(0)), five())
        elif kk == nk - 1:
            fz[kk - 1] = torch.where(r >= 0, five(), r * low_up(A(1), A(0), A(-1)))
        else:
            fz[kk - 1] = five()
    op = case["bc"] == 2
    inw, ine = (op & (ru[..., 0] >= 0)), (op & (ru[..., -1] <= 0))
    ins, inn = (op & (rv[:, 0] >= 0)), (op & (rv[:, -1] <= 0))
    fx[..., 0] = torch.where(inw, fx[..., 1], fx[..., 0])
    fx[..., -1] = torch.where(ine, fx[..., -2], fx[..., -1])
    fy[:, 0] = torch.where(ins, fy[:, 1], fy[:, 0])
    fy[:, -1] = torch.where(inn, fy[:, -2], fy[:, -1])
    ax, ay, az = -(fx[..., 1:] - fx[..., :-1]) / dx, -(fy[:, 1:] - fy[:, :-1]) / dx, -(fz[1:] - fz[:-1]) / dz
    dru, drv, drw = (ru[..., 1:] - ru[..., :-1]) / dx, (rv[:, 1:] - rv[:, :-1]) / dx, (rw[1:] - rw[:-1]) / dz
    ex, ey = torch.zeros_like(ax, dtype=torch.bool), torch.zeros_like(ay, dtype=torch.bool)
    ex[..., 0], ey[:, 0] = inw, ins
    ex[..., -1] |= ine
    ey[:, -1] |= inn
    ax, ay = ax - torch.where(ex, sc * dru, 0.0), ay - torch.where(ey, sc * drv, 0.0)
    if pdef:
        dt = s["dt"]
        m0 = g["rho0"][K, None, None] * q0[K, J, I]
        dumx = torch.where(ex, m0, m0 + dt * (ax + sc * dru))
        dumy = torch.where(ey, m0, m0 + dt * (ay + sc * drv))
        dumz = m0 + dt * (az + sc * drw)
        pad = dict(mode="replicate" if op else "circular")
        px = torch.nn.functional.pad(dumx, (3, 3), **pad)
        py = torch.nn.functional.pad(dumy.transpose(1, 2), (3, 3), **pad).transpose(1, 2)
        pz = torch.nn.functional.pad(dumz, (0, 0, 0, 0, 3, 3))
        for p, axis, n in ((px, 2, ni), (py, 1, nj), (pz, 0, nk)):
            m, hit = _pdef_fix(p, axis, 3, n)
            if axis == 2:
                ax = torch.where(hit, (dumx + m - m0) / dt - sc * dru, ax)
            elif axis == 1:
                ay = torch.where(hit, (dumy + m - m0) / dt - sc * drv, ay)
            else:
                az = torch.where(hit, (dumz + m - m0) / dt - sc * drw, az)
    out = s["sten"].double().clone()
    out[K, J, I] += (ax + ay + az + sc * s["divx"].double()[K, J, I]) * g["rr0"][K, None, None]
    return out


def _exact_advuvw(case, s, g, lay):
    ni, nj, nk = lay.ni, lay.nj, lay.nk
    dx, dz = float(s["ctx"].cfg.dx), float(s["ctx"].cfg.dz)
    K = slice(1, nk + 1)
    u, v, w = (s[n].double() for n in "uvw")
    ru, rv = g["rho0"][:, None, None] * u, g["rho0"][:, None, None] * v
    rf = torch.cat([g["rf0"], g["rf0"][-1:]])
    rw = rf[:, None, None] * w
    rw[:2] = 0.0
    rw[nk + 1:] = 0.0
    div = torch.zeros(lay.shape(1), dtype=torch.float64, device=DEV)
    div[K] = (ru[K, :, 1:] - ru[K, :, :-1]) / dx + (rv[K, 1:] - rv[K, :-1]) / dx + (rw[2:nk + 2] - rw[1:nk + 1]) / dz

    def horizontal(a, r, axis, n):
        """Flux difference along `axis` over n points from 3: r at the faces of points 3 .. 3+n."""
        f = _faces(r, [a.narrow(axis, d, n + 1) for d in range(6)], 0, 0, 0.0)
        return f.narrow(axis, 1, n) - f.narrow(axis, 0, n)

    def vertical(a, wb):
        """Face fluxes of a u- or v-column at w-levels 1 .. nk+1 (a and wb over the output points)."""
        f = torch.zeros((nk + 1,) + a.shape[1:], dtype=torch.float64, device=DEV)
        for kk in range(2, nk + 1):
            A = lambda d: a[min(max(kk + d, 0), nk + 1)]        # noqa: E731,B023
            r = wb[kk]
            lin = (1 - g["c2"][kk]) * A(-1) + g["c2"][kk] * A(0)
            up = lin if kk == 2 else _flx3(A(-2), A(-1), A(0)) if kk in (3, nk) else _flx5(*[A(d) for d in range(-3, 2)])
            dn = lin if kk == nk else _flx3(A(1), A(0), A(-1)) if kk in (2, nk - 1) else _flx5(*[A(d) for d in (2, 1, 0, -1, -2)])
            f[kk - 1] = r * torch.where(r >= 0, up, dn)
        return f

    J, I = slice(3, 3 + nj), slice(3, 3 + ni)
    rr0 = g["rr0"][K, None, None]
    # u at i = 1..ni+1
    J1, I1 = slice(3, 4 + nj), slice(3, 4 + ni)
    ubx = 0.5 * (ru[..., 1:] + ru[..., :-1])                    # s-points
    adv = -horizontal(u[K, J], ubx[K, J, 2:4 + ni], 2, ni + 1) / dx
    vb = 0.5 * (rv[K, 3:4 + nj, 3:4 + ni] + rv[K, 3:4 + nj, 2:3 + ni])
    adv -= horizontal(u[K, :, I1], vb, 1, nj) / dx
    fz = vertical(u[:, J, I1], 0.5 * (rw[:, J, 3:4 + ni] + rw[:, J, 2:3 + ni]))
    adv -= (fz[1:] - fz[:-1]) / dz
    ut = s["ut"].double().clone()
    ut[K, J, I1] += (adv + u[K, J, I1] * 0.5 * (div[K, J, 3:4 + ni] + div[K, J, 2:3 + ni])) * rr0
    # v at j = 1..nj+1
    ub = 0.5 * (ru[K, 3:4 + nj, 3:4 + ni] + ru[K, 2:3 + nj, 3:4 + ni])
    adv = -horizontal(v[K, J1], ub, 2, ni) / dx
    vby = 0.5 * (rv[:, 1:] + rv[:, :-1])
    adv -= horizontal(v[K, :, I], vby[K, 2:4 + nj, I], 1, nj + 1) / dx
    fz = vertical(v[:, J1, I], 0.5 * (rw[:, 3:4 + nj, I] + rw[:, 2:3 + nj, I]))
    adv -= (fz[1:] - fz[:-1]) / dz
    vt = s["vt"].double().clone()
    vt[K, J1, I] += (adv + v[K, J1, I] * 0.5 * (div[K, 3:4 + nj, I] + div[K, 2:3 + nj, I])) * rr0
    # w at k = 2..nk
    W, c1, c2 = slice(2, nk + 1), g["c1"][2:nk + 1, None, None], g["c2"][2:nk + 1, None, None]
    ub = (c2 * ru[W, J] + (1 - c2) * ru[1:nk, J])[..., 3:4 + ni]
    vb = (c2 * rv[W] + (1 - c2) * rv[1:nk])[:, 3:4 + nj, I]
    adv = -horizontal(w[W, J], ub, 2, ni) / dx - horizontal(w[W, :, I], vb, 1, nj) / dx
    col = w[:, J, I]
    f = torch.zeros((nk + 1, nj, ni), dtype=torch.float64, device=DEV)
    for kk in range(1, nk + 1):
        A = lambda d: col[min(max(kk + d, 0), nk + 2)]          # noqa: E731
        r = 0.5 * (rw[kk] + rw[kk + 1])[J, I]
        lin = 0.5 * (A(0) + A(1))
        up = lin if kk == 1 else _flx3(A(-1), A(0), A(1)) if kk in (2, nk) else _flx5(*[A(d) for d in range(-2, 3)])
        dn = lin if kk == nk else _flx3(A(2), A(1), A(0)) if kk in (1, nk - 1) else _flx5(*[A(d) for d in (3, 2, 1, 0, -1)])
        f[kk] = r * torch.where(r >= 0, up, dn)
    adv -= (f[2:] - f[1:-1]) / dz
    wt = s["wt"].double().clone()
    wt[W, J, I] += (adv + w[W, J, I] * (c2 * div[W, J, I] + c1 * div[1:nk, J, I])) * g["rrf0"][2:nk + 1, None, None]
    return dict(ut=ut, vt=vt, wt=wt)


def _exact_sound(case, s, g, lay):
    """The final stage's acoustic substeps on a periodic domain (sound.F, one column solve a step)."""
    ni, nj, nk, ns = lay.ni, lay.nj, lay.nk, case["nsound"]
    cfg = s["ctx"].cfg
    dx, dz, alph, kdiv, dts = float(cfg.dx), float(cfg.dz), float(cfg.alph), float(cfg.kdiv), s["dt"] / ns
    K, J, I = slice(1, nk + 1), slice(3, 3 + nj), slice(3, 3 + ni)
    a = {n: v.double() for n, v in s["a"].items()}
    P = {n: a[n][K, J, I] for n in ("piadv", "ppten", "thv", "ppterm", "ppi", "ppx")}
    u, v, w = a["ua"][K, J, I], a["va"][K, J, I], a["wa"][1:nk + 2, J, I].clone()
    uten, vten, wten = a["uten"][K, J, I], a["vten"][K, J, I], a["wten"][1:nk + 2, J, I]
    west, east = (lambda t: t.roll(1, 2)), (lambda t: t.roll(-1, 2))
    south, north = (lambda t: t.roll(1, 1)), (lambda t: t.roll(-1, 1))
    pia, thv, ppt = P["piadv"], P["thv"], P["ppterm"]
    rr0, rf0 = g["rr0"][K, None, None], g["rf0"]
    rf_lo, rf_up = rf0[1:nk + 1, None, None], rf0[2:nk + 2, None, None]
    c1, c2 = g["c1"][:, None, None], g["c2"][:, None, None]
    zero = torch.zeros_like(pia[:1])
    dn, up = torch.cat([zero, pia[:-1]]), torch.cat([pia[1:], zero])
    qk = dts / dz * ppt
    p2 = dts / dz * rr0 * rf_up * (-c2[2:nk + 2] * up + (1 - c1[2:nk + 2]) * pia)
    p1 = dts / dz * rr0 * rf_lo * (c1[1:nk + 1] * dn + (c2[1:nk + 1] - 1) * pia)
    p2[-1], p1[0] = 0.0, 0.0
    p1, p2 = p1 + qk, p2 - qk
    mm = dts / dz * CP * (c2[2:nk + 1] * thv[1:] + c1[2:nk + 1] * thv[:-1])     # w-levels 2..nk
    beta, asq = 1 - alph, alph * alph
    bb = 1 - asq * mm * (-p1[1:] + p2[:-1])
    aa, cc = -asq * mm * p1[:-1], asq * mm * p2[1:]
    pp, ppd = P["ppi"], P["ppx"]
    ru, rv, rw = torch.zeros_like(u), torch.zeros_like(v), w * beta
    for n in range(1, ns + 1):
        u = u + dts * (uten - 0.5 * CP / dx * (ppd - west(ppd)) * (thv + west(thv)))
        v = v + dts * (vten - 0.5 * CP / dx * (ppd - south(ppd)) * (thv + south(thv)))
        ru, rv = ru + u, rv + v
        div = (east(u) - u) / dx + (north(v) - v) / dx
        X = u * (pia - west(pia)) + east(u) * (east(pia) - pia)
        Y = v * (pia - south(pia)) + north(v) * (north(pia) - pia)
        f = pp + dts * (P["ppten"] - ppt * div) - (X + Y) * dts * 0.5 / dx + beta * (w[:-1] * p1 + w[1:] * p2)
        d = w[1:nk] + dts * wten[1:nk] - beta * mm * (pp[1:] - pp[:-1]) - alph * mm * (f[1:] - f[:-1])
        e1, e2 = torch.empty_like(d), torch.empty_like(d)
        for k in range(nk - 1):
            r = 1 / (bb[k] + (aa[k] * e1[k - 1] if k else 0.0))
            e1[k] = -cc[k] * r
            e2[k] = (d[k] - (aa[k] * e2[k - 1] if k else 0.0)) * r
        w = w.clone()
        for k in range(nk - 2, -1, -1):
            w[k + 1] = e2[k] + (e1[k] * w[k + 2] if k < nk - 2 else 0.0)
        new = f + alph * (w[:-1] * p1 + w[1:] * p2)
        step = kdiv * (new - pp)
        pp, ppd = new, new + step
        rw = rw + w * (alph if n == ns else 1.0)
    out = {n: a[n].clone() for n in SOUND_OUT}
    wrap = lambda t, axis: torch.cat([t, t.narrow(axis, 0, 1)], axis)            # noqa: E731
    out["u3d"][K, J, 3:4 + ni], out["rru"][K, J, 3:4 + ni] = wrap(u, 2), wrap(ru, 2) / ns
    out["v3d"][K, 3:4 + nj, I], out["rrv"][K, 3:4 + nj, I] = wrap(v, 1), wrap(rv, 1) / ns
    out["w3d"][2:nk + 1, J, I], out["rrw"][1:nk + 1, J, I] = w[1:nk], rw[:nk] / ns
    out["pp3d"][K, J, I], out["ppx"][K, J, I] = pp, step
    return out


def _rf(rho, g, cg, nk):
    """Density at the w-levels 1 .. nk+1 (rho: full array)."""
    f = torch.zeros_like(rho)
    f[2:nk + 1] = g["c1"][2:nk + 1, None, None] * rho[1:nk] + g["c2"][2:nk + 1, None, None] * rho[2:nk + 1]
    f[1] = cg[0] * rho[1] + cg[1] * rho[2] + cg[2] * rho[3]
    f[nk + 1] = cg[0] * rho[nk] + cg[1] * rho[nk - 1] + cg[2] * rho[nk - 2]
    return f


def _exact_turbsmag(case, s, g, lay):
    """Smagorinsky tendencies on a periodic domain; every array is held at 1 .. n and wrapped by roll."""
    ni, nj, nk = lay.ni, lay.nj, lay.nk
    cfg = s["ctx"].cfg
    dx, dz, csm, prinv = float(cfg.dx), float(cfg.dz), s["csm"], 3.0
    J, I = slice(3, 3 + nj), slice(3, 3 + ni)
    inner = lambda t: t.double()[..., J, I]                     # noqa: E731
    st = s["st"]
    u, v, w, rho, th = (inner(st[n]) for n in ("ua", "va", "wa", "rho", "tha"))
    W, E = (lambda t: t.roll(1, -1)), (lambda t: t.roll(-1, -1))
    S, N = (lambda t: t.roll(1, -2)), (lambda t: t.roll(-1, -2))
    K, Q = slice(1, nk + 1), slice(2, nk + 1)                   # s-levels, inner w-levels
    rf = _rf(rho, g, s["cg"], nk)
    dk = lambda t: (t[Q] - t[1:nk]) / dz                        # noqa: E731
    t11, t22 = rho * (E(u) - u) / dx, rho * (N(v) - v) / dx
    t33 = torch.zeros_like(rho)
    t33[K] = rho[K] * (w[2:nk + 2] - w[K]) / dz
    t12 = 0.5 * ((u - S(u)) / dx + (v - W(v)) / dx) * 0.25 * (W(S(rho)) + rho + W(rho) + S(rho))
    s13, s23 = torch.zeros_like(rf), torch.zeros_like(rf)
    s13[Q] = 0.5 * ((w[Q] - W(w)[Q]) / dx + dk(u)) * 0.5 * (W(rf)[Q] + rf[Q])
    s23[Q] = 0.5 * ((w[Q] - S(w)[Q]) / dx + dk(v)) * 0.5 * (S(rf)[Q] + rf[Q])
    c1, c2 = g["c1"][Q, None, None], g["c2"][Q, None, None]
    mid = lambda t: c1 * t[1:nk] + c2 * t[Q]                    # noqa: E731
    p12 = t12 ** 2
    sh = (2 * mid(t11 ** 2 + t22 ** 2 + t33 ** 2) + mid(p12 + E(N(p12)) + N(p12) + E(p12))) / rf[Q] ** 2
    sv = 2 * ((s13 ** 2 + E(s13 ** 2))[Q] + (s23 ** 2 + N(s23 ** 2))[Q]) / rf[Q] ** 2
    full = g["th0"][:, None, None] + th
    nm = torch.log(full[Q] / full[1:nk]) * 9.81 / dz
    km = [torch.zeros_like(rf), torch.zeros_like(rf)]
    if case["tconfig"] == 1:
        km[0][Q] = (csm * (dx * dx * dz) ** (1 / 3)) ** 2 * torch.sqrt((sv + sh - nm * prinv).clamp_min(1e-10))
        km[1] = km[0]
    else:
        km[0][Q] = (csm * dx) ** 2 * torch.sqrt(sh.clamp_min(1e-10))
        km[1][Q] = (csm * dz) ** 2 * torch.sqrt((sv - nm * prinv).clamp_min(1e-10))
    kh, kv = km
    tem = torch.zeros_like(rho)
    tem[K] = kh[K] + kh[2:nk + 2]
    t11, t22, t33 = t11 * tem, t22 * tem, t33 * tem
    t12 = t12 * 0.25 * (W(S(tem)) + tem + W(tem) + S(tem))
    t13, t23 = s13 * (W(kv) + kv), s23 * (S(kv) + kv)
    for t, vel, back in ((t13, u, W), (t23, v, S)):
        for row, lev, near, sign, free in ((1, 1, 2, 1.0, case["bbc"] == 1), (nk + 1, nk, nk, -1.0, case["tbc"] == 1)):
            t[row] = t[near] if free else sign * 2 * vel[lev] / dz * 0.5 * (back(rf)[row] + rf[row]) * 0.5 * (back(kv)[near] + kv[near])
    out = {n: t.double().clone() for n, t in s["ten"].items()}
    dz1 = lambda t: (t[2:nk + 2] - t[K]) / dz                   # noqa: E731
    wrap = lambda t, axis: torch.cat([t, t.narrow(axis, 0, 1)], axis)            # noqa: E731
    du = ((t11 - W(t11)) / dx + (N(t12) - t12) / dx)[K] + dz1(t13)
    dv = ((E(t12) - t12) / dx + (t22 - S(t22)) / dx)[K] + dz1(t23)
    out["uten1"][K, J, 3:4 + ni] += wrap(du / (0.5 * (W(rho) + rho))[K], 2)
    out["vten1"][K, 3:4 + nj, I] += wrap(dv / (0.5 * (S(rho) + rho))[K], 1)
    out["wten1"][Q, J, I] += ((E(t13) - t13 + N(t23) - t23)[Q] / dx + (t33[Q] - t33[1:nk]) / dz) / rf[Q]
    fields = [("thten1", None, full)] + [("ptten", n, inner(st["pta"][n])) for n in range(case["npt"])]
    for name, n, q in fields:
        fx = -0.125 * (rho + W(rho)) * prinv * (tem + W(tem)) * (q - W(q)) / dx
        fy = -0.125 * (rho + S(rho)) * prinv * (tem + S(tem)) * (q - S(q)) / dx
        fz = torch.zeros_like(rf)
        fz[Q] = -kv[Q] * prinv * dk(q) * rf[Q]
        if case["bcturbs"] == 2:                                # the flux of the nearest inner level, its own density
            fz[1], fz[nk + 1] = fz[2], fz[nk]
        d = -((E(fx) - fx + N(fy) - fy)[K] / dx + dz1(fz)) / rho[K]
        t = out[name] if n is None else out[name][n]
        t[K, J, I] += d
    # kmh and kmv carry one halo point all round; points beyond it stay zero
    for name, t in (("kmh", kh), ("kmv", kv)):
        o = torch.zeros(lay.shape(4), dtype=torch.float64, device=DEV)
        ring = lambda n: torch.arange(-1, n + 1, device=DEV) % n                 # noqa: E731
        o[:nk + 2, 2:4 + nj, 2:4 + ni] = t[:, ring(nj)][:, :, ring(ni)]
        out[name] = o
    return out


def _exact_diff2(case, s, g, lay):
    """Fixed-viscosity diffusion on a periodic domain."""
    ni, nj, nk = lay.ni, lay.nj, lay.nk
    cfg = s["ctx"].cfg
    dx, dz, coef = float(cfg.dx), float(cfg.dz), s["kdiff2"]
    J, I = slice(3, 3 + nj), slice(3, 3 + ni)
    inner = lambda t: t.double()[..., J, I]                     # noqa: E731
    st = s["st"]
    u, v, w, rho, th = (inner(st[n]) for n in ("ua", "va", "wa", "rho", "tha"))
    W, E = (lambda t: t.roll(1, -1)), (lambda t: t.roll(-1, -1))
    S, N = (lambda t: t.roll(1, -2)), (lambda t: t.roll(-1, -2))
    K, Q = slice(1, nk + 1), slice(2, nk + 1)
    rf = _rf(rho, g, s["cg"], nk)
    ux, vy = (E(u) - u) / dx, (N(v) - v) / dx
    wz = torch.zeros_like(rho)
    wz[K] = (w[2:nk + 2] - w[K]) / dz
    bulk = rho * (2 / 3) * (ux + vy + wz)
    t11, t22, t33 = (2 * coef * rho * d - bulk for d in (ux, vy, wz))
    t12 = coef * ((u - S(u)) / dx + (v - W(v)) / dx) * 0.25 * (W(S(rho)) + rho + W(rho) + S(rho))
    t13, t23 = torch.zeros_like(rf), torch.zeros_like(rf)
    t13[Q] = coef * ((u[Q] - u[1:nk]) / dz + (w - W(w))[Q] / dx)
    t23[Q] = coef * ((v[Q] - v[1:nk]) / dz + (w - S(w))[Q] / dx)
    for t, vel in ((t13, u), (t23, v)):
        t[1] = t[2] if case["bbc"] == 1 else coef * 2 * vel[1] / dz
        t[nk + 1] = t[nk] if case["tbc"] == 1 else -coef * 2 * vel[nk] / dz
    t13, t23 = t13 * 0.5 * (W(rf) + rf), t23 * 0.5 * (S(rf) + rf)
    out = {n: t.double().clone() for n, t in s["ten"].items()}
    dz1 = lambda t: (t[2:nk + 2] - t[K]) / dz                   # noqa: E731
    wrap = lambda t, axis: torch.cat([t, t.narrow(axis, 0, 1)], axis)            # noqa: E731
    du = ((t11 - W(t11)) / dx + (N(t12) - t12) / dx)[K] + dz1(t13)
    dv = ((E(t12) - t12) / dx + (t22 - S(t22)) / dx)[K] + dz1(t23)
    out["uten1"][K, J, 3:4 + ni] += wrap(du / (0.5 * (W(rho) + rho))[K], 2)
    out["vten1"][K, 3:4 + nj, I] += wrap(dv / (0.5 * (S(rho) + rho))[K], 1)
    out["wten1"][Q, J, I] += ((E(t13) - t13 + N(t23) - t23)[Q] / dx + (t33[Q] - t33[1:nk]) / dz) / rf[Q]
    fields = [("thten1", None, th)] + [("ptten", n, inner(st["pta"][n])) for n in range(case["npt"])]
    for name, n, q in fields:
        fx, fy = 0.5 * (rho + W(rho)) * (q - W(q)) / dx, 0.5 * (rho + S(rho)) * (q - S(q)) / dx
        fz = torch.zeros_like(rf)
        fz[Q] = rf[Q] * (q[Q] - q[1:nk]) / dz
        t = out[name] if n is None else out[name][n]
        t[K, J, I] += coef * ((E(fx) - fx + N(fy) - fy)[K] / dx + dz1(fz)) / rho[K]
    return out


def _exact_train(case, s):
    """The training step with operands rounded to BF16 where the network defines it, sums in 64 bits."""
    gelu = case["act"] == "gelu"
    bf = lambda t: t.float().bfloat16().double()                # noqa: E731
    act = (lambda z: 0.5 * z * (1 + torch.erf(z / math.sqrt(2)))) if gelu else (lambda z: z.clamp_min(0.0))

    def grad(z):
        if not gelu:
            return (z > 0).double()
        return 0.5 * (1 + torch.erf(z / math.sqrt(2))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi)

    p, x, n = s["p"].double(), s["x"].double(), case["n"]
    w1, b1, w2, b2, w3, b3 = (t for t in p.split([8 * 64, 64, 64 * 64, 64, 64 * 8, 8]))
    w1, w2, w3 = w1.view(8, 64), w2.view(64, 64), w3.view(64, 8)
    xb = bf(x)
    z1 = xb @ bf(w1) + b1
    h1 = bf(act(z1))
    z2 = h1 @ bf(w2) + b2
    h2 = bf(act(z2))
    y = h2 @ bf(w3) + b3
    y[:, 6:] = 0.0
    c = y[:, :6] + (1 - y[:, :6].sum(1, keepdim=True)) / 6
    e = s["m"].double() + s["d"].double() * (c * x[:, :6]).sum(1) - s["target"].double()
    wd = s["w"].double()
    dc = 2 * (wd * e * s["d"].double())[:, None] * x[:, :6]
    dy = torch.zeros_like(y)
    dy[:, :6] = dc - dc.sum(1, keepdim=True) / 6
    d2 = (dy @ bf(w3).T) * grad(z2)
    d1 = (d2 @ bf(w2).T) * grad(z1)
    xm = xb.clone()
    xm[:, 7] = 0.0
    g = torch.cat([(xm.T @ d1).reshape(-1), d1.sum(0), (h1.T @ d2).reshape(-1), d2.sum(0), (h2.T @ dy).reshape(-1), dy.sum(0)])
    gs, t = g / n, s["step"] + 1
    m1, m2 = 0.9 * s["m1"].double() + 0.1 * gs, 0.999 * s["m2"].double() + 0.001 * gs * gs
    new = p - 1e-3 * (m1 / (1 - 0.9 ** t)) / (torch.sqrt(m2 / (1 - 0.999 ** t)) + 1e-8)
    return dict(y=y, z1=z1, z2=z2, dy=dy, g=g, loss=(wd * e * e).sum().reshape(1), p=new, m1=m1, m2=m2)
