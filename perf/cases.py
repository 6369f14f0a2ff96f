"""Performance cases of the SPH step: the calls a program makes, at the sizes it makes them.

Workloads are the ones of this repository's configurations (lid-driven cavity, dam
break, heated channel, batched sweep, reverse mode, the GPU-C dam break and pressure
wave), in a developed state: disordered particles, moving, under pressure. Every pass
starts from the same input state (the arrays a call updates are put back first), so
passes are alike. `exact` restates the step in 64 bits with torch alone.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import armando_gb300 as ag
from armando_gb300._abi import Material

G = 9.81
DEV = "cuda"
H_DX = 1.3  # smoothing length over particle spacing of the CERN-scheme workloads
# arrays a call updates / only reads, with their components per particle (0: dim)
MUTABLE = (("x", 0), ("v", 0), ("rho", 1), ("p", 1), ("u", 1), ("dvdt", 0), ("dudt", 1))
FIXED = (("mass", 1), ("h", 1), ("itype", 1))


# ---- the cases -------------------------------------------------------------------

def listed():
    return [
        # The smallest call: a host code stepping a 40 x 40 cavity one iteration at a
        # time on device arrays, library defaults. Launches and latency.
        dict(name="cavity_step", family="cavity", n_side=40, call="step", reach=1, tpp=1, block=128, skin=0),
        # A cavity run on the device between two snapshots, physical viscosity, tuned.
        dict(name="cavity_run", family="cavity", n_side=160, call="run", steps=10, reach=2, tpp=1, block=128,
             skin=10),
        # One iteration of a mid-size dam break on device arrays, library defaults,
        # ragged sizes (nothing divides 32).
        dict(name="dam_step", family="dam", ny=283, call="step", reach=1, tpp=1, block=128, skin=0, options=0),
        # single_step's options: normalised density and the XSPH velocity.
        dict(name="dam_options", family="dam", ny=667, call="step", reach=3, tpp=1, block=256, skin=0, options=1),
        # The benchmark's run: 2.03 M particles between two snapshots, tuned.
        dict(name="dam_run", family="dam", ny=2000, call="run", steps=6, reach=3, tpp=1, block=128, skin=10,
             options=0),
        # The benchmark's end-to-end call: one iteration on page-locked host arrays.
        dict(name="dam_step_host", family="dam", ny=2000, call="host", reach=1, tpp=1, block=128, skin=0,
             options=0),
        # A small 3D channel section (art. heat, source, periodic x), tuned.
        dict(name="channel_section", family="channel", n_x=131, n_yz=33, call="run", steps=6, reach=3, tpp=1,
             block=128, skin=10),
        # The 3D channel of the configuration, 8.78 M particles: the largest system.
        dict(name="channel_run", family="channel", n_x=504, n_yz=126, call="run", steps=4, reach=3, tpp=1,
             block=128, skin=20),
        # A parameter sweep: 64 systems of 2e3 to 2e5 particles advancing together.
        dict(name="sweep", family="sweep", instances=64, layout=4, call="batch", steps=3, reach=2),
        # Reverse mode: forward with checkpoints, then the backward sweep.
        dict(name="adjoint", family="adjoint", ny=707, call="adjoint", steps=4, every=2, reach=3, tpp=1, block=128,
             skin=0),
        # The GPU-C scheme: the published dam break case 3 and pressure wave case 3.
        dict(name="gpuc_dam", family="gpuc_dam", scale=4, scheme=1, call="run", steps=5, reach=2, tpp=1, block=256,
             skin=10),
        dict(name="gpuc_wave", family="gpuc_wave", n_side=601, scheme=1, call="run", steps=5, reach=3, tpp=1,
             block=128, skin=10),
    ]


def draw(rng: random.Random) -> dict:
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    tuned = dict(reach=rng.choice((1, 2, 3)), tpp=1, block=rng.choice((128, 256)), skin=rng.choice((10, 10, 20)))
    plain = dict(reach=rng.choice((1, 1, 2, 3)), tpp=1, block=rng.choice((128, 256)), skin=0)
    kind = rng.choice(("cavity_step", "cavity_run", "dam_step", "dam_run", "dam_run", "dam_options", "dam_host",
                       "channel", "channel", "sweep", "adjoint", "gpuc_dam", "gpuc_wave"))
    if kind == "cavity_step":
        return dict(family="cavity", n_side=log_int(24, 240), call="step", **plain)
    if kind == "cavity_run":
        return dict(family="cavity", n_side=log_int(40, 240), call="run", steps=rng.randint(4, 10), **tuned)
    if kind == "dam_step":
        return dict(family="dam", ny=log_int(60, 1900), call="step", options=0, **plain)
    if kind == "dam_run":
        return dict(family="dam", ny=log_int(100, 1900), call="run", steps=rng.randint(3, 6), options=0, **tuned)
    if kind == "dam_options":
        return dict(family="dam", ny=log_int(100, 1200), call="step", options=1, **plain)
    if kind == "dam_host":
        return dict(family="dam", ny=log_int(200, 1900), call="host", options=0, **plain)
    if kind == "channel":
        n_yz = log_int(20, 100)
        return dict(family="channel", n_x=rng.randint(3 * n_yz, 4 * n_yz), n_yz=n_yz, call="run",
                    steps=rng.randint(2, 4), **tuned)
    if kind == "sweep":
        return dict(family="sweep", instances=log_int(8, 60), layout=rng.randint(5, 10 ** 6), call="batch",
                    steps=rng.randint(2, 4), reach=rng.choice((1, 2, 3)))
    if kind == "adjoint":
        return dict(family="adjoint", ny=log_int(80, 700), call="adjoint", steps=rng.randint(2, 4), every=2, **plain)
    if kind == "gpuc_dam":
        return dict(family="gpuc_dam", scale=rng.choice((1, 2, 3, 4)), scheme=rng.choice((1, 1, 2)), call="run",
                    steps=rng.randint(3, 5), **tuned)
    return dict(family="gpuc_wave", n_side=log_int(150, 590), scheme=1, call="run", steps=rng.randint(3, 5), **tuned)


# ---- inputs ----------------------------------------------------------------------

def _f32(v: float) -> float:
    """The value a float field of the parameters holds."""
    return float(np.float32(v))


def _kernel_sum(dim: int, h: float) -> float:
    """sum of W(|k|, h) over the unit lattice: the density of unit masses on it."""
    m = int(math.ceil(2 * h)) + 1
    ax = np.arange(-m, m + 1, dtype=np.float64)
    r = np.sqrt(sum(a * a for a in np.meshgrid(*([ax] * dim), indexing="ij")))
    t = np.clip(1.0 - 0.5 * r / h, 0.0, None)
    k = 7.0 / (4.0 * math.pi * h ** 2) if dim == 2 else 21.0 / (16.0 * math.pi * h ** 3)
    return float((k * t ** 4 * (1.0 + 2.0 * r / h)).sum())


def _lattice(*counts):
    ax = [torch.arange(a, b, dtype=torch.float64, device=DEV) for a, b in counts]
    return torch.stack([m.reshape(-1) for m in torch.meshgrid(*ax, indexing="ij")], 1)


def _noise(gen, *shape):
    return torch.randn(*shape, dtype=torch.float64, device=DEV, generator=gen)


def _jitter(gen, x, amount):
    return x + (2.0 * torch.rand(x.shape, dtype=torch.float64, device=DEV, generator=gen) - 1.0) * amount


def _swirl(x, lo, hi, speed):
    """A smooth flow of about `speed` with no flux through the box [lo, hi] (2D; z carried along)."""
    s = [(x[:, d] - lo[d]) / (hi[d] - lo[d]) * math.pi for d in range(2)]
    v = torch.zeros_like(x)
    v[:, 0] = speed * torch.sin(s[0]) * torch.cos(s[1])
    v[:, 1] = -speed * torch.cos(s[0]) * torch.sin(s[1])
    return v


def _pack(ph, xf, vf, xw, vw, mf, mw, rho, p, uf, uw, h, dx, gen, wall_type=0):
    """The step's arrays, fluid first; the previous rates are body force plus noise."""
    nf, nw, dim = len(xf), len(xw), xf.shape[1]
    n = nf + nw
    a = torch.zeros(n, dim, dtype=torch.float64, device=DEV)
    for d in range(dim):
        a[:nf, d] = ph["gravity"][d]
    a[:nf] += _noise(gen, nf, dim) * (0.002 * ph["c0"] ** 2 / dx)
    s = dict(x=torch.cat([xf, xw]), v=torch.cat([vf, vw]), mass=torch.cat([mf, mw]), rho=rho, p=p,
             u=torch.cat([uf, uw]), h=torch.full((n,), h, dtype=torch.float64, device=DEV),
             dvdt=a, dudt=torch.zeros(n, dtype=torch.float64, device=DEV))
    s = {k: t.reshape(-1).to(torch.float32).contiguous() for k, t in s.items()}
    s["itype"] = torch.cat([torch.ones(nf, dtype=torch.int32, device=DEV),
                            torch.full((nw,), wall_type, dtype=torch.int32, device=DEV)])
    return dict(ph=ph, dim=dim, nf=nf, nw=nw, arrays=s)


def _physics(**kw):
    ph = dict(dim=2, pa_sph=1, visc=0, visc_artificial=0, heat_artificial=0, heat_external=0, rho0=1000.0, c0=1.0,
              pmin=-math.inf, eta=0.0, av_alpha=1.0, av_beta=1.0, av_eta=0.1, ah_g1=0.1, ah_g2=1.0, ah_eta=0.1,
              gravity=(0.0, 0.0, 0.0), heat_q0=0.0, heat_sigma=1.0, heat_center=(0.0, 0.0, 0.0), period=0.0,
              scheme=0, density_form=0, average_velocity=0, material=None)
    ph.update(kw)
    return ph


def _params(ph):
    p = ag.Params.default(**{k: v for k, v in ph.items() if k not in ("period", "material", "dt")})
    if ph["period"]:
        p.set("periodic", (1, 0, 0))
        p.set("period_lo", (0.0, 0.0, 0.0))
        p.set("period_hi", (ph["period"], 0.0, 0.0))
    return p


def _tait_rho(p, rho0, c0):
    return rho0 * (1.0 + 7.0 * p / (rho0 * c0 * c0)) ** (1.0 / 7.0)


def _cavity(n_side, gen, length=1.0e-3, lid=1.0e-3, c0=0.01, eta=1.0e-3, alpha=None):
    """The lid-driven cavity: n_side^2 fluid particles, walls at half spacing."""
    dx = length / n_side
    h, rho0 = H_DX * dx, 1000.0
    ph = _physics(rho0=rho0, c0=c0, visc=1, eta=eta, dt=5.0e-5 * (40.0 / n_side) ** 2)
    if alpha is not None:
        ph.update(visc=0, eta=0.0, visc_artificial=1, av_alpha=alpha, av_beta=0.0, dt=0.2 * h / c0)
    xf = _jitter(gen, (_lattice((0, n_side), (0, n_side)) + 0.5) * dx, 0.15 * dx)
    k = torch.arange(2 * n_side, dtype=torch.float64, device=DEV) * (0.5 * dx)
    z, e = torch.zeros_like(k), torch.full_like(k, length)
    xw = torch.cat([torch.stack(s, 1) for s in ((k, z), (e, k), (length - k, e), (z, length - k))])
    vw = torch.zeros_like(xw)
    vw[4 * n_side:6 * n_side, 0] = lid
    vf = _swirl(xf, (0.0, 0.0), (length, length), 0.4 * lid) + _noise(gen, len(xf), 2) * (0.05 * lid)
    n = len(xf) + len(xw)
    zero = torch.zeros(n, dtype=torch.float64, device=DEV)
    return _pack(ph, xf, vf, xw, vw, torch.full((len(xf),), rho0 * dx * dx, dtype=torch.float64, device=DEV),
                 torch.full((len(xw),), 0.75 * rho0 * dx * dx, dtype=torch.float64, device=DEV),
                 zero + rho0, zero, zero[:len(xf)], zero[:len(xw)], h, dx, gen)


def _dam(ny, gen, dx=None, nx=None, options=0, alpha=0.01, c0=None, layers=3):
    """The dam break: a column of nx x ny particles in a tank four times as wide and half
    as high again, its origin in the column's middle; hydrostatic pressure and an impact's
    (a water hammer of rho c0 v inside the column, none at its edges)."""
    dx = 2.0 / ny if dx is None else dx
    nx = (ny + 1) // 2 if nx is None else nx
    h, rho0 = H_DX * dx, 1000.0
    w, top = nx * dx, ny * dx
    c0 = 10.0 * math.sqrt(2.0 * G * top) if c0 is None else c0
    ph = _physics(rho0=rho0, c0=c0, visc_artificial=1, av_alpha=alpha, av_beta=0.0, pmin=0.0,
                  gravity=(0.0, -G, 0.0), dt=0.1 * h / c0)
    if options:
        ph.update(density_form=2, average_velocity=1)
    ntx, nty = 4 * nx, (3 * ny) // 2
    lat = [_lattice((0, nx), (0, ny)), _lattice((-layers, ntx + layers), (-layers, 0)),
           _lattice((-layers, 0), (0, nty)), _lattice((ntx, ntx + layers), (0, nty))]
    mid = torch.tensor([0.5 * w, 0.5 * top], dtype=torch.float64, device=DEV)
    xf, xw = (lat[0] + 0.5) * dx - mid, (torch.cat(lat[1:]) + 0.5) * dx - mid
    x = torch.cat([xf, xw])
    s = [math.pi * (0.5 + x[:, 0] / w), math.pi * (0.5 + x[:, 1] / top)]
    inside = (x[:, 0].abs() < 0.5 * w) & (x[:, 1].abs() < 0.5 * top)
    p = rho0 * G * torch.clamp(0.5 * top - x[:, 1], min=0.0) * (x[:, 0] < 0.5 * w)
    p = p + inside * (0.25 * rho0 * c0 * c0) * torch.sin(s[0]) ** 2 * torch.sin(s[1]) ** 2
    rho = _tait_rho(p, rho0, c0)
    m = rho * dx * dx / _kernel_sum(2, H_DX)
    xf = _jitter(gen, xf, 0.15 * dx)
    nf, nw = len(xf), len(xw)
    vf = _swirl(xf, (-0.5 * w, -0.5 * top), (0.5 * w, 0.5 * top), 0.02 * c0) + _noise(gen, nf, 2) * (0.004 * c0)
    u = torch.full((nf,), 0.01 * c0 * c0, dtype=torch.float64, device=DEV)
    return _pack(ph, xf, vf, xw, torch.zeros_like(xw), m[:nf], m[nf:], rho, p, u,
                 torch.zeros(nw, dtype=torch.float64, device=DEV), h, dx, gen)


def _channel(n_x, n_yz, gen, layers=3):
    """The heated liquid-metal channel: periodic along x, walls on the four sides."""
    dx = 0.4 / 504
    h, rho0, c0, cp = H_DX * dx, 10500.0, 20.0, 146.0
    length, width = n_x * dx, n_yz * dx
    ph = _physics(dim=3, rho0=rho0, c0=c0, visc_artificial=1, heat_artificial=1, heat_external=1, av_alpha=0.02,
                  av_beta=0.0, ah_g1=0.1, ah_g2=0.1, heat_q0=1.0e8, heat_sigma=0.01,
                  heat_center=(0.25 * length, 0.5 * width, 0.5 * width), period=length, dt=0.2 * h / c0)
    lat = _lattice((0, n_x), (-layers, n_yz + layers), (-layers, n_yz + layers))
    ok = ((lat[:, 1:] >= 0) & (lat[:, 1:] < n_yz)).all(1)
    x = (lat + 0.5) * dx
    xf, xw = _jitter(gen, x[ok], 0.15 * dx), x[~ok]
    nf, n = len(xf), len(x)
    y = torch.sin(math.pi * xf[:, 1] / width) * torch.sin(math.pi * xf[:, 2] / width)
    p = 0.1 * rho0 * c0 * c0
    rho = _tait_rho(p, rho0, c0)
    m = torch.full((n,), rho * dx ** 3 / _kernel_sum(3, H_DX), dtype=torch.float64, device=DEV)
    vf = _noise(gen, nf, 3) * 0.1
    vf[:, 0] += y
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    return _pack(ph, xf, vf, xw, torch.zeros_like(xw), m[:nf], m[nf:], one * rho, one * p,
                 cp * (600.0 + _noise(gen, nf)), one[nf:] * (cp * 600.0), h, dx, gen)


def _gpuc_dam(scale, scheme, gen):
    """The GPU-C codes' dam break (published Tab.1 sizes at scales 1, 2, 4), moving, its origin in
    the column's middle, half the published time step."""
    dr, rho0, c0 = 0.02 / scale, 1000.0, 50.0
    nfx, nfy, ntx, nty = 100 * scale + 1, 50 * scale + 1, 269 * scale, 80 * scale
    ph = _physics(rho0=rho0, c0=c0, gravity=(0.0, -G, 0.0), scheme=scheme, dt=2.0e-4 / scale,
                  material=(4, (rho0, c0)))
    xf = _jitter(gen, (_lattice((0, nfx), (0, nfy)) + 0.5) * dr, 0.15 * dr)
    xw = torch.cat([_lattice((-3, ntx + 3), (-3, 0)), _lattice((-3, 0), (0, nty + 1)),
                    _lattice((ntx, ntx + 3), (0, nty + 1))]) * dr
    nf, n = len(xf), len(xf) + len(xw)
    mid = 0.5 * dr * torch.tensor([nfx, nfy], dtype=torch.float64, device=DEV)
    xf, xw, hi = xf - mid, xw - mid, mid.tolist()
    p = rho0 * G * torch.clamp(hi[1] - xf[:, 1], min=0.0)
    s = [0.5 * math.pi * (1.0 + xf[:, d] / hi[d]) for d in range(2)]
    p = p + 0.2 * rho0 * c0 * c0 * (torch.sin(s[0]) * torch.sin(s[1])) ** 2 * (1 + 0.1 * _noise(gen, nf))
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    rho, pp = one * rho0, one * 0.0
    rho[:nf], pp[:nf] = _tait_rho(p, rho0, c0), p
    vf = _swirl(xf, [-q for q in hi], hi, 1.0) + _noise(gen, nf, 2) * 0.5
    m = rho * dr * dr
    return _pack(ph, xf, vf, xw, torch.zeros_like(xw), m[:nf], m[nf:], rho, pp, one[:nf], one[nf:], 1.2 * dr, dr,
                 gen, wall_type=-1)


def _gpuc_wave(n_side, scheme, gen, size=0.1, radius=4.0e-3, e0=1400.0):
    """The pressure wave in mercury (published Tab.3 sizes at 401, 501, 601 a side)."""
    dr = size / (n_side - 1)
    rho0, c0, gamma = 13540.0, 1490.0, 1.96
    a1 = rho0 * c0 ** 2
    ph = _physics(rho0=rho0, c0=c0, scheme=scheme, dt=1.0e-4 / (2 * (n_side - 1)),
                  material=(2, (rho0, a1, 0.0, 0.0, gamma, 0.0, a1, 0.0)))
    x = _lattice((0, n_side), (0, n_side)) * dr - 0.5 * size
    n = len(x)
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    u = e0 * torch.exp(-(x * x).sum(1) / radius ** 2) + 20.0
    mu = 0.01 * torch.sin(60.0 * x[:, 0]) * torch.cos(60.0 * x[:, 1]) + 0.005 * _noise(gen, n)
    rho = rho0 * (1.0 + mu)
    p = a1 * mu + gamma * rho0 * u
    x = _jitter(gen, x, 0.1 * dr)
    v = 30.0 * _noise(gen, n, 2)
    none = x[:0]
    return _pack(ph, x, v, none, none, one * rho0 * dr * dr, one[:0], rho, p, u, one[:0], 1.2 * dr, dr, gen)


def _sweep(instances, layout, gen):
    """Alternating dam breaks and cavities of 2e3 to 2e5 particles, their own physics."""
    rng = random.Random(layout)
    out = []
    for k in range(instances):
        n = math.exp(rng.uniform(math.log(2.0e3), math.log(2.0e5)))
        alpha, c0, aspect = rng.uniform(0.005, 0.05), rng.uniform(20.0, 80.0), rng.uniform(0.5, 3.0)
        if k % 2 == 0:
            nx = max(4, int(round(math.sqrt(n / aspect))))
            out.append(_dam(max(4, int(round(aspect * nx))), gen, dx=1.0e-3, nx=nx, alpha=alpha, c0=c0))
        else:
            out.append(_cavity(max(4, int(round(math.sqrt(n)))), gen, length=1.0, lid=1.0, c0=c0, alpha=alpha))
    return out


def _systems(case, seed):
    gen = torch.Generator(DEV).manual_seed(int(seed))
    f = case["family"]
    if f == "cavity":
        return [_cavity(case["n_side"], gen)]
    if f in ("dam", "adjoint"):
        return [_dam(case["ny"], gen, options=case.get("options", 0))]
    if f == "channel":
        return [_channel(case["n_x"], case["n_yz"], gen)]
    if f == "gpuc_dam":
        return [_gpuc_dam(case["scale"], case["scheme"], gen)]
    if f == "gpuc_wave":
        return [_gpuc_wave(case["n_side"], case["scheme"], gen)]
    return _sweep(case["instances"], case["layout"], gen)


def _sensors(sy):
    """Cotangents of a linear observation: momentum along the flow, energy, pressure of a patch."""
    a = sy["arrays"]
    fl = a["itype"] > 0
    m = a["mass"] * fl
    near = torch.exp(-(a["x"].reshape(-1, 2) ** 2).sum(1) * 4.0)
    return {"v_bar": (m[:, None] * a["v"].reshape(-1, 2)).reshape(-1), "u_bar": m, "p_bar": 1.0e-3 * m * near}


ITS0 = 2  # the state carries the rates of an iteration before it


def prepare(case, seed):
    sys_ = _systems(case, seed)
    s0 = sys_[0]
    arrays = s0["arrays"] if len(sys_) == 1 else \
        {k: torch.cat([s["arrays"][k] for s in sys_]) for k in s0["arrays"]}
    host = case["call"] in ("host", "adjoint")
    sizes = [arrays[k].numel() for k, _ in MUTABLE]
    init = torch.cat([arrays[k] for k, _ in MUTABLE])
    work = torch.empty(init.shape, dtype=init.dtype, pin_memory=True) if host else torch.empty_like(init)
    call = dict(zip((k for k, _ in MUTABLE), work.split(sizes)))
    for k, _ in FIXED:
        call[k] = torch.empty(arrays[k].shape, dtype=arrays[k].dtype, pin_memory=True).copy_(arrays[k]) if host \
            else arrays[k]
    if host:
        call = {k: t.numpy() for k, t in call.items()}
    mem = ag.MEM_HOST if host else ag.MEM_DEVICE
    state = dict(case=case, init=init, work=work, arrays=call, dt=s0["ph"]["dt"])
    if case["call"] == "batch":
        ctx = ag.Batch([_params(s["ph"]) for s in sys_], [s["nf"] for s in sys_], [s["nw"] for s in sys_], mem=mem)
        ctx.set_tuning(case["reach"], 1, 128, 0)
        state["dt"] = [s["ph"]["dt"] for s in sys_]
    else:
        ctx = ag.Context(_params(s0["ph"]), s0["nf"], s0["nw"], mem=mem)
        ctx.set_tuning(case["reach"], case["tpp"], case["block"], case["skin"])
        if s0["ph"]["material"]:
            eos, prop = s0["ph"]["material"]
            ctx.set_materials([Material.make(eos, list(prop))] * 2)
    if case["call"] == "adjoint":
        state["bar"] = {k: t.cpu().numpy() for k, t in _sensors(s0).items()}
    state["ctx"] = ctx
    return state


def run(state):
    case, ctx, a = state["case"], state["ctx"], state["arrays"]
    state["work"].copy_(state["init"], non_blocking=True)
    if case["call"] in ("step", "host"):
        ctx.step(a, state["dt"], ITS0, wait=False)
    elif case["call"] == "run":
        ctx.integrate(a, state["dt"], ITS0, case["steps"], wait=False)
    elif case["call"] == "batch":
        ctx.integrate_batch(a, state["dt"], ITS0, case["steps"], wait=False)
    else:
        ctx.forward_checkpointed(a, state["dt"], ITS0, case["steps"], case["every"])
        g = ctx.backward(**state["bar"])
        return {"state": {k: a[k] for k, _ in MUTABLE}, "grad": {k: g[k] for k in ("x", "v", "u", "dvdt", "dudt")},
                "params": {k: g["params"][k] for k in ("av_alpha", "c0")}}
    return {k: a[k] for k, _ in MUTABLE}


def _counts(case):
    f = case["family"]
    if f == "cavity":
        return case["n_side"] ** 2 + 8 * case["n_side"]
    if f in ("dam", "adjoint"):
        ny, nx = case["ny"], (case["ny"] + 1) // 2
        return nx * ny + 3 * (4 * nx + 6) + 6 * ((3 * ny) // 2)
    if f == "channel":
        return case["n_x"] * (case["n_yz"] + 6) ** 2
    if f == "gpuc_dam":
        s = case["scale"]
        return (100 * s + 1) * (50 * s + 1) + 3 * (269 * s + 6) + 6 * (80 * s + 1)
    if f == "gpuc_wave":
        return case["n_side"] ** 2
    rng, n = random.Random(case["layout"]), 0
    for _ in range(case["instances"]):
        n += math.exp(rng.uniform(math.log(2.0e3), math.log(2.0e5)))
        for _ in range(3):
            rng.random()
    return int(n)


def work(case):
    """Bytes: the call's input and output arrays once each. Flops: the reference algorithm's
    own per particle and iteration (each pair once), RK3 three times, reverse mode with the
    forward, its replay and twice the forward's work for the adjoint."""
    dim = 3 if case["family"] == "channel" else 2
    n = _counts(case)
    out = 4.0 * n * (3 * dim + 4)
    per = 15700.0 if dim == 3 else 1920.0
    if case["family"] == "cavity":
        per = 2600.0
    if case["family"].startswith("gpuc"):
        per = 3 * 700.0
    if case["family"] == "adjoint":
        per *= 4.0
        out += 4.0 * n * 12
    return {"bytes": out + 4.0 * n * (3 * dim + 7), "flops": per * n * case.get("steps", 1)}


# ---- the step in 64 bits ---------------------------------------------------------

class _Cells:
    """Particles sorted by cells of twice the largest h, for the pair search."""

    def __init__(self, x, h, ph):
        dim, size = x.shape[1], 2.0 * float(h.max()) * (1.0 + 1e-9)
        self.period = ph["period"]
        lo = x.amin(0) - 1e-9
        n = (((x.amax(0) - lo) / size).floor().long() + 1).tolist()
        cell = torch.full((dim,), size, dtype=x.dtype, device=x.device)
        if self.period:
            n[0] = int(self.period // size)
            cell[0], lo[0] = self.period / n[0], 0.0
        self.n = n
        c = ((x - lo) / cell).floor().long()
        for d in range(dim):
            c[:, d].clamp_(0, n[d] - 1)
        key = c[:, 0].clone()
        for d in range(1, dim):
            key += c[:, d] * math.prod(n[:d])
        key, self.order = torch.sort(key, stable=True)
        self.c = c[self.order]
        self.start = torch.searchsorted(key, torch.arange(math.prod(n) + 1, device=x.device))

    def pairs(self, a, b, x, reach2):
        """Ordered pairs (i, j), i in [a, b), of the sorted x with |x_i - x_j|^2 < reach2(i, j)."""
        dim, found = x.shape[1], []
        slot = torch.arange(a, b, device=x.device)
        for off in torch.cartesian_prod(*([torch.arange(-1, 2)] * dim)).reshape(-1, dim).tolist():
            c = self.c[a:b] + torch.tensor(off, device=x.device)
            if self.period:
                c[:, 0] %= self.n[0]
            ok = torch.ones(b - a, dtype=torch.bool, device=x.device)
            key = torch.zeros(b - a, dtype=torch.long, device=x.device)
            for d in range(dim):
                ok &= (c[:, d] >= 0) & (c[:, d] < self.n[d])
                key += c[:, d].clamp(0, self.n[d] - 1) * math.prod(self.n[:d])
            first = self.start[key]
            cnt = torch.where(ok, self.start[key + 1] - first, 0)
            i = slot.repeat_interleave(cnt)
            j = torch.arange(len(i), device=x.device) + (first - cnt.cumsum(0) + cnt).repeat_interleave(cnt)
            d2 = (self.delta(x, i, j) ** 2).sum(1)
            keep = (d2 < reach2(i, j)) & (i != j)
            found.append((i[keep], j[keep]))
        return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])

    def delta(self, x, i, j):
        d = x[i] - x[j]
        if self.period:
            d0 = d[:, 0]
            d0 = d0 - self.period * torch.round(d0.detach() / self.period)
            d = torch.cat([d0[:, None], d[:, 1:]], 1)
        return d


def _sum_to(n, i, val):
    return torch.zeros((n,) + val.shape[1:], dtype=val.dtype, device=val.device).index_add(0, i, val)


def _ranges(n, dim):
    step = 1 << (20 if dim == 2 else 18)
    return [(a, min(a + step, n)) for a in range(0, n, step)]


def _kernel(d, hb, dim):
    """W and the factor gw of grad W = gw (x_i - x_j)."""
    r = (d * d).sum(1).sqrt()
    q = r / hb
    k = (7.0 / (4.0 * math.pi) if dim == 2 else 21.0 / (16.0 * math.pi)) / hb ** dim
    t = (1.0 - 0.5 * q).clamp(min=0.0)
    return k * t ** 4 * (1.0 + 2.0 * q), -5.0 * k / hb ** 2 * t ** 3


def _exact_cern(ph, dim, s, its, alpha=None, c0=None):
    """One leapfrog iteration of the CERN scheme (summation or normalised density) in 64 bits.
    s: x, v, a [n, dim], mass, rho, p, u, h, du [n], fluid; alpha, c0: tensors of the reverse mode."""
    f = {k: _f32(v) for k, v in ph.items() if isinstance(v, float)}
    c0 = f["c0"] if c0 is None else c0
    alpha = f["av_alpha"] if alpha is None else alpha
    dt, n = f["dt"], len(s["mass"])
    hdt, kdt = (0.0, 0.5 * dt) if its == 1 else (0.5 * dt, dt)
    cells = _Cells(s["x"].detach(), s["h"], ph)
    o = cells.order
    x, v, a, m, h, fl = (s[k][o] for k in ("x", "v", "a", "mass", "h", "fluid"))
    rho_in, p_in, u, du = (s[k][o] for k in ("rho", "p", "u", "du"))
    flv = fl[:, None]
    vh = torch.where(flv, v + hdt * a, v)
    uh = torch.where(fl, (u + hdt * du).clamp(min=0.0), u)
    xd = x.detach()

    def pairs(lo, hi):
        i, j = cells.pairs(lo, hi, xd, lambda i, j: (h[i] + h[j]) ** 2)
        d = cells.delta(x, i, j)
        hb = 0.5 * (h[i] + h[j])
        return (i, j, i - lo, d, hb) + _kernel(d, hb, dim)

    keep = [pairs(lo, hi) for lo, hi in _ranges(n, dim)] if n < 10_000_000 else None
    chunk = (lambda k, lo, hi: keep[k]) if keep else (lambda k, lo, hi: pairs(lo, hi))

    w0 = (7.0 / (4.0 * math.pi) if dim == 2 else 21.0 / (16.0 * math.pi)) / h ** dim
    rs, ns, ds = [], [], []
    for k, (lo, hi) in enumerate(_ranges(n, dim)):
        i, j, li, d, hb, w, gw = chunk(k, lo, hi)
        rs.append(_sum_to(hi - lo, li, m[j] * w))
        if ph["density_form"] == 2:
            ns.append(_sum_to(hi - lo, li, m[j] / rho_in[j] * w))
        if ph["heat_artificial"]:
            ds.append(_sum_to(hi - lo, li, m[j] * gw * ((vh[j] - vh[i]) * d).sum(1)))
    dens = m * w0 + torch.cat(rs)
    if ns:
        dens = dens / (m * w0 / rho_in + torch.cat(ns))
    rho0 = f["rho0"]
    e = dens / rho0 - 1.0
    p = rho0 * c0 ** 2 / 7.0 * ((1.0 + e) ** 7 - 1.0)
    clamp = p < ph["pmin"]
    rho = torch.where(fl, torch.where(clamp, torch.full_like(dens, rho0), dens), rho_in)
    p = torch.where(fl, torch.where(clamp, torch.zeros_like(p), p), p_in)
    pp = p / rho ** 2 if ph["pa_sph"] == 1 else p
    if ds:
        div = torch.cat(ds) / rho
        psi = f["ah_g1"] * h * c0 + f["ah_g2"] * h * h * (div.abs() - div)
    tau = None
    if ph["visc"]:
        ts = []
        for k, (lo, hi) in enumerate(_ranges(n, dim)):
            i, j, li, d, hb, w, gw = chunk(k, lo, hi)
            g, dv, c = gw[:, None] * d, vh[j] - vh[i], m[j] / rho[j]
            t = dv[:, :, None] * g[:, None, :]
            t = t + t.transpose(1, 2) - torch.eye(dim, dtype=t.dtype, device=t.device) * \
                (2.0 / 3.0 * (dv * g).sum(1))[:, None, None]
            ts.append(_sum_to(hi - lo, li, c[:, None, None] * t))
        tau = torch.cat(ts)
        tds = 0.5 * f["eta"] / rho * (tau * tau).sum((1, 2))
        tau = tau * (f["eta"] / rho ** 2 if ph["pa_sph"] == 1 else f["eta"])[:, None, None]
    acc, en, xs = [], [], []
    for k, (lo, hi) in enumerate(_ranges(n, dim)):
        i, j, li, d, hb, w, gw = chunk(k, lo, hi)
        g, dv, mj = gw[:, None] * d, vh[j] - vh[i], m[j]
        rb, vr = 0.5 * (rho[i] + rho[j]), (dv * d).sum(1)
        fs = -(pp[i] + pp[j])
        f_i = fs[:, None] * g
        if tau is not None:
            f_i = f_i + ((tau[i] + tau[j]) * g[:, None, :]).sum(2)
        if ph["pa_sph"] != 1:
            fs, f_i = fs / (rho[i] * rho[j]), f_i / (rho[i] * rho[j])[:, None]
        e_i = 0.5 * mj * fs * gw * vr
        if ph["visc_artificial"]:
            r2 = (d * d).sum(1)
            phi = torch.where(vr > 0, -hb * vr / (r2 + hb * hb * f["av_eta"] ** 2), torch.zeros_like(vr))
            pi = (f["av_beta"] * phi - alpha * c0) * phi / rb
            f_i = f_i - pi[:, None] * g
            e_i = e_i - 0.5 * mj * pi * gw * vr
        if ds:
            r2 = (d * d).sum(1)
            e_i = e_i + mj * (psi[i] + psi[j]) / (rb * (r2 + hb * hb * f["ah_eta"] ** 2)) * gw * r2 * (uh[i] - uh[j])
        acc.append(_sum_to(hi - lo, li, mj[:, None] * f_i))
        en.append(_sum_to(hi - lo, li, e_i))
        if ph["average_velocity"]:
            xs.append(_sum_to(hi - lo, li, (0.3 * mj * w / rb)[:, None] * dv))
    a_new = torch.cat(acc) + torch.tensor([_f32(g) for g in ph["gravity"][:dim]], dtype=x.dtype, device=x.device)
    du_new = torch.cat(en)
    if tau is not None:
        du_new = du_new + tds
    if ph["heat_external"]:
        hc = torch.tensor([_f32(c) for c in ph["heat_center"][:dim]], dtype=x.dtype, device=x.device)
        du_new = du_new + f["heat_q0"] * torch.exp(-((x - hc) ** 2).sum(1) / (2.0 * f["heat_sigma"] ** 2)) / rho
    a_new, du_new = a_new * flv, du_new * fl
    v_new = v + kdt * a_new
    if xs and its > 1:
        v_new = v_new + torch.cat(xs) * flv
    u_new = torch.where(fl, (u + kdt * du_new).clamp(min=0.0), u)
    x_new = torch.where(flv, x + dt * v_new, x)
    if ph["period"]:
        L = _f32(ph["period"])
        x_new = torch.cat([(x_new[:, :1].detach() % L) + (x_new[:, :1] - x_new[:, :1].detach()), x_new[:, 1:]], 1)
    back = torch.empty_like(o)
    back[o] = torch.arange(n, device=o.device)
    out = dict(x=x_new, v=v_new, rho=rho, p=p, u=u_new, a=a_new, du=du_new)
    return dict(s, **{k: t[back] for k, t in out.items()})


def _gpuc_eos(material, rho, u):
    eos, q = material[0], [_f32(v) for v in material[1]]
    rho = rho.clamp(min=0.9 * q[0])
    if eos == 4:
        return rho, q[0] * q[1] ** 2 / 7.0 * ((rho / q[0]) ** 7 - 1.0), torch.full_like(rho, q[1])
    mu = rho / q[0] - 1.0
    tension = q[6] * mu + q[7] * mu * mu + q[4] * q[0] * u
    press = q[1] * mu + q[2] * mu ** 2 + q[3] * mu ** 3 + (q[4] + q[5] * mu) * q[0] * u
    return rho, torch.where(mu < 0, tension, press), (q[1] / rho).sqrt()


def _exact_gpuc(ph, dim, s, its):
    """One TVD-RK3 step of the GPU-C schemes in 64 bits."""
    dt, n = _f32(ph["dt"]), len(s["mass"])
    cells = _Cells(s["x"], s["h"], ph)
    o = cells.order
    x0, v0, m, h = (s[k][o] for k in ("x", "v", "mass", "h"))
    rho0, u0, p, it = (s[k][o] for k in ("rho", "u", "p", "itype"))
    parts = [cells.pairs(lo, hi, x0, lambda i, j: (2.0 * h[i]) ** 2) for lo, hi in _ranges(n, dim)]
    i, j = (torch.cat([q[k] for q in parts]) for k in (0, 1))
    same, k0 = it[i] == it[j], 7.0 / (4.0 * math.pi)
    x, v, rho, u = x0, v0, rho0, u0
    c = _gpuc_eos(ph["material"], rho, u)[2]
    grav = torch.tensor([_f32(g) for g in ph["gravity"][:dim]], dtype=x.dtype, device=x.device) * (it > 0)[:, None]
    for al in (1.0, 0.25, 2.0 / 3.0):
        d = x[i] - x[j]
        r = (d * d).sum(1).sqrt()
        q = r / h[i]
        live = (r >= 0.01 * h[i])
        t = (1.0 - 0.5 * q).clamp(min=0.0)
        w = t ** 4 * (1.0 + 2.0 * q)  # over W(0)
        dw = -5.0 * q * t ** 3 * k0 / h[i] ** 3 * live
        dvr = (d * (v[i] - v[j])).sum(1)
        cs = 2.0 * c[i] / (rho[i] + rho[j])
        pair = same if ph["scheme"] == 2 else torch.ones_like(same)
        rd = _sum_to(n, i, m[j] * dw * (dvr / r + (rho[i] - rho[j]) * cs) * pair)
        pr = p[i] / rho[i] ** 2 + p[j] / rho[j] ** 2 if ph["scheme"] == 2 else (p[i] + p[j]) / (rho[i] * rho[j])
        shock = torch.where(dvr < 0, 0.03 * cs * dvr * h[i] / (0.01 * h[i] ** 2 + r * r), torch.zeros_like(r))
        f = m[j] * (shock - pr) * dw * pair
        if ph["scheme"] == 2:
            push = 0.5 * w * k0 / h[i] ** 2 * m[j] / (rho[j] * h[j]) * c[j] ** 2
        else:
            push = m[j] / (m[i] + m[j]) * 0.02 * w * c[i] * c[j] / r
        f = f + push * (~same & live)
        a = _sum_to(n, i, (f / r)[:, None] * d) + grav
        du = p * rd / rho ** 2
        x_n = x0 + al * (x + dt * v - x0)
        v_n = v0 + al * (v + dt * a - v0)
        rho_n = rho0 + al * (rho + dt * rd - rho0)
        u = u0 + al * (u + dt * du - u0)
        x, v = x_n, torch.where((it > 0)[:, None] | (ph["scheme"] == 2), v_n, v0)
        rho, p, c = _gpuc_eos(ph["material"], rho_n, u)
    back = torch.empty_like(o)
    back[o] = torch.arange(n, device=o.device)
    out = dict(x=x, v=v, rho=rho, p=p, u=u, a=a, du=du)
    return dict(s, **{k: t[back] for k, t in out.items()})


def exact(case, seed):
    systems = _systems(case, seed)
    if case["family"] == "gpuc_dam" and case["scheme"] == 2:
        return None  # its walls move under the push and leave the lattice: no well-conditioned value
    outs = []
    for sy in systems:
        ph, dim, a = sy["ph"], sy["dim"], sy["arrays"]
        s = {k: t.to(torch.float64) for k, t in a.items() if k != "itype"}
        for k in ("x", "v", "dvdt"):
            s[k] = s[k].reshape(-1, dim)
        s.update(a=s.pop("dvdt"), du=s.pop("dudt"), itype=a["itype"], fluid=a["itype"] > 0)
        ph = dict(ph, period=_f32(ph["period"]))
        if case["call"] == "adjoint":
            return _exact_adjoint(case, sy, ph, dim, s)
        step = _exact_gpuc if ph["scheme"] else _exact_cern
        for k in range(case.get("steps", 1)):
            s = step(ph, dim, s, ITS0 + k)
        outs.append(_layout(s))
    return {k: torch.cat([o[k] for o in outs]) for k in outs[0]}


def _layout(s):
    r = {k: s[k] for k in ("x", "v", "rho", "p", "u")}
    r.update(dvdt=s["a"], dudt=s["du"])
    return {k: r[k].detach().reshape(-1) for k, _ in MUTABLE}


def _exact_adjoint(case, sy, ph, dim, s):
    bar = {k: t.to(torch.float64) for k, t in _sensors(sy).items()}
    par = [torch.tensor(_f32(ph[k]), dtype=torch.float64, device=DEV, requires_grad=True) for k in ("av_alpha", "c0")]
    ins = {k: s[k].clone().requires_grad_() for k in ("x", "v", "u", "a", "du")}
    q = dict(s, **ins)
    for k in range(case["steps"]):
        q = _exact_cern(ph, dim, q, ITS0 + k, *par)
    loss = (q["v"].reshape(-1) * bar["v_bar"]).sum() + (q["u"] * bar["u_bar"]).sum() + (q["p"] * bar["p_bar"]).sum()
    g = torch.autograd.grad(loss, list(ins.values()) + par, allow_unused=True)
    out = {}
    for (name, t), d in zip(ins.items(), g):
        d = torch.zeros_like(t) if d is None else d.clone()
        d[~s["fluid"]] = 0.0  # walls are not integrated: the reverse mode returns zero for them
        out[dict(a="dvdt", du="dudt").get(name, name)] = d.reshape(-1)
    return {"state": _layout(q), "grad": out, "params": {"av_alpha": g[5].reshape(()), "c0": g[6].reshape(())}}
