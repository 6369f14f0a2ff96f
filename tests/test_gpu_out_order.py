"""Calls on both sides of the sizes at which their form changes: from 131,072
particles on outputs are written in the caller's order (armando.cu,
kGatherOutMin), above 262,144 a lazily sorting call's first step sorts inside
the conditional node like the later ones (kFirstPlainMax).

Two particles alone in a gap carry a system of one less over the size: they
interact with nobody and lie inside its bounds, so the grid, the order of every
sum and each output of the others stay the same to the bit.
"""
import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "rho", "p", "u", "dvdt", "dudt")
SIZES = {131071: (0.004, 131), 262143: (0.0028, 190)}  # dam dx, channel n_x


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _pick(c, idx):
    out = c.copy()
    for f in ("x", "v", "dvdt"):
        setattr(out, f, np.ascontiguousarray(getattr(c, f).reshape(-1, c.dim)[idx]).ravel())
    for f in ("mass", "rho", "p", "u", "h", "itype", "dudt"):
        setattr(out, f, np.ascontiguousarray(getattr(c, f)[idx]))
    return out


def _case(dim, below):
    """`below` particles around a gap, and two wall particles inside it."""
    dx, n_x = SIZES[below]
    if dim == 2:
        c = cases.perturbed(cases.dam_break(dx=dx, jitter=0.1), seed=95, dv=0.1)
    else:
        c = cases.perturbed(cases.channel(n_x=n_x, n_yz=33, length=n_x * 7.9e-4, width=33 * 7.9e-4,
                                          layers=3, jitter=0.01), seed=95, dv=0.02)
        c.params.periodic[:] = (0, 0, 0)
    x = c.x.reshape(-1, dim)
    fl = np.flatnonzero(c.itype > 0)
    centre = x[fl].mean(axis=0)
    d = np.linalg.norm(x - centre, axis=1)
    d[c.itype <= 0] = np.inf
    keep = np.sort(np.argsort(-d, kind="stable")[:below])
    few = _pick(c, keep)
    wall = np.flatnonzero(few.itype <= 0)[:2]
    many = _pick(few, np.concatenate([np.arange(below), wall]))
    y = many.x.reshape(-1, dim)
    y[-2:] = centre.astype(np.float32)
    y[-1, 0] += np.float32(0.5) * c.h[0]
    gap = np.linalg.norm(few.x.reshape(-1, dim) - centre, axis=1).min()
    assert gap > 4.0 * c.h.max()
    return few, many


def _run(c, call):
    import torch

    dev = {f: torch.from_numpy(getattr(c, f).copy()).cuda() for f in
           ("x", "v", "mass", "rho", "p", "u", "h", "itype", "dvdt", "dudt")}
    with ag.Context(c.params, c.n_fluid, c.n_wall, mem=ag.MEM_DEVICE) as ctx:
        if call == "run":
            ctx.set_tuning(2, 1, 128, 10)
            ctx.integrate(dev, c.dt, 1, 2)
        else:
            ctx.step(dev, c.dt, 3)
    return {f: dev[f].cpu().numpy() for f in FIELDS}


@pytest.mark.parametrize("call", ["step", "run"])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("below", sorted(SIZES))
def test_outputs_alike_on_both_sides(below, dim, call):
    few, many = _case(dim, below)
    a, b = _run(few, call), _run(many, call)
    for f in FIELDS:
        u, w = a[f].reshape(below, -1), b[f].reshape(below + 2, -1)[:below]
        assert np.array_equal(u, w), f
