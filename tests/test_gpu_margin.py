"""Entries of a neighbour list beyond the support (the sort skin's margin) whose
state is not finite.

A wall particle without mass and without mass near it has no density, so its
pressure over density squared is not finite. Within the support such a particle
has none of its own (the neighbour's mass is there); in the margin, between 2h
and 2h + skin from a fluid particle, it is on that particle's list and adds
nothing: the run with lists stays finite and agrees with the cell walk to 1e-5
(one iteration, normwise relative, every output).
"""
import os

import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from helpers import FIELDS, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _with_empty_wall(c):
    """c and a massless wall particle 2.05 h above its topmost fluid particle, the
    other fluid particles 0.01 h lower."""
    x = c.x.reshape(-1, c.dim).copy()
    fl = np.flatnonzero(c.itype > 0)
    top = fl[np.argmax(x[fl, 1])]
    rest = fl[fl != top]
    x[rest, 1] = np.minimum(x[rest, 1], x[top, 1] - np.float32(0.01) * c.h[0])
    add = x[top].copy()
    add[1] += np.float32(2.05) * c.h[0]
    out = c.copy()
    out.x = np.concatenate([x, add[None]]).ravel().astype(np.float32)
    for f in ("v", "dvdt"):
        a = getattr(c, f).reshape(-1, c.dim)
        setattr(out, f, np.concatenate([a, np.zeros((1, c.dim), np.float32)]).ravel())
    wall = np.flatnonzero(c.itype <= 0)[0]
    for f in ("mass", "rho", "p", "u", "h", "itype", "dudt"):
        a = getattr(c, f)
        setattr(out, f, np.concatenate([a, a[wall:wall + 1]]))
    out.mass[-1] = out.rho[-1] = 0.0
    return out


def _run(c, lists, its):
    old = os.environ.get("ARMANDO_NEIGHBOUR_LISTS")
    os.environ["ARMANDO_NEIGHBOUR_LISTS"] = "1" if lists else "0"
    try:
        out = c.copy()
        with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
            ctx.set_tuning(2, 1, 128, 20)
            ctx.integrate(out, c.dt, its, 1)
        return out
    finally:
        if old is None:
            del os.environ["ARMANDO_NEIGHBOUR_LISTS"]
        else:
            os.environ["ARMANDO_NEIGHBOUR_LISTS"] = old


@pytest.mark.parametrize("option", [{}, {"visc": 1, "eta": 1e-3}, {"visc": 1, "eta": 1e-3, "pa_sph": 0},
                                    {"heat_artificial": 1}, {"density_form": 1}, {"density_form": 2},
                                    {"wall_model": 2}],
                         ids=lambda o: "_".join(f"{k}{v:g}" for k, v in o.items()) or "lean")
def test_margin_entry_without_density(option):
    c = cases.perturbed(cases.dam_break(dx=0.02, jitter=0.1), seed=91, dv=0.1)
    for k, val in option.items():
        c.params.set(k, val)
    c = _with_empty_wall(c)
    a, b = _run(c, True, 3), _run(c, False, 3)
    fl = c.itype > 0
    for f in FIELDS:
        u, w = getattr(a, f).reshape(c.n, -1)[fl], getattr(b, f).reshape(c.n, -1)[fl]
        assert np.isfinite(u).all(), f
        assert rel_err(u, w) <= 1e-5, (f, rel_err(u, w))
