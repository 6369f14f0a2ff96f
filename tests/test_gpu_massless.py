"""Fluid particles without mass and without mass near them (no density: their pressure
over density squared is infinite) that share their warps with ordinary ones. They have
no pairs, so they fall freely: one iteration against one FP64 oracle iteration (1e-5,
normwise relative, every output), on the cells, staged, on lists, with several lanes a
particle and with the options that are finite for such a particle.
"""
import os

import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from helpers import FIELDS, step_errors

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _case(dim):
    if dim == 2:
        c = cases.perturbed(cases.dam_break(dx=0.04, jitter=0.1), seed=141, dv=0.1)
        side = 1
    else:
        c = cases.perturbed(cases.channel(n_x=16, n_yz=8, length=16 * 7.9e-4, width=8 * 7.9e-4, layers=2,
                                          jitter=0.1), seed=142, dv=0.05, du=200.0)
        c.params.heat_artificial = c.params.heat_external = 0
        c.params.set("periodic", (0, 0, 0))
        side = 0
    c.params.pmin = -np.inf
    # every seventh fluid particle of the last column, drawn out of it and without mass
    x = c.x.reshape(-1, dim)
    fl = np.flatnonzero(c.itype > 0)
    last = fl[x[fl, 0] > x[fl, 0].max() - 0.5 * c.meta["dx"]]
    out = last[3::7] if dim == 2 else last[::9]  # (above the floor walls' reach)
    x[out, 0] = x[fl, 0].max() + 5.0 * c.h[0] * (1 + np.arange(len(out)))
    if side == 0:
        x[out, 1] = x[last[len(last) // 2], 1]
    c.mass[out] = 0.0
    return c


def _check(O, c, tuning):
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(*tuning)
        errs, got, _ = step_errors(O, ctx, c, its=1)
    assert (got.rho[(c.itype > 0) & (c.mass == 0)] == 0).all()
    for f in FIELDS:
        assert np.isfinite(getattr(got, f)).all() and errs[f] <= 1e-5, (f, errs[f])


@pytest.mark.parametrize("option", [{}, {"average_velocity": 1}, {"wall_model": 2}, {"pa_sph": 0},
                                    {"heat_artificial": 1}, {"av_eta": 0.0}],
                         ids=lambda o: "_".join(f"{k}{v:g}" for k, v in o.items()) or "lean")
@pytest.mark.parametrize("tuning", [(1, 1, 128, 0), (2, 1, 256, 0), (2, 1, 128, 20), (1, 2, 128, 0), (1, 4, 128, 0)])
@pytest.mark.parametrize("dim", [2, 3])
def test_lone_particles_without_mass(O, dim, tuning, option):
    c = _case(dim)
    for k, v in option.items():
        c.params.set(k, v)
    _check(O, c, tuning)


@pytest.mark.parametrize("dim", [2, 3])
def test_lone_particles_without_mass_staged(O, dim, monkeypatch):
    monkeypatch.setenv("ARMANDO_STAGING", "1")
    _check(O, _case(dim), (1, 1, 128, 0))
