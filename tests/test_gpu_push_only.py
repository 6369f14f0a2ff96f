"""wall_model 1, where the push is the only interaction of particles of different type:
the pressure, velocity and energy that a wall carries play no part. Walls where these are
infinite or not a number: the fluid's results are those of walls with none, to the bit, on
the cells and on lists.
"""
import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from helpers import FIELDS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _case(dim, p):
    if dim == 2:
        c = cases.perturbed(cases.dam_break(dx=0.04, jitter=0.1), seed=181, dv=0.1)
    else:
        c = cases.perturbed(cases.channel(n_x=16, n_yz=8, length=16 * 7.9e-4, width=8 * 7.9e-4, layers=2,
                                          jitter=0.1), seed=182, dv=0.05, du=50.0)
    c.params.wall_model = 1
    c.p[c.itype <= 0] = p
    return c


@pytest.mark.parametrize("p", [np.nan, np.inf])
@pytest.mark.parametrize("tuning", [(1, 1, 128, 0), (2, 1, 128, 20), (1, 2, 128, 0)])
@pytest.mark.parametrize("dim", [2, 3])
def test_wall_pressure_plays_no_part(dim, tuning, p):
    out = []
    for q in (0.0, p):
        c = _case(dim, q)
        with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
            ctx.set_tuning(*tuning)
            ctx.step(c, c.dt, 1)
        out.append(c)
    fl = out[0].itype > 0
    for f in FIELDS:
        a, b = (getattr(c, f).reshape(c.n, -1)[fl] for c in out)
        assert np.isfinite(b).all() and np.array_equal(a, b), f


@pytest.mark.parametrize("option", [{}, {"visc": 1, "eta": 1e-3}, {"heat_artificial": 1}, {"average_velocity": 1},
                                    {"visc": 1, "eta": 1e-3, "pa_sph": 0, "heat_artificial": 1}],
                         ids=lambda o: "_".join(f"{k}{v:g}" for k, v in o.items()) or "lean")
@pytest.mark.parametrize("tuning", [(1, 1, 128, 0), (2, 1, 128, 20), (1, 2, 128, 0)])
@pytest.mark.parametrize("dim", [2, 3])
def test_wall_velocity_and_energy_play_no_part(dim, tuning, option):
    out = []
    for q in (0.0, np.nan):
        c = _case(dim, q)
        c.params.heat_artificial = 0
        for k, v in option.items():
            c.params.set(k, v)
        wall = c.itype <= 0
        c.v.reshape(-1, dim)[wall] = q
        c.u[wall] = q
        with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
            ctx.set_tuning(*tuning)
            ctx.step(c, c.dt, 1)
        out.append(c)
    fl = out[0].itype > 0
    for f in FIELDS:
        a, b = (getattr(c, f).reshape(c.n, -1)[fl] for c in out)
        assert np.isfinite(b).all() and np.array_equal(a, b), f
