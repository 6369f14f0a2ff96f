"""The force pass with av_eta = ah_eta = 0 (no lower bound of the art_visc and art_heat
quotients) at ordinary and at low densities, against one FP64 oracle iteration
(1e-5, normwise relative, every output), on the cells and on lists, with artificial
viscosity on and off (its quotient is formed either way).

The low densities are the same systems with every mass, density and pressure scaled
by 2^-17 and 2^-27. Particles in the same place as another one have r = 0 in a real
pair, not only where a lane's list has ended.
"""
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


def _case(dim, scale, av, coincident):
    if dim == 2:
        c = cases.perturbed(cases.dam_break(dx=0.04, jitter=0.1), seed=131, dv=0.1)
    else:
        c = cases.perturbed(cases.channel(n_x=16, n_yz=8, length=16 * 7.9e-4, width=8 * 7.9e-4, layers=2,
                                          jitter=0.1), seed=132, dv=0.05, du=200.0)
    s = np.float32(2.0 ** scale)
    for f in ("mass", "rho", "p"):
        setattr(c, f, getattr(c, f) * s)
    for f in ("rho0", "heat_q0"):
        c.params.set(f, getattr(c.params, f) * float(s))
    c.params.visc_artificial, c.params.av_beta = av, 0.3
    c.params.av_eta = 0.0
    # art_heat of a pair at r = 0 is 0/0 in the written formula without its eta
    c.params.ah_eta = 0.1 if coincident else 0.0
    if coincident:
        fl = np.flatnonzero(c.itype > 0)
        x = c.x.reshape(-1, dim)
        x[fl[5::50]] = x[fl[4::50][:len(fl[5::50])]]
    return c


@pytest.mark.parametrize("coincident", [False, True], ids=["apart", "coincident"])
@pytest.mark.parametrize("av", [0, 1])
@pytest.mark.parametrize("scale", [0, -17, -27])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("tuning", [(1, 1, 128, 0), (2, 1, 128, 10), (1, 2, 128, 0)])
def test_step_without_eta(O, tuning, dim, scale, av, coincident):
    c = _case(dim, scale, av, coincident)
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(*tuning)
        errs, got, _ = step_errors(O, ctx, c, its=1)
    for f in FIELDS:
        assert np.isfinite(getattr(got, f)).all() and errs[f] <= 1e-5, (f, errs[f])
