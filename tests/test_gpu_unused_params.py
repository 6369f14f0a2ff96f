"""Parameters of physics that is switched off play no part, whatever they hold: one step
with every such float undefined or infinite against one with the defaults, to the bit.
"""
import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from helpers import FIELDS

pytestmark = pytest.mark.gpu

UNUSED = {"visc_artificial": ("av_alpha", "av_beta", "av_eta"), "heat_artificial": ("ah_g1", "ah_g2", "ah_eta"),
          "visc": ("eta",), "heat_external": ("heat_q0", "heat_sigma")}


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("on", [(), ("heat_artificial",), ("visc",), ("visc_artificial", "heat_artificial")],
                         ids=lambda o: "_".join(o) or "none")
@pytest.mark.parametrize("tuning", [(1, 1, 128, 0), (2, 1, 128, 20), (1, 2, 128, 0)])
@pytest.mark.parametrize("dim", [2, 3])
def test_parameters_of_what_is_off(dim, tuning, on, value):
    out = []
    for bad in (False, True):
        if dim == 2:
            c = cases.perturbed(cases.dam_break(dx=0.04, jitter=0.1), seed=191, dv=0.1, du=1.0)
        else:
            c = cases.perturbed(cases.channel(n_x=16, n_yz=8, length=16 * 7.9e-4, width=8 * 7.9e-4, layers=2,
                                              jitter=0.1), seed=192, dv=0.05, du=50.0)
        for k in UNUSED:
            c.params.set(k, 1 if k in on else 0)
        if "visc" in on:
            c.params.eta = 1e-3
        for k, names in UNUSED.items():
            for name in names if bad and k not in on else ():
                c.params.set(name, value)
        with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
            ctx.set_tuning(*tuning)
            ctx.step(c, c.dt, 2)
        out.append(c)
    for f in FIELDS:
        a, b = (getattr(c, f) for c in out)
        assert np.isfinite(b).all() and np.array_equal(a, b), f
