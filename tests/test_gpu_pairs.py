"""The neighbour passes' pair arithmetic, two entries at a time (csrc/pair2.cuh).

With every particle's h alike the passes take the h factors as constants; one
differing h (here: one ulp, on one wall particle) takes the general form. Both,
in cells and in lists, against one FP64 oracle iteration at the one-step gate
1e-5 (normwise relative, every output), in 2D and 3D, with odd neighbour counts
(jittered, at free surfaces and walls), with and without physical viscosity and
artificial heat, across a coordinate's zero and a periodic end, and with
coincident particles, whose pair has no direction and adds no force.
"""
import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from helpers import FIELDS, history_state, rel_err, step_errors

pytestmark = pytest.mark.gpu

TOL_STEP = 1e-5


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _dam(shift=0.0):
    c = cases.perturbed(cases.dam_break(dx=0.02, jitter=0.1), seed=81, dv=0.1)
    c.x = (c.x - np.float32(shift)).astype(np.float32)
    c.params.av_beta = 0.4
    return c


def _cavity():
    c = cases.perturbed(cases.cavity(n_side=23, jitter=0.1), seed=82, dv=2e-4)
    c.params.visc_artificial, c.params.av_alpha = 1, 0.1
    return c


def _channel():
    return cases.perturbed(cases.channel(n_x=27, n_yz=11, length=27 * 7.9e-4, width=11 * 7.9e-4,
                                         layers=3, jitter=0.1), seed=83, dv=0.05, du=50.0)


CASES = {"dam": _dam, "dam_centred": lambda: _dam(0.5), "cavity": _cavity, "channel": _channel}


def _check(O, c, tuning):
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(*tuning)
        errs, _, _ = step_errors(O, ctx, c, its=3)
    for f in FIELDS:
        assert errs[f] <= TOL_STEP, (tuning, f, errs[f])


@pytest.mark.parametrize("tuning", [(1, 1, 128, 0), (3, 1, 256, 0), (2, 1, 128, 10)])
@pytest.mark.parametrize("alike", [True, False], ids=["h_alike", "h_differs"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_pair_terms_parity(O, name, alike, tuning):
    c = CASES[name]()
    if not alike:
        c.h[-1] = np.nextafter(c.h[-1], np.float32(0.0))
    _check(O, history_state(O, c, steps=2), tuning)


@pytest.mark.parametrize("tuning", [(1, 1, 128, 0), (3, 1, 128, 10)])
def test_coincident_particles(O, tuning):
    """Two fluid particles at one place, moving apart: no force between them, the
    kernel's maximum in their densities."""
    c = _dam()
    fl = np.flatnonzero(c.itype > 0)
    i, j = fl[len(fl) // 2], fl[len(fl) // 2 + 1]
    x = c.x.reshape(-1, 2)
    x[j] = x[i]
    ref = O.State(c)
    O.step(ref, 1, c.dt)
    got = c.copy()
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(*tuning)
        ctx.step(got, c.dt, 1)
    for f in FIELDS:
        assert rel_err(getattr(got, f), getattr(ref, f)) <= TOL_STEP, f
