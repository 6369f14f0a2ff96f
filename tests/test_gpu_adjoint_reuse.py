"""Reverse mode on a context that has run before: its results are those of a fresh
context, to the bit (every sum of the reverse mode has a fixed order).

* The parameters turn physics on (or off) between two forward/backward pairs: the
  buffers of the new physics are there, and none of the old tape is left in use.
* backward after a forward whose parameters have changed since is refused.
"""
import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases

pytestmark = pytest.mark.gpu

STEPS, EVERY = 4, 2


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _case(dim):
    if dim == 2:
        return cases.perturbed(cases.dam_break(dx=0.05), seed=101, dv=0.1, du=1.0)
    c = cases.perturbed(cases.channel(n_x=14, n_yz=6, length=0.1, width=0.04, jitter=0.05), seed=102, dv=0.05,
                        du=10.0)
    c.params.heat_artificial = 0
    return c


def _cotangents(c):
    rng = np.random.default_rng(103)
    return dict(x_bar=rng.standard_normal(c.n * c.dim), v_bar=rng.standard_normal(c.n * c.dim),
                u_bar=rng.standard_normal(c.n), p_bar=1e-4 * rng.standard_normal(c.n))


def _reverse(ctx, c):
    s = c.copy()
    ctx.forward_checkpointed(s, c.dt, 1, STEPS, EVERY)
    return s, ctx.backward(**_cotangents(c))


def _fresh(c, tuning=None):
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        if tuning:
            ctx.set_tuning(*tuning)
        return _reverse(ctx, c)


def _same(a, b):
    for f in ("x", "v", "rho", "p", "u", "dvdt", "dudt"):
        assert np.array_equal(getattr(a[0], f), getattr(b[0], f)), f
    for k in ("x", "v", "u", "dvdt", "dudt"):
        assert np.isfinite(b[1][k]).all(), k
        assert np.array_equal(a[1][k], b[1][k]), k
    assert a[1]["params"] == b[1]["params"]


PHYSICS = {"visc": dict(visc=1, eta=1e-2), "heat": dict(heat_artificial=1),
           "both": dict(visc=1, eta=1e-2, heat_artificial=1)}


@pytest.mark.parametrize("physics", list(PHYSICS))
@pytest.mark.parametrize("dim", [2, 3])
def test_physics_turned_on_and_off_between_calls(dim, physics):
    c = _case(dim)
    d = c.copy()
    for k, v in PHYSICS[physics].items():
        d.params.set(k, v)
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        first = _reverse(ctx, c)
        ctx.set_params(d.params)
        on = _reverse(ctx, d)
        ctx.set_params(c.params)
        off = _reverse(ctx, c)
    _same(on, _fresh(d))
    _same(first, off)
    _same(off, _fresh(c))


def test_backward_needs_a_forward_of_the_present_parameters():
    c = _case(2)
    d = c.copy()
    d.params.av_alpha = 0.5
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        s = c.copy()
        ctx.forward_checkpointed(s, c.dt, 1, STEPS, EVERY)
        ctx.set_params(d.params)
        with pytest.raises(ag.ArmandoError):
            ctx.backward(**_cotangents(c))
        s = d.copy()
        ctx.forward_checkpointed(s, d.dt, 1, STEPS, EVERY)
        ctx.set_params(d.params)  # the same values again
        got = (s, ctx.backward(**_cotangents(d)))
    _same(got, _fresh(d))
