"""Calls of one context whose state buffers have swapped roles since an earlier call
with the same time step: the results are those of a fresh context, to the bit.

* The fused predictor swaps two buffers on every iteration of a call with a skin and
  lists; reverse mode in between runs without it.
* An open run compacts the particles into a second buffer on every step.
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


def _cotangents(c):
    rng = np.random.default_rng(111)
    return dict(x_bar=rng.standard_normal(c.n * c.dim), v_bar=rng.standard_normal(c.n * c.dim))


def _integrate(ctx, c, steps):
    s = c.copy()
    ctx.integrate(s, c.dt, 1, steps)
    return {f: getattr(s, f) for f in FIELDS}


def _reverse(ctx, c):
    s = c.copy()
    ctx.forward_checkpointed(s, c.dt, 1, 4, 2)
    g = ctx.backward(**_cotangents(c))
    return {**{f: getattr(s, f) for f in FIELDS}, **{"bar_" + k: g[k] for k in ("x", "v", "u", "dvdt", "dudt")}}


def _same(a, b):
    for f in b:
        assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("tuning", [(2, 1, 128, 10), (1, 1, 256, 20)])
def test_integrate_and_reverse_mode_alternate(tuning):
    c = cases.perturbed(cases.dam_break(dx=0.05), seed=110, dv=0.1)

    def fresh(f, *args):
        with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
            ctx.set_tuning(*tuning)
            return f(ctx, c, *args)

    rev, run3, run4 = fresh(_reverse), fresh(_integrate, 3), fresh(_integrate, 4)
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(*tuning)
        for steps in (3, 3, 4, 3, 1, 4):
            got = _integrate(ctx, c, steps)
            if steps != 1:
                _same(got, run3 if steps == 3 else run4)
            _same(_reverse(ctx, c), rev)


@pytest.mark.parametrize("skin", [0, 10])
@pytest.mark.parametrize("steps", [1, 2, 3])
def test_integrate_after_an_open_run(steps, skin):
    c = cases.gpuc_dam_break(scale=1, fluid=(20, 10), tank=(50, 20))
    x = c.x.reshape(-1, 2)
    box = (x.min(0) - 0.5 * c.h[0], x.max(0) + 0.5 * c.h[0])  # (no more cells than the first call's)
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(2, 1, 128, skin)
        want = _integrate(ctx, c, 4)
        ctx.set_open_boundaries([], [], box)
        a = {k: v.copy() for k, v in c.arrays().items()}
        assert ctx.integrate_open(a, c.dt, 1, steps, c.n) == c.n
        _same(_integrate(ctx, c, 4), want)
