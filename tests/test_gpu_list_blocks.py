"""How k_build_list stores a list: in blocks of entries, near ones first, shifted
particles for the rows across a periodic end.

One iteration on the lists against one FP64 oracle iteration (1e-5, normwise
relative, every output): patches whose lists hold a few up to more entries than
fit (one, two and three times the lattice's density; skins of 10, 40 and 100%),
and boxes periodic in x, y and (3D) z with particles on both ends.
"""
import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from helpers import FIELDS, step_errors
from test_gpu_lists import _with_extra_copies

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _check(O, c, tuning):
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(*tuning)
        errs, _, _ = step_errors(O, ctx, c, its=1)
    for f in FIELDS:
        assert errs[f] <= 1e-5, (f, errs[f])


@pytest.mark.parametrize("skin", [10, 40, 100])
@pytest.mark.parametrize("offsets", [[], [0.33], [0.5], [0.33, 0.66]], ids=["x1", "x2", "x2b", "x3"])
def test_lists_up_to_and_beyond_their_capacity(O, offsets, skin):
    c = cases.perturbed(cases.dam_break(dx=0.02, jitter=0.05), seed=92, dv=0.05)
    fl = np.flatnonzero(c.itype > 0)
    x = c.x.reshape(-1, 2)
    patch = fl[np.argsort(np.linalg.norm(x[fl] - x[fl[len(fl) // 2]], axis=1))[:60]]
    _check(O, _with_extra_copies(c, patch, offsets), (1, 1, 128, skin))


def _box(dim, axes):
    """A jittered lattice that fills a box of the given periodic axes."""
    n = (23, 17, 13)[:dim]
    h = 0.01
    dx = h / 1.2
    rng = np.random.default_rng(93)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, dim)
    c = cases.perturbed(cases.channel(n_x=27, n_yz=11, length=27 * 7.9e-4, width=11 * 7.9e-4, layers=3)
                        if dim == 3 else cases.cavity(n_side=23), seed=94)
    m = len(g)
    c.x = ((g + 0.5 + rng.uniform(-0.1, 0.1, g.shape)) * dx).astype(np.float32)
    c.x[0, 0] = 0.0
    c.x = c.x.ravel()
    c.v = rng.normal(0.0, 0.01, m * dim).astype(np.float32)
    c.dvdt = np.zeros(m * dim, np.float32)
    c.mass = np.full(m, 1000.0 * dx ** dim, np.float32)
    c.rho = np.full(m, 1000.0, np.float32)
    c.h = np.full(m, h, np.float32)
    c.itype = np.where(np.arange(m) < m - 3, np.abs(c.itype[0]), -np.abs(c.itype[0])).astype(c.itype.dtype)
    c.p, c.u, c.dudt = (np.zeros(m, np.float32) for _ in range(3))
    for a in range(3):
        c.params.periodic[a] = int(a in axes)
        c.params.period_lo[a], c.params.period_hi[a] = 0.0, (n[a] * dx if a < dim else 0.0)
    c.params.heat_external = 0
    c.params.rho0 = 1000.0
    c.dt = 1e-6
    return c


@pytest.mark.parametrize("skin", [10, 60])
@pytest.mark.parametrize("dim,axes", [(2, (0,)), (2, (1,)), (2, (0, 1)), (3, (0,)), (3, (1, 2)), (3, (0, 1, 2))])
def test_lists_across_periodic_ends(O, dim, axes, skin):
    _check(O, _box(dim, axes), (1, 1, 128, skin))
