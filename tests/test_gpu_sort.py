"""The counting sort of the particles by cell (k_cell_count ... k_cell_rank).

The neighbour sets it yields must be link_list's exactly: for particle counts
around a CTA's 256, grids of one scan tile (8,192 cells) and of several, with
cell counts at a tile's edge and mostly empty cells, a clump that fills one cell,
and repeated runs (the order within a cell does not depend on the counters'
timing). A batch with an instance that has no grid reports it and ends.
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


def _points(x, h):
    """Fluid particles at x (k x 2) with the dam break's physics."""
    c = cases.dam_break(dx=0.1)
    n = len(x)
    c.x = np.ascontiguousarray(x, np.float32).ravel()
    c.v, c.dvdt = np.zeros(2 * n, np.float32), np.zeros(2 * n, np.float32)
    c.h = np.full(n, h, np.float32)
    c.mass = np.full(n, 1000.0 * (h / 1.3) ** 2, np.float32)
    c.rho = np.full(n, 1000.0, np.float32)
    c.p, c.u, c.dudt = (np.zeros(n, np.float32) for _ in range(3))
    c.itype = np.ones(n, np.int32)
    c.dt = 0.2 * h / float(c.params.c0)
    return c


def _rows(O, c):
    pi, pj, _, _ = O.link_list(c.x, c.h, c.dim, fp32=True, params=c.params)
    a, b = np.concatenate([pi, pj]), np.concatenate([pj, pi])
    o = np.lexsort((b, a))
    return np.concatenate([[0], np.cumsum(np.bincount(a, minlength=c.n))]), b[o].astype(np.int32)


def _check(O, c, reach=1):
    offs, nbr = _rows(O, c)
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(reach=reach)
        got_offs, got = ctx.neighbours(c.x, c.h)
        again = ctx.neighbours(c.x, c.h)
    assert np.array_equal(got_offs, offs) and np.array_equal(got, nbr)
    assert np.array_equal(again[0], offs) and np.array_equal(again[1], nbr)


@pytest.mark.parametrize("n", [3, 255, 256, 257, 1000])
def test_counts_around_a_cta(O, n):
    rng = np.random.default_rng(n)
    _check(O, _points(rng.random((n, 2)) * np.sqrt(n) * 0.01, 0.013))


@pytest.mark.parametrize("cells", [8190, 8191, 8192, 8193, 16384, 60000])
@pytest.mark.parametrize("reach", [1, 3])
def test_scan_tiles(O, cells, reach):
    """`cells` cells of 2 h in one row, particles in clusters far apart and in the
    last cells."""
    h = 0.5
    rng = np.random.default_rng(cells + reach)
    # bounding box expanded by h: cells = floor((span + 2 h) / (2 h)) + 1
    span = (cells - 1.5) * 2 * h
    at = np.concatenate([[0.0, span], rng.choice(cells - 4, 40) + 1.3])
    x = np.concatenate([a + rng.random(7) * 1.5 for a in at])
    x = np.concatenate([[0.0, span], np.clip(x, 0.0, span)])
    _check(O, _points(np.stack([x, rng.random(len(x)) * 0.4], 1), h), reach)


def test_clump_in_one_cell(O):
    rng = np.random.default_rng(5)
    x = np.concatenate([rng.random((700, 2)) * 0.005, rng.random((50, 2)) * 0.3])
    _check(O, _points(x, 0.013))


def test_repeated_runs_are_the_same_bits():
    c = cases.perturbed(cases.dam_break(dx=0.01), seed=91, dv=0.2)
    outs = []
    for _ in range(3):
        s = c.copy()
        with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
            ctx.integrate(s, c.dt, 1, 4)
        outs.append(s)
    for s in outs[1:]:
        for f in FIELDS:
            assert np.array_equal(getattr(s, f), getattr(outs[0], f)), f


def test_batch_instance_without_a_grid():
    """A periodic box shorter than three cells in one instance of a batch."""
    insts = [cases.dam_break(dx=0.05), cases.cavity(n_side=12), cases.dam_break(dx=0.05)]
    bad = insts[1].params
    bad.set("periodic", (1, 0, 0))
    bad.set("period_lo", (0.0, 0.0, 0.0))
    bad.set("period_hi", (float(insts[1].h[0]), 0.0, 0.0))
    arrays, _ = cases.pack(insts)
    with ag.Batch([c.params for c in insts], [c.n_fluid for c in insts],
                  [c.n_wall for c in insts]) as b:
        with pytest.raises(ag.ArmandoError):
            b.integrate_batch(arrays, [c.dt for c in insts], 1, 2)
