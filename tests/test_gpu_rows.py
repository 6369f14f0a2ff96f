"""The cell walk by rows (density, shear and force passes, one lane a particle).

One iteration against one FP64 oracle iteration (1e-5, normwise relative, every
output) where a lane leaves its candidate lists off full and goes on, where a
particle's neighbour bits are more than one list or one word of a row holds, and
where rows continue across a periodic end: patches at up to six times the
lattice's density, every reach, with and without physical viscosity, and boxes
periodic along one axis or all.
"""
import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from helpers import FIELDS, step_errors
from test_gpu_list_blocks import _box
from test_gpu_lists import _with_extra_copies

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _check(O, c, reach, block):
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(reach, 1, block, 0)
        errs, _, _ = step_errors(O, ctx, c, its=1)
    for f in FIELDS:
        assert errs[f] <= 1e-5, (f, errs[f])


@pytest.mark.parametrize("visc", [0, 1])
@pytest.mark.parametrize("reach", [1, 2, 3])
@pytest.mark.parametrize("copies", [1, 2, 3, 6])
def test_full_lists_and_words(O, copies, reach, visc):
    c = cases.perturbed(cases.dam_break(dx=0.02, jitter=0.05), seed=96, dv=0.05)
    if visc:
        c.params.visc, c.params.eta = 1, 1e-3
    fl = np.flatnonzero(c.itype > 0)
    x = c.x.reshape(-1, 2)
    patch = fl[np.argsort(np.linalg.norm(x[fl] - x[fl[len(fl) // 2]], axis=1))[:60]]
    _check(O, _with_extra_copies(c, patch, [k / copies for k in range(1, copies)]), reach, 128)


@pytest.mark.parametrize("reach", [1, 3])
@pytest.mark.parametrize("dim,axes", [(2, (0,)), (2, (1,)), (2, (0, 1)), (3, (0,)), (3, (0, 1, 2))])
def test_rows_across_periodic_ends(O, dim, axes, reach):
    _check(O, _box(dim, axes), reach, 256)
