"""The cell walk by rows in 3D with full candidate lists and words: one iteration
against one FP64 oracle iteration (1e-5, normwise relative, every output) of a channel
section with patches at one to three times the lattice's density (70 to 220 neighbours,
up to 1,400 candidates: a lane leaves its lists off full many times, and its bits exceed
what the words hold), every reach, with and without physical viscosity, cells and lists.
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


def _dense_patch(c, copies):
    x = c.x.reshape(-1, 3)
    fl = np.flatnonzero(c.itype > 0)
    idx = fl[np.argsort(np.linalg.norm(x[fl] - x[fl[len(fl) // 2]], axis=1))[:120]]
    rep = np.concatenate([np.arange(c.n)] + [idx] * (copies - 1))
    out = c.copy()
    for f in ("mass", "rho", "p", "u", "h", "itype", "dudt"):
        setattr(out, f, getattr(c, f)[rep])
    for f in ("x", "v", "dvdt"):
        setattr(out, f, getattr(c, f).reshape(-1, 3)[rep].copy())
    for k in range(1, copies):
        part = slice(c.n + (k - 1) * len(idx), c.n + k * len(idx))
        out.x[part] += np.float32(k / copies * c.meta["dx"])
    for f in ("x", "v", "dvdt"):
        setattr(out, f, np.ascontiguousarray(getattr(out, f).ravel()))
    return out


@pytest.mark.parametrize("visc", [0, 1])
@pytest.mark.parametrize("reach,skin", [(1, 0), (2, 0), (3, 0), (1, 40)])
@pytest.mark.parametrize("copies", [1, 2, 3])
def test_full_lists_and_words_3d(O, copies, reach, skin, visc):
    c = cases.perturbed(cases.channel(n_x=16, n_yz=10, length=16 * 7.9e-4, width=10 * 7.9e-4, layers=2, jitter=0.05),
                        seed=171, dv=0.05, du=50.0)
    if visc:
        c.params.visc, c.params.eta = 1, 1e-3
    c = _dense_patch(c, copies)
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(reach, 1, 128, skin)
        errs, _, _ = step_errors(O, ctx, c, its=1)
    for f in FIELDS:
        assert errs[f] <= 1e-5, (f, errs[f])
