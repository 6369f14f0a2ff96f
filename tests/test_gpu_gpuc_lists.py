"""The GPU-C schemes' stages on the neighbour lists of a lazily sorting context
against the same stages walking the cells: the same pairs (the candidate test is
exact in both), so the two agree within the gates that the schemes are held to
(normwise relative; pressure and what follows from it carry the density's last
bit, 0.15 Pa at rho = 1000 and c0 = 50 m/s).

Cases: 2D and 3D, both schemes, over steps that sort and steps that do not; block
sizes; and a patch at two and three times the lattice's density, whose lists have
more than 32 entries and more than fit, beside listed particles.
"""
import os

import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from test_gpu_gpuc import TOL, rel
from test_gpu_lists import _with_extra_copies

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _dam(scheme):
    c = cases.gpuc_dam_break(1, fluid=(40, 20), tank=(110, 34), scheme=scheme)
    rng = np.random.default_rng(90 + scheme)
    v = c.v.reshape(-1, 2)
    v[c.itype > 0] = rng.normal(0.0, 0.05, size=(c.n_fluid, 2))
    c.v = v.ravel().astype(np.float32)
    return c


def _patch(scheme, offsets):
    c = _dam(scheme)
    fl = np.flatnonzero(c.itype > 0)
    x = c.x.reshape(-1, 2)
    patch = fl[np.argsort(np.linalg.norm(x[fl] - x[fl[len(fl) // 2]], axis=1))[:100]]
    return _with_extra_copies(c, patch, offsets)


def _block(scheme):
    c = cases.channel(n_x=14, n_yz=6, length=14 * 7.9e-4, width=6 * 7.9e-4, layers=2, jitter=0.01)
    c.params.scheme = scheme
    c.params.periodic[:] = (0, 0, 0)
    c.params.heat_external = 0
    return c


CASES = {"dam": _dam, "block": _block,
         "twofold": lambda s: _patch(s, [0.33]), "threefold": lambda s: _patch(s, [0.33, 0.66])}


@pytest.mark.parametrize("tuning,steps", [((1, 1, 128, 20), 1), ((2, 1, 256, 40), 4)])
@pytest.mark.parametrize("scheme", [1, 2])
@pytest.mark.parametrize("name", sorted(CASES))
def test_stage_lists_match_the_cell_walk(name, scheme, tuning, steps):
    if name not in ("dam", "block"):
        steps = 1
    c = CASES[name](scheme)
    out = {}
    old = os.environ.get("ARMANDO_NEIGHBOUR_LISTS")
    try:
        for lists in ("1", "0"):
            os.environ["ARMANDO_NEIGHBOUR_LISTS"] = lists
            got = c.copy()
            with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
                ctx.set_tuning(*tuning)
                ctx.integrate(got, c.dt, 1, steps)
            out[lists] = got
    finally:
        if old is None:
            del os.environ["ARMANDO_NEIGHBOUR_LISTS"]
        else:
            os.environ["ARMANDO_NEIGHBOUR_LISTS"] = old
    fl = c.itype > 0
    for f, g in (("x", "x"), ("v", "v"), ("rho", "rho"), ("p", "p"), ("u", "u"), ("dvdt", "dv"), ("dudt", "du")):
        a = getattr(out["1"], f).reshape(c.n, -1)[fl]
        b = getattr(out["0"], f).reshape(c.n, -1)[fl]
        assert np.isfinite(b).all(), f
        assert rel(a, b) <= TOL[g], (f, rel(a, b))
