"""Reverse mode where a lane's neighbour list ends before the other lanes' of its warp.

* A pair's gradients do not depend on which particles share its warp: isolated pairs
  alone, and with clusters beyond their reach between them, to the bit.
* art_visc and art_heat without their eta terms (av_eta = ah_eta = 0), where the
  quotients have no lower bound: one iteration against the FP64 tangent-linear at the
  reverse mode's gate (test_gpu_adjoint.py).
"""
import numpy as np
import pytest

import armando_gb300 as ag
from armando_gb300 import cases
from test_gpu_adjoint import TOL_ONE, _gpu_all, _tangent_all, adjoint_case, gpu_gradients, heat_case, spec_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from armando_gb300 import build

    build.build_library()
    ag.load_library()


def _pairs(dim, clusters, physics):
    """16 pairs of particles 12 h apart along x, with or without a cluster midway."""
    h, dx, m = 0.01, 0.008, 16
    rng = np.random.default_rng(121)
    a = np.zeros((2 * m, 3))
    a[::2, 0] = 0.12 * np.arange(m)
    a[1::2] = a[::2] + np.array([0.011, 0.003, 0.002])
    v, u = rng.normal(0.0, 0.1, (2 * m, 3)), rng.normal(0.0, 1.0, 2 * m)
    if clusters:
        k = np.arange(5) - 2
        g = np.stack(np.meshgrid(k, k, k if dim == 3 else [0], indexing="ij"), -1).reshape(-1, 3) * dx
        b = np.concatenate([g + np.array([0.12 * q + 0.06, 0.0, 0.0]) for q in range(m - 1)])
        a = np.concatenate([a, b + rng.uniform(-0.1, 0.1, b.shape) * dx])
        v = np.concatenate([v, rng.normal(0.0, 0.1, b.shape)])
        u = np.concatenate([u, rng.normal(0.0, 1.0, len(b))])
    n = len(a)
    P = ag.Params.default(dim=dim, visc_artificial=1, av_beta=0.3, rho0=1000.0, c0=10.0, **physics)
    f32 = lambda q: np.ascontiguousarray(q, np.float32)
    return cases.Case("pairs", P, dim, f32(a[:, :dim]).ravel(), f32(v[:, :dim]).ravel(),
                      f32(np.full(n, 1000.0 * dx ** dim)), f32(np.full(n, 1000.0)), f32(np.zeros(n)), f32(u),
                      f32(np.full(n, h)), np.ones(n, np.int32), dt=1e-5, steps=1)


@pytest.mark.parametrize("physics", [{}, {"visc": 1, "eta": 1e-2}, {"heat_artificial": 1}],
                         ids=["lean", "visc", "heat"])
@pytest.mark.parametrize("dim", [2, 3])
def test_gradients_do_not_depend_on_the_warp(dim, physics):
    out = []
    for clusters in (False, True):
        c = _pairs(dim, clusters, physics)
        s = c.copy()
        with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
            ctx.forward_checkpointed(s, c.dt, 1, 1, 1)
            g = ctx.backward(x_bar=np.full(c.n * dim, 0.3), v_bar=np.full(c.n * dim, 0.7), u_bar=np.full(c.n, 0.1))
        out.append(g)
    for k, w in (("x", dim), ("v", dim), ("u", 1), ("dvdt", dim), ("dudt", 1)):
        a, b = out[0][k], out[1][k][:len(out[0][k])]
        assert np.isfinite(a).all() and np.array_equal(a, b), (k, np.abs(a - b).max(), np.abs(a).max())


@pytest.mark.parametrize("dim", [2, 3])
def test_art_heat_without_eta(O, dim):
    c = heat_case(dim)
    c.params.ah_eta = 0.0
    _, g = gpu_gradients(c, spec_for(O), K=1, steps=1)
    got, ref = _gpu_all(c, g), _tangent_all(O, c, 1)
    for k in ref:
        assert abs(got[k] - ref[k]) <= TOL_ONE * abs(ref[k]), (k, got[k], ref[k])


def test_art_visc_without_eta(O):
    c = adjoint_case()
    c.params.av_eta = 0.0
    _, g = gpu_gradients(c, spec_for(O), K=1, steps=1)
    got, ref = _gpu_all(c, g), _tangent_all(O, c, 1)
    for k in ref:
        assert abs(got[k] - ref[k]) <= TOL_ONE * abs(ref[k]), (k, got[k], ref[k])
