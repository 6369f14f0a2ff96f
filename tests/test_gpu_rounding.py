"""The passes' packed division, reciprocal and square root (pair2.cuh) on random operands.

* div2, rcp2_rn and sqrt2 against CUDA's correctly rounded __fdiv_rn, __frcp_rn and
  __fsqrt_rn: equal, or one ulp apart where the exact value is within 2^-19 ulp of a tie.
  (rcp.approx is off by 2^-23, rsqrt.approx by 2^-22.4, and the product that starts a
  quotient or root by 2^-24 more; the correction leaves the square of that, at most
  2^-43.9 of the value or 2^-19.9 ulp.)
* recip_ff2: the rounded reciprocal and its residual, off by the residual's square and by
  the rounding of the low part, 2^-48 each: 2^-47.
* sqrt_ff2: one Newton correction of a root off by at most 2^-22: half its square, 2^-45,
  and roundings of the low part that add up to less than as much: 2^-44.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 20


@pytest.fixture(scope="module")
def helpers(tmp_path_factory):
    here = os.path.dirname(os.path.abspath(__file__))
    so = str(tmp_path_factory.mktemp("pair2") / "pair2_driver.so")
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O3", "-gencode",
                    "arch=compute_103a,code=sm_103a", "-Xcompiler", "-fPIC", "-shared", "-o", so,
                    os.path.join(here, "pair2_driver.cu")], check=True)
    lib = C.CDLL(so)

    def run(what, a, b):
        a, b = (np.ascontiguousarray(q, np.float32) for q in (a, b))
        out = np.zeros(2 * a.size, np.float32)
        assert lib.run_helpers(what, *[C.c_void_p(q.ctypes.data) for q in (a, b)], a.size,
                               C.c_void_p(out.ctypes.data)) == 0
        return out[:a.size], out[a.size:]

    return run


def _operands(seed, spread):
    rng = np.random.default_rng(seed)
    m = 1.0 + rng.random((2, N))
    return (m * 2.0 ** rng.integers(-spread, spread + 1, (2, N))).astype(np.float32)


@pytest.mark.parametrize("spread", [0, 30])
@pytest.mark.parametrize("what,exact", [(0, lambda a, b: a / b), (1, lambda a, b: 1.0 / b),
                                        (2, lambda a, b: np.sqrt(a))], ids=["div2", "rcp2_rn", "sqrt2"])
def test_rounded_like_ieee(helpers, what, exact, spread):
    a, b = _operands(151 + what, spread)
    got, want = helpers(what, a, b)
    off = np.flatnonzero(got != want)
    ulp = np.spacing(want[off]).astype(np.float64)
    assert (np.abs(got[off].astype(np.float64) - want[off]) <= ulp).all()
    v = exact(a[off].astype(np.float64), b[off].astype(np.float64)) / ulp
    assert (np.abs(v - np.floor(v) - 0.5) <= 2.0 ** -19).all(), off.size


def test_float_float_reciprocal(helpers):
    a, b = _operands(161, 30)
    hi, lo = helpers(3, a, b)
    # 1 - a (hi + lo), exact products in the longer type
    a, hi, lo = (q.astype(np.longdouble) for q in (a, hi, lo))
    assert np.abs(1 - a * hi - a * lo).max() <= 2.0 ** -47


def test_float_float_square_root(helpers):
    a, b = _operands(162, 30)
    low = (np.spacing(a) * 0.49 * np.sin(b)).astype(np.float32)
    hi, lo = (q.astype(np.longdouble) for q in helpers(4, a, low))
    want = np.sqrt(a.astype(np.longdouble) + low)
    assert np.abs((hi + lo - want) / want).max() <= 2.0 ** -44
