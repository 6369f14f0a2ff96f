"""A sort skin on a GPU-C context when the device has no room for neighbour lists: the
tuning is taken, and the steps are those of a context without lists, to the bit.
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


def _fill(torch, leave):
    """Allocations (never written) that leave less than `leave` bytes of the device free."""
    held = []
    chunk = torch.cuda.mem_get_info()[0]
    while torch.cuda.mem_get_info()[0] >= leave and chunk >= (2 << 20):
        try:
            held.append(torch.empty(min(chunk, torch.cuda.mem_get_info()[0]), dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            chunk //= 2
    assert torch.cuda.mem_get_info()[0] < leave
    return held


def test_skin_without_room_for_lists(monkeypatch):
    torch = pytest.importorskip("torch")
    c = cases.gpuc_dam_break(scale=8)
    tuning = (2, 1, 128, 10)
    monkeypatch.setenv("ARMANDO_NEIGHBOUR_LISTS", "0")
    want = c.copy()
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.set_tuning(*tuning)
        ctx.integrate(want, c.dt, 1, 3)
    monkeypatch.delenv("ARMANDO_NEIGHBOUR_LISTS")
    got = c.copy()
    with ag.Context(c.params, c.n_fluid, c.n_wall) as ctx:
        ctx.step(c.copy(), c.dt, 1)
        held = _fill(torch, leave=288 * c.n // 2)  # 288 bytes of lists a particle
        try:
            ctx.set_tuning(*tuning)
        finally:
            held.clear()
            torch.cuda.empty_cache()
        ctx.integrate(got, c.dt, 1, 3)
    for f in FIELDS:
        assert np.array_equal(getattr(got, f), getattr(want, f)), f
