"""What follows a neighbour list that outgrew its capacity: the step that meets
it reports the overflow, the capacity grows, and the next step runs on complete
lists. A context whose lists are built once more from the same positions before
that step (by a change of the cell order and back) is the reference: the same
lists in the same order, so the tolerance is zero. Where there is no room for
what has to be allocated (a limit on the context's memory stands in for a full
GPU), the call reports it, the context keeps its state, and once there is room
it goes on like one that never met the limit.
"""
import ctypes as C

import numpy as np
import pytest

from sph2o_b200 import api
from sph2o_b200 import scenes as S
from sph2o_b200.api import Scene, Simulation, SphError, lib

pytestmark = pytest.mark.gpu
NONE = np.zeros((0, 3), np.float32)
OVERFLOW, NO_MEMORY = -4, -2


def block_of(method, dims=(14, 13, 12), r=0.02):
    ext = [2 * r * k for k in dims]
    sc = Scene.from_dict(S.scene(
        method=method, radius=r, blocks=[S.block(dims, r, (2 * r,) * 3)],
        tank=((0, 0, 0), (ext[0] + 8 * r, ext[1] + 8 * r, ext[2] + 8 * r)), time_step=5e-4, jitter=0.3, seed=3))
    return sc.desc(), sc.fluid()[0]


def limit_memory(sim, limit):
    """Sets the limit (0: none); the bytes that the context holds."""
    held = C.c_size_t()
    assert lib().sph_debug_limit_memory(sim._h, limit, C.byref(held)) == 0
    return held.value


def overflowing(desc, x, squeeze, limit=None, code=OVERFLOW):
    """A context whose last step met more neighbours (74 at 0.82, 78 at 0.8) than its lists hold (64)."""
    sim = Simulation(desc, x, NONE)
    if limit is not None:
        if limit == "held":
            # all but what DFSPH and PCISPH keep beside their list entries, which
            # would make room for longer lists
            beside = {S.WCSPH: 0, S.PCISPH: 16, S.DFSPH: 8}[desc.simulation_method]
            limit = limit_memory(sim, 0) - (len(x) + 31) // 32 * 32 * 64 * beside
        limit_memory(sim, limit)
    sim.set_state((np.float32(0.1) + x * np.float32(squeeze)).astype(np.float32), np.zeros_like(x))
    with pytest.raises(SphError) as e:
        sim.step(1)
    assert e.value.code == code
    return sim


@pytest.mark.parametrize("method", [S.WCSPH, S.PCISPH, S.DFSPH])
@pytest.mark.parametrize("squeeze", [0.82, 0.8])
def test_step_after_the_capacity_has_grown(method, squeeze):
    desc, x = block_of(method)
    got = []
    for rebuilt in (False, True):
        sim = overflowing(desc, x, squeeze)
        if rebuilt:
            sim.set_option(api.OPT_CELL_ORDER, 1)
            sim.set_option(api.OPT_CELL_ORDER, 0)
        sim.step(1)
        got.append(sim.state())
        sim.close()
    for grown, again in zip(*got):
        assert np.array_equal(grown, again)


@pytest.mark.parametrize("method", [S.WCSPH, S.PCISPH, S.DFSPH])
@pytest.mark.parametrize("limit", ["held", 1])
def test_no_room_to_grow(method, limit):
    """With the limit at the bytes held by lists and state the lists keep their
    capacity; with one byte not even these can be had again."""
    desc, x = block_of(method)
    still = np.zeros_like(x)
    got = []
    for full in (False, True):
        sim = overflowing(desc, x, 0.82, limit if full else None, NO_MEMORY if full else OVERFLOW)
        before = sim.state()
        if full and limit == 1:
            for call in (lambda: sim.step(1), sim.neighbors, lambda: sim.phase(api.PHASE_DENSITY),
                         lambda: sim.set_state(x, still), lambda: sim.set_option(api.OPT_CELL_ORDER, 1),
                         lambda: sim.autotune(1)):
                with pytest.raises(SphError) as e:
                    call()
                assert e.value.code == NO_MEMORY
            for a, b in zip(before, sim.state()):
                assert np.array_equal(a, b)
            limit_memory(sim, 0)
            sim.set_option(api.OPT_CELL_ORDER, 0)
        sim.set_state(x, still)
        sim.step(2)
        got.append(sim.state())
        sim.close()
    for roomy, limited in zip(*got):
        assert np.array_equal(roomy, limited)


def test_adjoint_where_each_allocation_fails():
    desc, x = block_of(S.WCSPH)
    target = x + np.float32(0.01)
    got = []
    for full in (False, True):
        sim = Simulation(desc, x, NONE)
        held = limit_memory(sim, 0)
        failures, limit = 0, held
        while full:
            limit_memory(sim, limit)
            try:
                sim.wcsph_forward(4, target, ckpt_every=2)
                break
            except SphError as e:
                assert e.code == NO_MEMORY
                failures += 1
                limit += 16 * len(x)
        assert failures > 10 or not full
        sim.set_state(x, np.zeros_like(x))
        loss = sim.wcsph_forward(4, target, ckpt_every=2)
        got.append((loss, *sim.wcsph_backward(want_x0=True).values()))
        sim.close()
    for roomy, limited in zip(*got):
        assert np.array_equal(roomy, limited)
