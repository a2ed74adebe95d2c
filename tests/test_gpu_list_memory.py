"""The DFSPH and PCISPH solvers keep kernel factors or gradients beside the list
entries where the GPU has room for them, and compute the same values again where
it has not: with the same operations, so the tolerance is zero. A limit on the
context's memory, one byte below what it takes with them, stands in for a GPU
that is full.
"""
import ctypes as C

import numpy as np
import pytest

from sph2o_b200 import scenes as S
from sph2o_b200.api import Batch, Scene, Simulation, lib

pytestmark = pytest.mark.gpu
CAPACITY = 64


def scene_of(method, dims, r=0.02):
    ext = [2 * r * k for k in dims]
    return Scene.from_dict(S.scene(
        method=method, radius=r, blocks=[S.block(dims, r, (2 * r,) * 3)],
        tank=((0, 0, 0), (ext[0] + 8 * r, ext[1] + 8 * r, ext[2] + 8 * r)), time_step=5e-4 if method == S.DFSPH else 2e-4,
        jitter=0.3, seed=dims[0]))


def held(sim, limit=0):
    out = C.c_size_t()
    assert lib().sph_debug_limit_memory(sim._h, limit, C.byref(out)) == 0
    return out.value


def both_ways(build, monkeypatch):
    """(sim with everything kept, sim with nothing kept), and the bytes between them."""
    full = build()
    limit, init = held(full) - 1, lib().sph_init

    def limited_init(h):
        assert lib().sph_debug_limit_memory(h, limit, None) == 0
        return init(h)

    with monkeypatch.context() as m:
        m.setattr(lib(), "sph_init", limited_init)
        small = build()
    return full, small, held(full) - held(small)


def stirred(n, seed):
    return np.random.default_rng(seed).uniform(-0.5, 0.5, (n, 3)).astype(np.float32)


# 105 particles; 9,000; 67,032 (two lanes below 2^16 particles, one above)
@pytest.mark.parametrize("dims", [(7, 5, 3), (30, 20, 15), (57, 42, 28)])
@pytest.mark.parametrize("method", [S.PCISPH, S.DFSPH])
def test_steps_without_kept_values(method, dims, monkeypatch):
    sc = scene_of(method, dims)
    x = sc.fluid()[0]
    *sims, saved = both_ways(lambda: Simulation(sc.desc(), x, sc.boundary()), monkeypatch)
    assert saved == (len(x) + 31) // 32 * 32 * CAPACITY * 16
    got = []
    for sim in sims:
        sim.set_state(x, stirred(len(x), 3))
        st = sim.step(3)
        sim.set_state(None, stirred(len(x), 4))
        st2 = sim.step(2)
        got.append((*sim.state(), st["total_iterations"], st["total_iterations_v"], st2["total_iterations"]))
        sim.close()
    for kept, again in zip(*got):
        assert np.array_equal(kept, again)


def test_batch_without_kept_values(monkeypatch):
    scenes = [scene_of(S.DFSPH, d) for d in ((7, 5, 3), (12, 10, 9), (20, 11, 8))]
    *sims, saved = both_ways(lambda: Batch(scenes), monkeypatch)
    assert saved > 0
    for sim in sims:
        sim.step(4)
    for s in range(len(scenes)):
        for kept, again in zip(*[sim.scene_state(s) for sim in sims]):
            assert np.array_equal(kept, again)


def test_scene_without_boundary_keeps_no_boundary_factors(monkeypatch):
    sc = scene_of(S.DFSPH, (12, 10, 9))
    x = sc.fluid()[0]
    *sims, saved = both_ways(lambda: Simulation(sc.desc(), x, np.zeros((0, 3), np.float32)), monkeypatch)
    assert saved == ((len(x) + 31) // 32 * 32 * CAPACITY + 1) * 8
    for sim in sims:
        sim.set_state(x, stirred(len(x), 3))
        sim.step(3)
    for kept, again in zip(*[sim.state() for sim in sims]):
        assert np.array_equal(kept, again)
