"""Forms of one computation that have to agree bit for bit, because they do the
same FP32 operations in the same order: the DFSPH neighbour passes with one and
two lanes per particle (list lengths on every remainder of a round, walls
included), their records after an upload of velocities alone, a division by h
that is replaced by a checked product, PCISPH densities with more accepted
candidates than a lane keeps, and the allocation-free densities of a cluster
denser than a lane's batch. The tolerance is therefore zero, against the CPU
oracle where the other form is not in the library (a PCISPH step: 1e-5 of the
positions, the bar of its accelerations).
"""
import ctypes as C

import numpy as np
import pytest

from oracle.oracle import Oracle
from sph2o_b200 import api
from sph2o_b200 import scenes as S
from sph2o_b200.api import Scene, Simulation, lib

pytestmark = pytest.mark.gpu
NONE = np.zeros((0, 3), np.float32)


def scene_of(method, dims, r=0.02):
    ext = [2 * r * k for k in dims]
    return Scene.from_dict(S.scene(
        method=method, radius=r, blocks=[S.block(dims, r, (2 * r,) * 3)],
        tank=((0, 0, 0), (ext[0] + 8 * r, ext[1] + 8 * r, ext[2] + 8 * r)), time_step=5e-4, jitter=0.3, seed=dims[0]))


def stirred(n, seed):
    return np.random.default_rng(seed).uniform(-0.5, 0.5, (n, 3)).astype(np.float32)


# 105 particles; 9,000; 67,032 (one lane by itself, fewer below 2^16 take two)
@pytest.mark.parametrize("dims", [(7, 5, 3), (30, 20, 15), (57, 42, 28)])
@pytest.mark.parametrize("occupancy", [4, 8])
def test_dfsph_lanes_agree(dims, occupancy):
    sc = scene_of(S.DFSPH, dims)
    desc, x, b = sc.desc(), sc.fluid()[0], sc.boundary()
    got = []
    for lanes in (1, 2):
        sim = Simulation(desc, x, b)
        sim.set_option(api.OPT_SOLVER_OCCUPANCY, occupancy)
        sim.set_option(api.OPT_SOLVER_LANES, lanes)
        sim.set_state(x, stirred(len(x), 3))
        st = sim.step(3)
        got.append((*sim.state(), st["total_iterations"], st["total_iterations_v"]))
        sim.close()
    for one, two in zip(*got):
        assert np.array_equal(one, two)


@pytest.mark.parametrize("dims", [(7, 5, 3), (30, 20, 15)])
def test_dfsph_velocities_alone(dims):
    sc = scene_of(S.DFSPH, dims)
    desc, x, b = sc.desc(), sc.fluid()[0], sc.boundary()
    v = stirred(len(x), 4)
    got = []
    for uploads in ([(x, v)], [(x, -v), (None, v)]):
        sim = Simulation(desc, x, b)
        for u in uploads:
            sim.set_state(*u)
        sim.step(2)
        got.append(sim.state())
        sim.close()
    for full, alone in zip(*got):
        assert np.array_equal(full, alone)


@pytest.mark.parametrize("r", [0.0123, 0.017, 0.02500001, 0.0499, 0.1, 0.3333333, 1.7])
def test_densities_for_any_support_radius(r):
    sc = scene_of(S.PCISPH, (9, 8, 7), r)
    desc, x, b = sc.desc(), sc.fluid()[0], sc.boundary()
    sim, o = Simulation(desc, x, b), Oracle(desc, x, b)
    assert np.array_equal(sim.phase(api.PHASE_DENSITY), o.phase(0).astype(np.float32))
    sim.close()
    o.close()


# up to 41, 50 and 58 neighbours, around the 44 candidates that a lane keeps
@pytest.mark.parametrize("squeeze", [0.95, 0.9, 0.87])
def test_pcisph_step_of_squeezed_fluid(squeeze):
    sc = scene_of(S.PCISPH, (14, 13, 12))
    desc, x, b = sc.desc(), sc.fluid()[0], sc.boundary()
    x = (np.float32(0.1) + x * np.float32(squeeze)).astype(np.float32)
    sim, o = Simulation(desc, x, NONE), Oracle(desc, x, NONE)
    assert np.array_equal(sim.phase(api.PHASE_DENSITY), o.phase(0).astype(np.float32))
    sim.step(1)
    o.step(1)
    # the step's accelerations are held to 1e-5 of the reference's, not to its bits
    got, want = sim.state()[0], o.state()[0]
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    sim.close()
    o.close()


@pytest.mark.parametrize("copies", [1, 3, 12])
def test_noalloc_dense_cluster(copies):
    """`copies` of a few lattice particles on top of one another: up to some
    hundred accepted candidates for a particle, whose lanes keep 24 each."""
    import torch

    L = lib()
    L.sph_density_noalloc.restype = C.c_int
    L.sph_density_noalloc.argtypes = [C.c_float, C.c_float, C.c_void_p, C.c_uint, C.c_void_p, C.c_uint,
                                      C.POINTER(C.c_float), C.POINTER(C.c_float), C.c_void_p, C.c_void_p]
    sc = scene_of(S.WCSPH, (9, 8, 7))
    desc, base = sc.desc(), sc.fluid()[0]
    rng = np.random.default_rng(6)
    x = np.concatenate([base] + [base[:150] + rng.uniform(-0.01, 0.01, (150, 3)).astype(np.float32)
                                 for _ in range(copies - 1)]).astype(np.float32)
    o = Oracle(desc, x, NONE)
    want = o.phase(0).astype(np.float32)
    o.close()
    xt = torch.from_numpy(x).cuda()
    out = torch.full((len(x),), -1.0, dtype=torch.float32, device="cuda")
    lo, hi = (C.c_float * 3)(*x.min(0)), (C.c_float * 3)(*x.max(0))
    rc = L.sph_density_noalloc(desc.particle_radius, desc.density0, xt.data_ptr(), len(x), None, 0, lo, hi,
                               out.data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    assert np.array_equal(out.cpu().numpy(), want)
