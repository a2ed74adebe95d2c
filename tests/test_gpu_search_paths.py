"""Neighbour search on both sides of every line where its kernel changes (a
warp, four lanes or one lane per particle; densities in the search kernel or
in a pass of their own), against the CPU oracle: neighbour lists, densities and
boundary volumes entry for entry and bit for bit. The scenes stand against
their walls, so fluid and boundary lists are both exercised. A cluster of particles
with more neighbours than a list holds is checked by its counts; columns so dense
that one of the four lanes accepts more than its batch holds are checked by value.
"""
import numpy as np
import pytest

from oracle.oracle import Oracle
from sph2o_b200 import api
from sph2o_b200 import scenes as S
from sph2o_b200.api import Scene, Simulation

pytestmark = pytest.mark.gpu


def brute_force_counts(x, y, h, chunk=512):
    """|{j : |x_i - y_j| <= h}| with the reference's FP32 rounding."""
    out = np.zeros(len(x), np.int64)
    for a in range(0, len(x), chunk):
        d = x[a:a + chunk, None, :] - y[None, :, :]
        s = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
        out[a:a + chunk] = (np.sqrt(s) <= h).sum(1)
    return out


def scene_of(method, dims, order=0):
    r = 0.02
    ext = [2 * r * k for k in dims]
    return S.scene(method=method, radius=r, blocks=[S.block(dims, r, (2 * r,) * 3)],
                   tank=((0, 0, 0), (ext[0] + 8 * r, ext[1] + 8 * r, ext[2] + 8 * r)), time_step=1e-4, jitter=0.05,
                   seed=dims[0])


# 7 x 5 x 3; 16,383 and 16,384; 49,104 and 49,152; 262,088 and 262,144 particles
@pytest.mark.parametrize("dims", [(7, 5, 3), (129, 127, 1), (32, 32, 16), (48, 33, 31), (48, 32, 32), (181, 8, 181),
                                  (64, 64, 64)])
@pytest.mark.parametrize("method", [S.WCSPH, S.DFSPH])
def test_densities_at_the_kernel_lines(dims, method):
    sc = Scene.from_dict(scene_of(method, dims))
    desc, x, b = sc.desc(), sc.fluid()[0], sc.boundary()
    sim = Simulation(desc, x, b)
    o = Oracle(desc, x, b)
    assert np.array_equal(sim.boundary_volume(), o.boundary_volume().astype(np.float32))
    assert np.array_equal(sim.phase(api.PHASE_DENSITY), o.phase(0).astype(np.float32))
    for got, want in zip(sim.neighbors(), o.neighbors()):
        assert np.array_equal(got, want)
    sim.close()
    o.close()


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("copies", [1, 40])
def test_dense_cluster_counts(order, copies):
    """`copies` jittered copies of the lattice's first particles on top of it:
    hundreds of candidates in a row of cells; lists longer than their capacity are
    reported as an overflow, never written past it."""
    r = 0.02
    rng = np.random.default_rng(5)
    base = np.stack(np.meshgrid(*[np.arange(n) * 2 * r for n in (30, 25, 24)], indexing="ij"), -1).reshape(-1, 3)
    n_dense = 60 if copies > 1 else 0
    x = np.concatenate([base] + [base[:n_dense] + rng.uniform(-0.4 * r, 0.4 * r, (n_dense, 3))
                                 for _ in range(copies - 1)]).astype(np.float32)
    sc = Scene.from_dict(scene_of(S.WCSPH, (4, 4, 4)))
    desc = sc.desc()
    h = np.float32(4.0) * np.float32(desc.particle_radius)
    want = brute_force_counts(x, x, h)
    if copies > 1:
        assert want.max() > 64
        with pytest.raises(api.SphError) as e:
            Simulation(desc, x, np.zeros((0, 3), np.float32), options={api.OPT_CELL_ORDER: order})
        assert e.value.code == -4
        return
    sim = Simulation(desc, x, np.zeros((0, 3), np.float32), options={api.OPT_CELL_ORDER: order})
    off, idx, boff, bidx = sim.neighbors()
    assert np.array_equal(np.diff(off.astype(np.int64)), want)


def columns(nx, nz, h, offset=0.0):
    """nx x nx columns of nz particles, 1.05 h apart, h / 14 between particles: a
    particle's neighbours lie in its own column."""
    k = np.arange(nx, dtype=np.float64) * 1.05 * h
    z = np.arange(nz, dtype=np.float64) * h / 14
    x = np.stack(np.meshgrid(k, k, z, indexing="ij"), -1).reshape(-1, 3) + h + offset
    return x.astype(np.float32)


def lane_counts(x, y, h):
    """Accepted candidates of each particle of x among y by the lane that walks
    them: the nine (x, y) rows of cells in candidate order go 3, 2, 2, 2 to four."""
    from scipy.spatial import cKDTree

    cell_x, cell_y = np.floor(x / h).astype(np.int64), np.floor(y / h).astype(np.int64)
    out = np.zeros((len(x), 4), np.int64)
    for i, near in enumerate(cKDTree(y.astype(np.float64)).query_ball_point(x.astype(np.float64), 1.01 * float(h))):
        j = np.asarray(near, np.int64)
        d = x[i] - y[j]
        j = j[np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]) <= h]
        step = cell_y[j] - cell_x[i]
        lanes = np.array([0, 0, 0, 1, 1, 2, 2, 3, 3])[(step[:, 0] + 1) * 3 + step[:, 1] + 1]
        out[i] = np.bincount(lanes, minlength=4)
    return out


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("method", [S.WCSPH, S.PCISPH])
@pytest.mark.parametrize("dense", ["fluid", "boundary"])
def test_more_candidates_than_a_lane_holds(dense, method, order):
    """Densities against the oracle. A step against the same particles among so
    many others, out of reach, that one lane per particle searches (and as many
    lanes as before sum the forces, and PCISPH iterates as often): the lists, and
    so the states, are the same, and the tolerance is zero."""
    sc = Scene.from_dict(scene_of(method, (4, 4, 4)))
    desc = sc.desc()
    desc.min_iterations = desc.max_iterations = 3
    h = np.float32(4.0) * np.float32(desc.particle_radius)
    tall, flat = columns(8, 40, h), columns(8, 40, h, 0.1 * h)
    x, b = (tall, flat[::9]) if dense == "fluid" else (tall[::9], flat)
    rest = np.stack(np.meshgrid(*[np.arange(k) * 0.5 * h for k in (30, 30, 20)], indexing="ij"), -1).reshape(-1, 3)
    x = np.concatenate([x, (rest + 14 * h).astype(np.float32)])
    fluid, boundary = lane_counts(x, x, h), lane_counts(x, b, h)
    assert 16384 <= len(x) < 49152 and (fluid if dense == "fluid" else boundary).max() > 24
    assert max(fluid.sum(1).max(), boundary.sum(1).max()) <= 64
    far = np.stack(np.meshgrid(*[np.arange(k) * 0.5 * h for k in (40, 40, 20)], indexing="ij"), -1).reshape(-1, 3)
    more = np.concatenate([x, (far + 40 * h).astype(np.float32)])
    assert 49152 <= len(more) < 65536
    states = []
    for fluid_set in (x, more):
        sim, o = Simulation(desc, fluid_set, b, options={api.OPT_CELL_ORDER: order}), Oracle(desc, fluid_set, b)
        assert np.array_equal(sim.phase(api.PHASE_DENSITY), o.phase(0).astype(np.float32))
        sim.step(1)
        states.append([a[:len(x)] for a in sim.state()])
        sim.close()
        o.close()
    for four_lanes, one_lane in zip(*states):
        assert np.array_equal(four_lanes, one_lane)
