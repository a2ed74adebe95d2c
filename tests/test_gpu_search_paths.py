"""Neighbour search on both sides of every line where its kernel changes (a
warp, four lanes or one lane per particle; densities in the search kernel or
in a pass of their own), against the CPU oracle: neighbour lists, densities and
boundary volumes entry for entry and bit for bit. The scenes stand against
their walls, so fluid and boundary lists are both exercised; a cluster so dense
that a lane's batch of accepted candidates overflows is checked by its counts.
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
