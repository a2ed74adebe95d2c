"""What follows a neighbour list that outgrew its capacity: the step that meets
it reports the overflow, the capacity grows, and the next step runs on complete
lists. A context whose lists are built once more from the same positions before
that step (by a change of the cell order and back) is the reference: the same
lists in the same order, so the tolerance is zero.
"""
import numpy as np
import pytest

from sph2o_b200 import api
from sph2o_b200 import scenes as S
from sph2o_b200.api import Scene, Simulation, SphError

pytestmark = pytest.mark.gpu
NONE = np.zeros((0, 3), np.float32)
OVERFLOW = -4


def block_of(method, dims=(14, 13, 12), r=0.02):
    ext = [2 * r * k for k in dims]
    sc = Scene.from_dict(S.scene(
        method=method, radius=r, blocks=[S.block(dims, r, (2 * r,) * 3)],
        tank=((0, 0, 0), (ext[0] + 8 * r, ext[1] + 8 * r, ext[2] + 8 * r)), time_step=5e-4, jitter=0.3, seed=3))
    return sc.desc(), sc.fluid()[0]


def overflowing(desc, x, squeeze):
    """A context whose last step met more neighbours (74 at 0.82, 78 at 0.8) than its lists hold (64)."""
    sim = Simulation(desc, x, NONE)
    sim.set_state((np.float32(0.1) + x * np.float32(squeeze)).astype(np.float32), np.zeros_like(x))
    with pytest.raises(SphError) as e:
        sim.step(1)
    assert e.value.code == OVERFLOW
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
