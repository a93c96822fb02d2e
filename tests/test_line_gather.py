"""Line-line projections on gathered cable nodes, and in place when a mesh has
more cable nodes than shared memory has room for: many crossing pairs far
apart move as one pair alone does, in either form."""
import numpy as np
import pytest

import simwing_b200 as sw
from simwing_b200 import abi
from tests.conftest import step_settings

pytestmark = pytest.mark.gpu

RADIUS = 0.004


def pairs(count, pitch=0.5, apart=0.002):
    side = int(np.ceil(np.sqrt(count)))
    nodes, cons = [], []
    for k in range(count):
        x, y = (k % side - side // 2) * pitch, (k // side - side // 2) * pitch
        o = len(nodes)
        nodes += [(x - 0.1, y, 0.5 * apart, 0.01, False), (x + 0.1, y, 0.5 * apart, 0.01, False),
                  (x, y - 0.1, -0.5 * apart, 0.01, False), (x, y + 0.1, -0.5 * apart, 0.01, False)]
        cons += [(abi.CABLE, o, o + 1, 0.2, 1e-8), (abi.CABLE, o + 2, o + 3, 0.2, 1e-8)]
    centre = np.array([[(k % side - side // 2) * pitch, (k // side - side // 2) * pitch, 0.0] for k in range(count)])
    return sw.definition_from_arrays(nodes, constraints=cons), centre


# 3,600 pairs: 14,400 cable nodes want 245 KB
@pytest.mark.parametrize("count", [1, 3, 33, 3600])
def test_pairs_move_alike(cuda_device, count):
    st = step_settings(iterations=4, gravity=(0.0, 0.0, 0.0), damping=0.0)
    d, centre = pairs(count)
    s = sw.Structure(d)
    s.set_line_contact(RADIUS, 0.002)
    s.step(st)
    x = s.positions().reshape(count, 4, 3) - centre[:, None, :]
    # pushed 2 x radius apart along z, both ends of a segment alike; FP32
    # offsets of up to 15 m round at 5e-7 m, four iterations of four roundings
    tol = 4 * 4 * 5.0e-7
    gap = x[:, :2, 2].mean(axis=1) - x[:, 2:, 2].mean(axis=1)
    assert np.abs(gap - 2 * RADIUS).max() <= tol
    assert np.abs(x[:, 0, 2] - x[:, 1, 2]).max() <= tol and np.abs(x[:, 2, 2] - x[:, 3, 2]).max() <= tol
    assert np.abs(x[:, :, 2].sum(axis=1)).max() <= 2 * tol


def test_far_pairs_stay(cuda_device):
    """Within the margin, not too near: the contact moves no node (the cables
    themselves round their lengths)."""
    st = step_settings(iterations=4, gravity=(0.0, 0.0, 0.0), damping=0.0)
    d, _ = pairs(5, apart=2.1 * RADIUS)
    alone, s = sw.Structure(d), sw.Structure(d)
    s.set_line_contact(RADIUS, 0.002)
    alone.step(st)
    s.step(st)
    np.testing.assert_array_equal(s.positions(), alone.positions())
