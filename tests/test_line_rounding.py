"""Line-line projections at the edge of contact: pairs a rounding or two from
2 x radius apart, at offsets of several metres, where a coordinate's own
rounding (0.5 um) is as large as what decides.  Gathered nodes and nodes in
place take the same decisions and move alike to the last bit."""
import numpy as np
import pytest

import simwing_b200 as sw
from simwing_b200 import abi
from tests.conftest import step_settings

pytestmark = pytest.mark.gpu

RADIUS, PITCH, SIDE = 0.002, 0.3, 60
TESTED = 400  # pairs of the gathered form; with the others (3,600 pairs) there is no room to gather


def pairs(count, seed):
    """Crossing segments in random directions on a grid, the corners of the
    grid's box pinned, so that the offsets' origin is the same for any count."""
    rng = np.random.default_rng(seed)
    nodes, cons = [], []
    for k in range(count):
        o = len(nodes)
        centre = np.array([(k * 7919 % SIDE**2 % SIDE + 0.5) * PITCH, (k * 7919 % SIDE**2 // SIDE + 0.5) * PITCH, 7.0])
        u, v = np.linalg.qr(rng.normal(size=(3, 2)))[0].T
        n = np.cross(u, v)
        v = v + rng.uniform(-0.9, 0.9) * u
        half = 0.5 * n * 2 * RADIUS * (1.0 + 2.0e-4 * rng.normal())
        for p in (centre + half - rng.uniform(0.02, 0.1) * u, centre + half + rng.uniform(0.02, 0.1) * u,
                  centre - half - rng.uniform(0.02, 0.1) * v, centre - half + rng.uniform(0.02, 0.1) * v):
            nodes.append((*p, 0.01 * rng.uniform(0.5, 2.0), False))
        for a, b in ((o, o + 1), (o + 2, o + 3)):
            rest = float(np.linalg.norm(np.subtract(nodes[a][:3], nodes[b][:3])))
            cons.append((abi.CABLE, a, b, 1.01 * rest, 1e-8))  # slack
    nodes += [(0.0, 0.0, 6.0, 1.0, True), (SIDE * PITCH, SIDE * PITCH, 8.0, 1.0, True)]
    return sw.definition_from_arrays(nodes, constraints=cons)


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("iterations", [1, 5])
def test_gathered_and_in_place_round_alike(cuda_device, seed, iterations):
    st = step_settings(iterations=iterations, gravity=(0.0, 0.0, 0.0), damping=0.0)
    moved = []
    for count in (TESTED, SIDE**2):
        s = sw.Structure(pairs(count, seed))
        before = s.positions()[: 4 * TESTED]
        s.set_line_contact(RADIUS, 0.001)
        s.step(st)
        after = s.positions()[: 4 * TESTED]
        moved.append(after)
        touched = (after != before).any(axis=1).sum()
        assert TESTED < touched < 3 * TESTED  # about half of the pairs are in contact
    np.testing.assert_array_equal(moved[0], moved[1])
