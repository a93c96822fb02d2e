"""A contact step refused because a feature's closest points cannot be
certified: a free triangle that the prediction flattens onto a line, inside the
envelope of a pinned one.  The refusal is the step's result whatever the
cluster: the same message and feature, the state as it was."""
import numpy as np
import pytest

import simwing_b200 as sw
from tests.conftest import step_settings

pytestmark = pytest.mark.gpu

DT = 1.0 / 128.0
HEIGHT = 2.0 ** -10  # of the free triangle; a load of -16 N on its tip takes it to 0 exactly


def scene(copies, pitch=4.0):
    nodes, tris, tips = [], [], []
    for k in range(copies):
        x, o = k * pitch, len(nodes)
        nodes += [(x, 0.0, 0.0, 1.0, 0), (x + 1.0, 0.0, 0.0, 1.0, 0), (x + 0.25, HEIGHT, 0.0, 1.0, 0),
                  (x + 0.5, 0.0, -0.005, 1.0, 1), (x + 0.5, -1.0, -0.005, 1.0, 1), (x + 1.5, -1.0, -0.005, 1.0, 1)]
        tris += [(o, o + 1, o + 2), (o + 3, o + 4, o + 5)]
        tips.append(o + 2)
    return sw.definition_from_arrays(nodes, tris, contact=(0.01, 0.0, 0.0, 0.0)), tips


@pytest.mark.parametrize("copies", [1, 200])
def test_uncertified_geometry_fails_the_step(cuda_device, copies):
    d, tips = scene(copies)
    st = step_settings(iterations=4, dt=DT, gravity=(0.0, 0.0, 0.0), damping=0.0)
    seen = []
    for ctas in (1, 4, 16):
        tried, twin = (sw.Structure(d, sw.SolverOptions(cluster_ctas=ctas)) for _ in range(2))
        for s in (tried, twin):
            for tip in tips:
                s.add_external_force(tip, (0.0, -16.0, 0.0))
        for _ in range(3):
            with pytest.raises(sw.ContactStepError) as err:
                tried.step(st)
            seen.append((str(err.value), err.value.key))
        assert tried.checkpoint() == twin.checkpoint()
        assert tried.accepted_step_count() == 0
    assert len(set(seen)) == 1, seen
    assert "Contact endpoint geometry is not certifiable" in seen[0][0]
    # the first feature in key order that has the flattened triangle: the
    # first copy's pinned vertex under it
    assert seen[0][1][2][0] == 3, seen[0]
