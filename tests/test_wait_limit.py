"""Hand-over waits that run out, on the nodes of a CTA that leaves its sweep
out: the step, the rollout's forward and its backward report it in bounded
time, leave the state as it was, and the structure goes on afterwards."""
import numpy as np
import pytest

import simwing_b200 as sw
from tests.conftest import step_settings
from tests.test_hand_over import random_net

pytestmark = pytest.mark.gpu

LIMIT = 2_000_000  # cycles, about a millisecond


def make(kind):
    if kind == "patch":
        return sw.generate_patch(nx=97, ny=61)
    return sw.generate_wing(cells=10, chordwise=30, spanwise_per_cell=3, rib_layers=2)


@pytest.mark.parametrize("held", [0, 9, 15])
@pytest.mark.parametrize("kind", ["patch", "wing"])
def test_hand_over_wait_runs_out(cuda_device, kind, held):
    d = make(kind)
    st = step_settings()
    options = sw.SolverOptions(cluster_ctas=16)
    s, twin = sw.Structure(d, options), sw.Structure(d, options)
    for bad in ((-1, -1), (0, 16), (0, -2)):
        with pytest.raises(sw.InvalidArgument):
            s.set_wait_limit(*bad)
    s.step(st)
    twin.step(st)
    before = s.node_states()
    s.set_wait_limit(LIMIT, held)
    for _ in range(3):
        with pytest.raises(sw.SyncTimeout, match="handed over"):
            s.step(st)
        np.testing.assert_array_equal(s.node_states(), before)
        assert s.accepted_step_count() == 1
    s.set_wait_limit()
    s.step(st)
    twin.step(st)
    np.testing.assert_array_equal(s.node_states(), twin.node_states())


def test_rollout_waits_run_out(cuda_device):
    d = make("wing")
    st = step_settings()
    s = sw.Structure(d, sw.SolverOptions(cluster_ctas=16))
    target, weights = s.positions() + 0.01, np.ones(d.node_count)
    with sw.Rollout(s, 2, 1) as r:
        loss = r.forward(st, target, weights)
        want = r.backward()
        s.set_wait_limit(LIMIT, 5)
        with pytest.raises(sw.SyncTimeout):
            r.backward()
        with pytest.raises(sw.SyncTimeout):
            r.forward(st, target, weights)
        s.set_wait_limit()
        assert r.forward(st, target, weights) == loss
        got = r.backward()
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


def test_direct_schedules_have_no_waits(cuda_device):
    d = random_net()
    st = step_settings(iterations=4)
    s, twin = sw.Structure(d), sw.Structure(d)
    s.set_wait_limit(LIMIT, 3)
    target, weights = s.positions() + 0.01, np.ones(d.node_count)
    grads = []
    for x in (s, twin):
        with sw.Rollout(x, 1, 1) as r:
            r.forward(st, target, weights)
            grads.append(r.backward())
        x.step(st)
    np.testing.assert_array_equal(s.node_states(), twin.node_states())
    for k in grads[0]:
        np.testing.assert_array_equal(grads[0][k], grads[1][k], err_msg=k)
