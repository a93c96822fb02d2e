"""Hand-over of nodes between the CTAs of a cluster, at the sizes where it can
go wrong: blocks narrower than a stage (several rounds, boundary records past
the first), odd cluster widths, patches of a few nodes, and meshes whose
boundary does not fit beside their patches (direct schedules).

A structure's result belongs to its colouring alone, so the block size must
not change a bit of it; against the FP64 oracle one step stays within the
parity bound of the other schedules (1e-5 relative: FP32 positions of a few
metres are rounded at 5e-7 per projection).
"""
import numpy as np
import pytest

import simwing_b200 as sw
from oracle import oracle as O
from simwing_b200 import abi
from tests.conftest import step_settings
from tests.test_gpu_parity import REL_TOL, per_step_errors


def random_net(nodes=24000, per_node=9, seed=7):
    """Springs between nodes drawn at random from a box: nearly every spring
    spans two patches, and a CTA touches most of its neighbours' nodes."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-5.0, 5.0, (nodes, 3))
    a = np.repeat(np.arange(nodes), per_node)
    b = (a + rng.integers(1, nodes, a.size)) % nodes
    keep = np.unique(np.sort(np.stack([a, b], 1), axis=1), axis=0)
    rest = np.linalg.norm(x[keep[:, 0]] - x[keep[:, 1]], axis=1) * rng.uniform(0.97, 1.03, len(keep))
    return sw.definition_from_arrays([(*p, 1.0, i % 50 == 0) for i, p in enumerate(x)],
                                     constraints=[(abi.DISTANCE, int(u), int(v), float(r), 1e-4)
                                                  for (u, v), r in zip(keep, rest)])


def test_direct_schedule_invariants():
    # the schedule verifier walks the hand-overs of both directions
    d = random_net()
    r, order, _ = sw.plan_schedule(d)
    assert r.cluster_ctas == 16
    assert sorted(order.tolist()) == list(range(d.view.constraint_count))


@pytest.mark.parametrize("ctas", [2, 3, 7, 16])
@pytest.mark.parametrize("nx,ny", [(5, 4), (37, 23)])
def test_hand_over_invariants(nx, ny, ctas):
    d = sw.generate_patch(nx=nx, ny=ny)
    for flags in (0, abi.OPT_SPLIT_STAGES):
        r, _, _ = sw.plan_schedule(d, sw.SolverOptions(cluster_ctas=ctas, flags=flags))
        assert r.cluster_ctas == ctas


@pytest.mark.gpu
@pytest.mark.parametrize("ctas", [1, 3, 16])
@pytest.mark.parametrize("kind", ["patch", "wing", "fabric"])
def test_block_size_changes_nothing(cuda_device, kind, ctas):
    d = {"patch": lambda: sw.generate_patch(nx=37, ny=23),
         "wing": lambda: sw.generate_wing(cells=5, chordwise=14, spanwise_per_cell=3, rib_layers=2),
         "fabric": lambda: sw.generate_wing(cells=5, chordwise=14, spanwise_per_cell=3, rib_layers=2, fabric=1)}[kind]()
    want = None
    for threads in (0, 32, 64, 96, 512, 768):
        s = sw.Structure(d, sw.SolverOptions(cluster_ctas=ctas, block_threads=threads))
        s.step_many(step_settings(), 3)
        got = s.node_states()
        want = got if want is None else want
        np.testing.assert_array_equal(got, want, err_msg=f"{threads} threads")


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,ctas", [(5, 4, 16), (9, 9, 7), (37, 23, 3)])
def test_small_patches_parity(cuda_device, nx, ny, ctas):
    errs, _, _ = per_step_errors(sw.generate_patch(nx=nx, ny=ny), 4, step_settings(),
                                 sw.SolverOptions(cluster_ctas=ctas))
    assert max(errs) <= REL_TOL, errs


@pytest.mark.gpu
def test_direct_schedule_parity(cuda_device):
    d = random_net()
    st = step_settings(iterations=6)
    errs, dev, _ = per_step_errors(d, 3, st)
    # no ghosts in the layout: the patches (1,500 nodes) and the multipliers
    # (13,500 records per CTA) alone
    assert dev.schedule_report().shared_bytes < 100 * 1024
    assert max(errs) <= REL_TOL, errs


@pytest.mark.gpu
def test_direct_schedule_in_a_batch(cuda_device):
    defs = [random_net(), sw.generate_patch(nx=20, ny=20), sw.generate_wing(cells=4, chordwise=10, spanwise_per_cell=2)]
    st = step_settings(iterations=6)
    st_wing = step_settings()
    with sw.Batch(defs[:2], sw.BatchOptions(graph_steps=2)) as batch:
        assert not batch.step(st, 3).any()
        for i in range(2):
            plain = sw.Structure(defs[i], sw.SolverOptions(
                cluster_ctas=batch.structure(i).schedule_report().cluster_ctas))
            for _ in range(3):
                plain.step(st, diagnostics=False)
            np.testing.assert_array_equal(batch.structure(i).node_states(), plain.node_states())
    # a cluster of hand-over structures beside each other
    with sw.Batch(defs[1:], sw.BatchOptions(graph_steps=2, target_patch_nodes=128)) as batch:
        assert not batch.step(st_wing, 3).any()
        for i in range(2):
            plain = sw.Structure(defs[1 + i], sw.SolverOptions(
                cluster_ctas=batch.structure(i).schedule_report().cluster_ctas))
            for _ in range(3):
                plain.step(st_wing, diagnostics=False)
            np.testing.assert_array_equal(batch.structure(i).node_states(), plain.node_states())


@pytest.mark.gpu
@pytest.mark.parametrize("per_node", [5, 9])
def test_direct_schedule_gradient(cuda_device, per_node):
    """Reverse sweep of a direct schedule (nine springs a node), and a direct
    reverse of a schedule that hands over (five a node: the reverse keeps
    more per record and has no room for the ghosts), against the FP64 adjoint (the bound
    of the other rollout gradients, 1e-3 of the gradient's norm; two short
    steps keep both solvers on one trajectory to 1e-6)."""
    d = random_net(per_node=per_node)
    st = step_settings(iterations=4)
    s = sw.Structure(d)
    target = s.positions() + 0.01
    weights = np.ones(d.node_count)
    with sw.Rollout(s, 2, 2) as r:
        r.forward(st, target, weights)
        g = r.backward()
    order = s.sweep_order(abi.SWEEP_DISTANCE)
    ref = np.empty(len(order))
    ref[order] = O.rollout_gradient(s.oracle_definition(), st, 2, target, weights)["d_rest"]
    assert np.linalg.norm(g["d_rest"] - ref) <= 1e-3 * np.linalg.norm(ref)
