"""The pilot's line iteration beside the sweep's stages, where the window is
all of them: riser endpoints that no constraint touches.  The window decides
only when the line iteration runs, so a block too narrow to have one gives the
same bits, forward and in a rollout's gradients."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import simwing_b200 as sw
from simwing_b200 import abi
from tests.conftest import step_settings

ITERATIONS = 8
ATTACHMENT, HARNESS = 1, 3  # segment endpoint kinds


def net_with_pilot(nx=30, ny=20):
    """A net of edge springs (four stages) and a pilot on four free nodes
    beside it."""
    rng = np.random.default_rng(5)
    nodes = [(0.1 * i, 0.1 * j, 0.01 * rng.normal(), 0.01, i == 0) for j in range(ny) for i in range(nx)]
    cons = [(abi.DISTANCE, j * nx + i, j * nx + i + 1, 0.1, 1e-6) for j in range(ny) for i in range(nx - 1)]
    cons += [(abi.DISTANCE, j * nx + i, (j + 1) * nx + i, 0.1, 1e-6) for j in range(ny - 1) for i in range(nx)]
    o = len(nodes)
    corners = [(1.0, 0.6), (2.0, 0.6), (1.0, 1.4), (2.0, 1.4)]
    nodes += [(x, y, 0.0, 0.2, False) for x, y in corners]
    com = (1.5, 1.0, -3.0)
    harness = [(20 + k, (0.1 * (x - 1.5), 0.1 * (y - 1.0), 0.2)) for k, (x, y) in enumerate(corners)]
    segments = []
    for k, (x, y) in enumerate(corners):
        end = np.array(com) + harness[k][1]
        rest = 0.999 * float(np.linalg.norm(np.array((x, y, 0.0)) - end))
        segments.append((30 + k, (ATTACHMENT, 10 + k), (HARNESS, 20 + k), rest, 5.0e4, 1.0))
    suspension = dict(pilot_mass=80.0, pilot_com_world=com, pilot_inertia=(8.0, 8.0, 4.0),
                      attachments=[(10 + k, o + k) for k in range(4)], harness=harness, segments=segments,
                      solver_iterations=ITERATIONS, maximum_line_residual=1.0)
    return sw.definition_from_arrays(nodes, constraints=cons, suspension=suspension)


@pytest.mark.parametrize("ctas", [1, 4])
def test_window_of_every_stage_is_planned(ctas):
    r, _, _ = sw.plan_schedule(net_with_pilot(), sw.SolverOptions(cluster_ctas=ctas))
    # a window: no barrier of the line iteration's own beside the stages
    assert 2 <= r.local_stages_per_iteration <= 8
    assert r.cluster_barriers_per_iteration == r.local_stages_per_iteration


def test_window_of_a_block(tmp_path):
    """tests/cpp/line_window_test.cpp: the window for every block width."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    lib = os.path.join(root, "simwing_b200")
    out = tmp_path / "line_window_test"
    subprocess.run([cxx, "-std=c++20", "-O1", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(root, "include"),
                    os.path.join(root, "tests", "cpp", "line_window_test.cpp"), "-L", lib, "-lsimwing_b200",
                    f"-Wl,-rpath,{lib}", "-o", str(out)], check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("ctas", [1, 4, 16])
def test_window_changes_nothing(cuda_device, ctas):
    d = net_with_pilot()
    st = step_settings(iterations=ITERATIONS)
    target = d.positions() + 0.01
    want = None
    for threads in (0, 512, 32):  # 32: no window
        s = sw.Structure(d, sw.SolverOptions(cluster_ctas=ctas, block_threads=threads))
        with sw.Rollout(s, 4, 2) as r:
            loss = r.forward(st, target, np.ones(d.node_count))
            grad = r.backward()
        s.step_many(st, 4)
        p = s.suspension_state()
        got = [s.node_states(), np.array([*p.center_of_mass, *p.body_to_world, *p.linear_velocity, *p.angular_velocity]),
               loss] + [grad[k] for k in sorted(grad)]
        assert np.abs(got[0][-4:, 0, :] - d.positions()[-4:]).max() > 1e-6  # the lines pull
        if want is None:
            want = got
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b, err_msg=f"{threads} threads")
