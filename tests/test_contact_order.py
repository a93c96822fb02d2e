"""Key-ordered contact passes whose links stay in global memory (surfaces with
more candidates in contact than shared memory holds links for) against the
same scene alone, whose links fit: many copies of a landed sheet far apart
do not touch each other, so each moves as the single one does."""
import numpy as np
import pytest

import simwing_b200 as sw

pytestmark = pytest.mark.gpu


def copies(n, count, pitch):
    """`count` copies of stacked_sheets(n), `pitch` apart along x."""
    one = sw.stacked_sheets(n=n, compliance=1e-3)
    nodes, cons, tris = one.nodes(), one.constraints(), one.triangles()
    N = one.node_count
    p = one.positions()
    all_nodes, all_tris, all_cons = [], [], []
    for k in range(count):
        all_nodes += [(x + k * pitch, y, z, m, bool(f)) for (x, y, z), m, f in zip(p, nodes["mass"], nodes["fixed"])]
        all_tris += [tuple(int(v) + k * N for v in t) for t in tris["nodes"]]
        all_cons += [(int(c["kind"]), int(c["first_node"]) + k * N, int(c["second_node"]) + k * N,
                      float(c["rest_length"]), float(c["compliance"])) for c in cons]
    return one, sw.definition_from_arrays(all_nodes, all_tris, all_cons, contact=(0.002, 1e-3, 0.4, 0.25))


@pytest.mark.parametrize("n,count", [(8, 40), (16, 12)])
def test_links_in_global_memory(cuda_device, n, count):
    one, many = copies(n, count, 1.5)
    st = sw.StepSettings(time_step=1.0 / 120.0, substeps=1, constraint_iterations=8, gravity=(2.0, 0.0, -9.81),
                         velocity_damping=0.25)
    a, b = sw.Structure(one), sw.Structure(many)
    da, db = a.step(st), b.step(st)
    assert da.active_contact_count > 0
    x = a.positions()
    y = b.positions().reshape(count, one.node_count, 3)
    # FP32 offsets of up to 30 m are rounded at 1e-6 m (half a spacing); a
    # node takes about six corrections in each of the eight iterations
    tol = 8 * 6 * 1.0e-6
    for k in range(count):
        assert np.abs(y[k] - [k * 1.5, 0.0, 0.0] - x).max() <= tol
    assert abs(db.maximum_contact_penetration - da.maximum_contact_penetration) <= tol


def test_order_of_a_single_contact(cuda_device):
    """The smallest surfaces: a few candidates, one round."""
    st = sw.StepSettings(time_step=1.0 / 120.0, substeps=1, constraint_iterations=2, gravity=(0.0, 0.0, -9.81),
                         velocity_damping=0.0)
    s = sw.Structure(sw.stacked_sheets(n=2, compliance=1e-3))
    d = s.step(st)
    assert d.finite == 1 and d.active_contact_count > 0
