"""Performance cases: the structural step as programs call it.

Every case goes through the package's public entry points with the
settings of the benchmark (dt 1/120 s, 48 iterations, gravity, velocity
damping 0.25, 30 Pa in the wings) and gives back whole states: positions,
previous positions and velocities of every node, the pilot and the step's
diagnostics, the loss and every gradient of a rollout.

kinds
  cloth    a hanging patch (two pinned corners, or free), `steps` steps, then
           its nodes: a cloth viewer's frame; the smallest calls.
  wing     one ram-air wing in a coupled loop: nodal loads in (from the host,
           or from device memory through the coupling caller), one step with
           diagnostics, nodes and pilot out.  `steps` > 1 is an animation
           frame instead (that many steps at the loads' last values, no
           diagnostics between).  Options: `fabric` (membrane elements
           instead of edge constraints), `lines` (line-line contact of the
           cascaded lines).
  contact  a sheet landed on a pinned one, fabric self-contact with friction:
           a step from a restored checkpoint (a coupled run's retry), 8
           iterations.
  batch    several wings of uneven sizes stepped together, then all nodes.
  gradient rollouts side by side, forward and backward: one optimiser step of
           a line trim calibration.  Options: `ground` (a contact plane inside
           the trailing edge) and `lines`.

Sizes span the repository's own: patches from 9 x 9 to the benchmark's 33 x 33
and three times that, wings from the smoke test's few hundred triangles to the
benchmark's 40 cells x 60 chordwise (68,412 triangles), sheets of 12 to 40
nodes a side.
"""
import math

import numpy as np
import torch

import simwing_b200 as sw

WING = dict(kind="wing", cells=40, chordwise=60, spanwise=4, attachments=1, fabric=False, lines=False, loads="host",
            steps=1)


def _wing(name, **kw):
    return dict(WING, name=name, **kw)


def listed():
    return [
        # the smallest call: a coarse cloth in a viewer, one step a frame
        dict(name="cloth_9", kind="cloth", nx=9, ny=9, free=False, steps=1),
        # the benchmark's patch, a 60 Hz frame of two 120 Hz steps
        dict(name="cloth_33", kind="cloth", nx=33, ny=33, free=False, steps=2),
        # a large free sheet (the momentum guard runs), odd sizes
        dict(name="cloth_free_97x61", kind="cloth", nx=97, ny=61, free=True, steps=2),
        # a coarse wing of a preview run, coupled from the host
        _wing("wing_6x14_host", cells=6, chordwise=14, spanwise=3),
        # the calibration wing, coupled from device memory
        _wing("wing_20x30_device", cells=20, chordwise=30, attachments=2, loads="device"),
        # the benchmark's wing, coupled from the host: nodal loads in, nodes out
        _wing("wing_40x60_host", loads="host"),
        # the same as an animation frame (two 60 Hz frames of 120 Hz steps)
        _wing("wing_40x60_frame", steps=4),
        # the same with membrane fabric
        _wing("wing_40x60_fabric", fabric=True, loads="device"),
        # line-line contact of the cascaded lines on a wing of the trim workload
        _wing("wing_31x45_lines", cells=31, chordwise=45, lines=True),
        # fabric self-contact, a landed sheet
        dict(name="contact_24", kind="contact", side=24),
        # uneven wings stepped together
        dict(name="batch_8", kind="batch", wings=8, cells=20, chordwise=30, steps=4),
        # one optimiser step of the line calibration on the calibration wing
        dict(name="gradient_20x30", kind="gradient", cells=20, chordwise=30, wings=1, steps=16, ground=False,
             lines=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cloth", "wing", "wing", "wing", "contact", "batch", "gradient"])
    if kind == "cloth":
        return dict(kind=kind, nx=_log(rng, 9, 97), ny=_log(rng, 9, 97), free=rng.random() < 0.3,
                    steps=rng.randint(1, 4))
    if kind == "wing":
        fabric = rng.random() < 0.25
        return dict(WING, cells=_log(rng, 4, 40), chordwise=_log(rng, 10, 60), spanwise=rng.randint(2, 4),
                    attachments=rng.randint(1, 2), fabric=fabric, lines=not fabric and rng.random() < 0.25,
                    loads=rng.choice(["host", "device"]), steps=rng.choice([1, 1, 1, 3]))
    if kind == "contact":
        return dict(kind=kind, side=_log(rng, 12, 40))
    if kind == "batch":
        return dict(kind=kind, wings=rng.randint(3, 8), cells=_log(rng, 6, 20), chordwise=_log(rng, 12, 30),
                    steps=rng.randint(1, 4))
    contact = rng.random() < 0.35
    return dict(kind=kind, cells=_log(rng, 6, 18), chordwise=_log(rng, 12, 28), wings=rng.randint(1, 2),
                steps=rng.randint(4, 8 if contact else 16), ground=contact, lines=contact)


# ---- inputs ---------------------------------------------------------------------
def _settings(iterations=48, gravity=(0.0, 0.0, -9.81)):
    return sw.StepSettings(time_step=1.0 / 120.0, substeps=1, constraint_iterations=iterations, gravity=gravity,
                           velocity_damping=0.25)


def _wing_definition(case, seed):
    return sw.generate_wing(cells=case["cells"], chordwise=case["chordwise"],
                            spanwise_per_cell=case.get("spanwise", 4),
                            attachments_per_cell=case.get("attachments", 1), compliance_jitter=0.1, seed=seed + 1,
                            **({"fabric": 1} if case.get("fabric") else {}))


def _gust(definition, seed):
    """Nodal loads of a gust: every node's weight times a smooth random field
    of a few tenths of gravity (newtons, definition order)."""
    rng = np.random.default_rng(seed)
    x = definition.positions()
    mass = definition.nodes()["mass"]
    k = rng.normal(0.0, 1.0, (3, 3))
    phase = rng.uniform(0.0, 2.0 * np.pi, 3)
    return 2.0 * np.sin(x @ k + phase) * mass[:, None]


def _prepare_cloth(case, seed):
    d = sw.generate_patch(nx=case["nx"], ny=case["ny"], seed=seed + 1, pin_top_corners=0 if case["free"] else 1)
    return {"structure": sw.Structure(d), "settings": _settings()}


def _prepare_wing(case, seed):
    d = _wing_definition(case, seed)
    s = sw.Structure(d)
    if case["lines"]:
        s.set_line_contact(0.001, 0.002)
    loads = _gust(d, seed)
    state = {"structure": s, "settings": _settings(), "loads": loads}
    if case["loads"] == "device":
        state["coupling"] = sw.Coupling(s, np.arange(d.node_count))
        state["impulses"] = torch.from_numpy(loads * state["settings"].time_step).cuda()
    return state


def _prepare_contact(case, seed):
    rng = np.random.default_rng(seed)
    d = sw.stacked_sheets(n=case["side"], gap=0.003 + rng.uniform(-1.0e-4, 1.0e-4), compliance=1.0e-3)
    s = sw.Structure(d)
    return {"structure": s, "settings": _settings(8, (2.0, 0.0, -9.81)), "image": s.checkpoint()}


def _prepare_batch(case, seed):
    rng = np.random.default_rng([case["wings"], case["cells"], case["chordwise"]])
    defs = []
    for i in range(case["wings"]):
        size = dict(cells=max(4, int(round(case["cells"] * rng.uniform(0.5, 1.5)))),
                    chordwise=max(10, int(round(case["chordwise"] * rng.uniform(0.6, 1.4)))),
                    aspect_ratio=float(rng.uniform(4.5, 7.0)))
        defs.append(sw.generate_wing(compliance_jitter=0.2, seed=1000 * (seed + 1) + i, **size))
    return {"batch": sw.Batch(defs), "settings": _settings()}


def _prepare_gradient(case, seed):
    rng = np.random.default_rng(seed)
    settings = _settings()
    state = {"settings": settings, "structures": [], "rollouts": [], "targets": [], "weights": []}
    for i in range(case["wings"]):
        d = sw.generate_wing(cells=case["cells"], chordwise=case["chordwise"], attachments_per_cell=2,
                             compliance_jitter=0.1, seed=1000 * (seed + 1) + i)
        s = sw.Structure(d)
        s.step_many(settings, 20)
        x = s.positions()
        if case["ground"]:
            s.set_ground((-1.0, 0.0, 0.0), -(float(x[:, 0].max()) - 0.01), 0.0)
        if case["lines"]:
            s.set_line_contact(0.001, 0.002)
        w = np.zeros(d.node_count)
        w[d.triangles()["nodes"].astype(np.int64).ravel()] = 1.0
        state["structures"].append(s)
        state["targets"].append(x + rng.normal(0.0, 2.0e-3, x.shape))
        state["weights"].append(w)
        state["rollouts"].append(sw.Rollout(s, case["steps"], 16))
    return state


def prepare(case, seed):
    state = {"cloth": _prepare_cloth, "wing": _prepare_wing, "contact": _prepare_contact, "batch": _prepare_batch,
             "gradient": _prepare_gradient}[case["kind"]](case, seed)
    state["case"] = dict(case)
    return state


# ---- one pass --------------------------------------------------------------------
def _diagnostics(d):
    """The diagnostics as plain numbers."""
    return {"active_contacts": int(d.active_contact_count), "finite": int(d.finite),
            "center_of_mass": np.array([d.center_of_mass.x, d.center_of_mass.y, d.center_of_mass.z]),
            "momentum": np.array([d.linear_momentum.x, d.linear_momentum.y, d.linear_momentum.z]),
            "kinetic_energy": d.kinetic_energy, "distance_error": d.maximum_distance_error,
            "cable_extension": d.maximum_cable_extension, "membrane_strain": d.maximum_absolute_membrane_strain}


def _pilot(s):
    p = s.suspension_state()
    return np.concatenate([p.center_of_mass, p.body_to_world, p.linear_velocity, p.angular_velocity])


def run(state):
    case, settings = state["case"], state["settings"]
    kind = case["kind"]
    if kind == "cloth":
        s = state["structure"]
        s.step_many(settings, case["steps"])
        return {"nodes": s.node_states()}
    if kind == "wing":
        s = state["structure"]
        if case["steps"] > 1:
            s.step_many(settings, case["steps"])
            return {"nodes": s.node_states(), "pilot": _pilot(s)}
        if case["loads"] == "device":
            d = state["coupling"].advance_impulses(state["impulses"], settings.time_step, settings)
        else:
            s.set_external_forces(state["loads"])
            d = s.step(settings)
        return {"nodes": s.node_states(), "pilot": _pilot(s), "diagnostics": _diagnostics(d)}
    if kind == "contact":
        s = state["structure"]
        s.restore(state["image"])
        d = s.step(settings)
        return {"nodes": s.node_states(), "diagnostics": _diagnostics(d)}
    if kind == "batch":
        b = state["batch"]
        b.step(settings, case["steps"])
        return {"nodes": [b.structure(i).node_states() for i in range(len(b))]}
    losses = sw.rollout_forward_many(state["rollouts"], settings, state["targets"], state["weights"])
    return {"losses": losses, "gradients": sw.rollout_backward_many(state["rollouts"])}


# ---- work -------------------------------------------------------------------------
def _counts(case):
    """(nodes, triangles, constraints, dihedrals, membranes) of a case's
    structures together, and iterations a step: the generators' own counts."""
    kind = case["kind"]
    if kind == "cloth":
        defs = [sw.generate_patch(nx=case["nx"], ny=case["ny"])]
    elif kind == "wing":
        defs = [_wing_definition(case, 0)]
    elif kind == "contact":
        defs = [sw.stacked_sheets(n=case["side"], compliance=1.0e-3)]
    elif kind == "gradient":
        defs = [sw.generate_wing(cells=case["cells"], chordwise=case["chordwise"], attachments_per_cell=2)] * case["wings"]
    else:
        defs = [sw.generate_wing(cells=case["cells"], chordwise=case["chordwise"])] * case["wings"]
    c = [d.counts() for d in defs]
    return [sum(x[k] for x in c) for k in ("nodes", "triangles", "constraints", "dihedrals", "membranes")]


def work(case):
    """Per pass: the states in and out (FP32 position, previous position and
    velocity), every constraint record and triangle read once a step; per
    iteration 40 flops a distance-type constraint, 190 a dihedral, 300 a
    membrane element.  A gradient reads the inputs of every projection once
    more in reverse and does its arithmetic three times (forward, taped
    forward, reverse); a contact step adds 400 flops for each of a free
    sheet's features (nine candidates a feature) and iteration."""
    n, t, c, h, m = _counts(case)
    steps = case.get("steps", 1)
    iterations = 8 if case["kind"] == "contact" else 48
    flops = steps * iterations * (40.0 * c + 190.0 * h + 300.0 * m)
    moved = n * (3 * 24.0 + 48.0) + steps * (16.0 * (c + h) + 96.0 * m + 16.0 * t)
    if case["kind"] == "gradient":
        flops *= 3.0
        moved += steps * iterations * (32.0 * c + 64.0 * h)
    if case["kind"] == "contact":
        flops += iterations * 400.0 * 9.0 * 0.5 * (n + 2.5 * t)
    return {"bytes": moved, "flops": flops}


def exact(case, seed):
    """None: the result of a fixed number of Gauss-Seidel sweeps belongs to the
    sweep order, which the solver's schedule chooses, so no value exists
    without it."""
    return None
