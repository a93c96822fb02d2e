"""Reads of a structure from one thread while another runs a rollout of it: a
rollout leaves the committed state alone, so every read gives that state, and
the loads a forward uploads are the caller's."""
import threading

import numpy as np
import pytest

import simwing_b200 as sw
from tests.conftest import step_settings

pytestmark = pytest.mark.gpu


def test_reads_beside_a_rollout(cuda_device):
    d = sw.generate_patch(nx=97, ny=61)
    st = step_settings(iterations=2)
    s = sw.Structure(d)
    want = s.node_states()
    target = want[:, 0, :] + 0.01
    weights = np.ones(d.node_count)
    rng = np.random.default_rng(3)
    loads = 1.0e-3 * rng.normal(size=(d.node_count, 3))
    stop, wrong = threading.Event(), []

    def read():
        while not stop.is_set():
            got = s.node_states()
            if not np.array_equal(got, want):
                wrong.append(np.abs(got - want).max())

    with sw.Rollout(s, 1, 1) as r:
        s.set_external_forces(loads)
        loss = r.forward(st, target, weights)
        reader = threading.Thread(target=read)
        reader.start()
        try:
            for _ in range(400):
                s.set_external_forces(loads)
                assert r.forward(st, target, weights) == loss
        finally:
            stop.set()
            reader.join()
    assert not wrong
