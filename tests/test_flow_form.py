"""Which sweeps hand nodes over and which reach them in place
(tests/cpp/flow_form_test.cpp), and the plan's check of both directions."""
import os
import shutil
import subprocess

import pytest

import simwing_b200 as sw
from simwing_b200 import abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_forms(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    lib = os.path.join(ROOT, "simwing_b200")
    out = tmp_path / "flow_form_test"
    subprocess.run([cxx, "-std=c++20", "-O1", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "flow_form_test.cpp"), "-L", lib, "-lsimwing_b200",
                    f"-Wl,-rpath,{lib}", "-o", str(out)], check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("ctas", [2, 5, 16])
@pytest.mark.parametrize("flags", [0, abi.OPT_SPLIT_STAGES])
def test_wing_flows_in_both_directions(ctas, flags):
    d = sw.generate_wing(cells=5, chordwise=14, spanwise_per_cell=3, rib_layers=2)
    r, _, _ = sw.plan_schedule(d, sw.SolverOptions(cluster_ctas=ctas, flags=flags))
    assert r.cluster_ctas == ctas
