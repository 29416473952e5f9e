"""The stage kernel that a simulation reports is the one that runs: the names of
the launched kernels, from the profiler in a process of its own."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import json, sys
import numpy as np, torch
from torch.profiler import ProfilerActivity, profile
from hydroflux_b200 import sim
torch.zeros(1, device="cuda")
out = []
for kind, nr, nc in json.loads(sys.argv[1]):
    zero = np.zeros((nr, nc))
    with sim.Simulation(sim.Mesh2D(zero, 1.0, 1.0, 0.03), (zero + 1.0, zero, zero),
                        sim.SimulationConfig()) as s:
        if kind != "created":
            s.set_stage_kernel(kind)
        s.run_steps(1)
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            s.run_steps(2)
            torch.cuda.synchronize()
        names = {e.name.split("::")[1] for e in p.events() if "k_stage_pf" in e.name}
        out.append((s.stage_kernel(), sorted(names)))
print("RESULT" + json.dumps(out))
"""


def launched(cases):
    """(reported kind, geometries of the launched stage kernels) of each (kind, rows,
    columns); kind "created" leaves the choice of the creation alone."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", CHILD, json.dumps(cases)], cwd=ROOT, text=True,
                       capture_output=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.split("RESULT")[1])


# Below, at and above 100 tiles of 32 x 32; there where one, two, three and five
# waves of 32 x 8 tiles are the shorter ones, and thin grids
AUTO = [(64, 64), (200, 300), (288, 320), (1, 3168), (1, 3169), (31, 3200), (320, 320),
        (199, 481), (400, 400), (600, 600), (640, 640), (800, 800)]


def test_reported_kernel_is_the_launched_one():
    cases = [(kind, *shape) for shape in AUTO for kind in ("created", "auto")]
    for case, (kind, names) in zip(cases, launched(cases)):
        assert len(names) == 1, (case, names)
        assert (kind == "tile32") == (names == ["g32"]), (case, kind, names)


def test_forced_kernel_is_the_launched_one():
    """'tile' is the 32 x 8 tile by 256 threads and 'tile32' the 32 x 32 one on
    every grid, those too where auto takes other CTAs: up to 148 tiles of 32 x 4,
    up to 148 and 296 of 32 x 8, and more."""
    cases = [(kind, *shape) for shape in [(1, 1), (48, 64), (160, 200), (256, 256), (400, 400)]
             for kind in ("tile", "tile32")]
    for case, (kind, names) in zip(cases, launched(cases)):
        assert kind == case[0]
        assert names == ["g8" if kind == "tile" else "g32"], (case, names)
