"""remc_set_params to another crowder model or cutoff: the next sweep runs that
model's kernels, also those that costly systems take apart on clusters. Each
case is a process of its own, in which no other handle has set those up."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys
import numpy as np
sys.path.insert(0, "tests")
from test_gpu_sweep_groups import _system
from remcdockingsimulator_b200 import synth
from remcdockingsimulator_b200.engine import Engine, make_params
from remcdockingsimulator_b200.model import geometric_ladder

models = {"wall": synth.benchmark_params(), "reference": make_params(),
          "cutoff": make_params()}
models["cutoff"].crowder_cutoff = 15.0
layout, first, then = sys.argv[1:4]
if layout == "apart":
    systems = [_system(k, [20, 25 + k], 10 * k, 6.0, 120.0) for k in range(7)]
    systems.insert(3, _system(11, [250, 260, 240, 230], 80, 6.0, 300.0))
    R = 20
else:  # a replica on clusters of four
    systems, R = [_system(4, [90, 100], 60, 6.0, 220.0)], 5


def state(start):
    n = len(systems)
    with Engine(systems, R, start) as eng:
        eng.set_replica_params([geometric_ladder(290.0, 480.0, R)] * n,
                               np.full(n, 0.9, np.float32), np.full(n, 0.3))
        if start is not models[then]:
            eng.set_params(models[then])
        eng.energy_full()
        eng.run(2, 40, 5)
        return list(eng.download_state()) + [eng.energies()] + list(eng.counters())


for a, b in zip(state(models[first]), state(models[then])):
    assert np.array_equal(a, b)
"""


@pytest.mark.parametrize("layout", ["apart", "spread"])
@pytest.mark.parametrize("first,then", [("wall", "reference"), ("wall", "cutoff"),
                                        ("reference", "wall"), ("reference", "cutoff")])
def test_sweeps_after_set_params(built_lib, layout, first, then):
    r = subprocess.run([sys.executable, "-c", SCRIPT, layout, first, then], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
