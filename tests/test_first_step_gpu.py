"""A process's first step loads the forms of the one force kernel variant it uses (first step of the process / of a
later world, which records its graph again: about 7; 58 with all variants' forms in one unit)."""

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import time
import torch
from cellflow_gb300 import inputs
from cellflow_gb300.world import ParticleSimulation
torch.zeros(1, device="cuda")
torch.cuda.synchronize()
w = inputs.Workload("first", n=2048, num_types=6, radius=0.1, steps=1, seed=3)
times = []
for _ in range(5):
    sim = ParticleSimulation(w.n, w.num_types, 2.0, 2.0, 2.0)
    sim.set_particles(w.positions(), w.types())
    sim.sync()
    t = time.perf_counter()
    sim.simulate(w.params(), 1)
    sim.sync()
    times.append(time.perf_counter() - t)
    sim.close()
print(times[0] / sorted(times[1:])[1])
"""


def test_first_step_loads_one_variant(cflib):
    pytest.importorskip("torch")
    ratios = []
    for _ in range(3):
        out = subprocess.run([sys.executable, "-c", CHILD], cwd=Path(__file__).resolve().parent.parent,
                             capture_output=True, text=True, timeout=300)
        assert out.returncode == 0, out.stderr
        ratios.append(float(out.stdout))
    assert min(ratios) < 20.0, ratios
