"""A world's first edge list and mesh: what they allocate, and that the first call (run directly) and the later ones
(from a recorded graph) agree, also where calls alternate."""

import numpy as np
import pytest

from cellflow_gb300 import inputs
from cellflow_gb300._lib import check
from cellflow_gb300.world import ParticleSimulation

pytestmark = pytest.mark.gpu

N, T = 50_000, 8
CUDA_ERROR_MEMORY_ALLOCATION = 2


def make_world():
    sim = ParticleSimulation(N, T, 2.0, 2.0, 2.0)
    sim.set_particles(inputs.blob_positions(N, 400, 0.03, 3), inputs.uniform_types(N, T, 3))
    sim.sync()
    return sim


# slots, counts, tile sums, offsets with populations, output staging: a sixth allocation would fail here
@pytest.mark.parametrize("call", ["proximity_edges", "triangle_mesh"])
def test_first_call_allocates_five_buffers(cflib, call):
    sim = make_world()
    check(cflib.cf_inject_cuda_error(b"cudaMalloc", CUDA_ERROR_MEMORY_ALLOCATION, 5), "")
    try:
        getattr(sim, call)(0.05, 5)
        assert cflib.cf_injection_pending() == 1
    finally:
        cflib.cf_inject_cuda_error(None, 0, 0)
    sim.close()


def test_direct_and_recorded_calls_agree(cflib):
    sim = make_world()
    first = sim.proximity_edges(0.05, 5)
    for _ in range(3):
        assert np.array_equal(sim.proximity_edges(0.05, 5), first)
    other = sim.proximity_edges(0.03, 4)
    assert np.array_equal(sim.proximity_edges(0.05, 5), first)
    assert np.array_equal(sim.proximity_edges(0.03, 4), other)
    sim.set_particles(inputs.blob_positions(N, 400, 0.03, 4), inputs.uniform_types(N, T, 3))
    moved = sim.proximity_edges(0.03, 4)  # (recorded with other positions)
    assert not np.array_equal(moved, other)
    sim.close()
    sim = make_world()
    sim.set_particles(inputs.blob_positions(N, 400, 0.03, 4), inputs.uniform_types(N, T, 3))
    assert np.array_equal(sim.proximity_edges(0.03, 4), moved)
    sim.close()
