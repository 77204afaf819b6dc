"""The selections under a device memory limit: what a list over all types fits in is enough, the lists by type
taking coarser cells (and giving way to other buffers) where memory is short, with the same results."""

import ctypes as C

import numpy as np
import pytest

from cellflow_gb300 import inputs
from cellflow_gb300.world import ParticleSimulation

pytestmark = pytest.mark.gpu

N, T, DISTANCE, CONN = 60_000, 8, 0.05, 5


def in_use(lib):
    v = C.c_size_t()
    assert lib.cf_device_memory_in_use(C.byref(v)) == 0
    return v.value


@pytest.fixture
def limit(cflib):
    yield lambda spare: cflib.cf_set_device_memory_limit(in_use(cflib) + spare)
    cflib.cf_set_device_memory_limit(0)


def make_world():
    sim = ParticleSimulation(N, T, 2.0, 2.0, 2.0)
    sim.set_particles(inputs.blob_positions(N, 500, 0.03, 3), inputs.uniform_types(N, T, 3))
    sim.setForceTable(inputs.gaussian_table(T, 0.0, 0.5, 3))
    sim.setRadioByType(np.zeros(T, np.float32))
    return sim


# bytes of a call's buffers, with the offsets of one grid over all types (floor(2 / 0.05) = 39 or 40 cells a
# row, 33 for the mesh's 1.2 times the distance)
EDGES = 4 * (N * 16 + N + 1 + 2 * N * CONN + 40**3 + 1) + 8 * (40**3 // 2048 + 259)
MESH = 4 * (N * 32 + N + 1 + 33**3 + 1) + 8 * (33**3 // 2048 + 259)


def test_edges_in_what_one_grid_takes(cflib, limit):
    sim = make_world()
    want = sim.proximity_edges(DISTANCE, CONN)
    sim.close()
    sim = make_world()
    limit(EDGES)
    for _ in range(3):
        assert np.array_equal(sim.proximity_edges(DISTANCE, CONN), want)
    sim.close()


def test_mesh_in_what_one_grid_takes(cflib, limit):
    sim = make_world()
    want = sim.triangle_mesh(DISTANCE, 8)
    sim.close()
    sim = make_world()
    limit(MESH + 12 * len(want))
    for _ in range(3):
        assert np.array_equal(sim.triangle_mesh(DISTANCE, 8), want)
    sim.close()


def test_steps_and_selections_in_turn(cflib, limit):
    """Under a limit that holds one grid's offsets beside everything else: every call gives way to the next."""
    params = inputs.Workload("turns", n=N, num_types=T, radius=0.1, steps=1, seed=3).params()

    def calls(sim):
        edges = sim.proximity_edges(DISTANCE, CONN)
        sim.simulate(params, 1)
        edges2 = sim.proximity_edges(DISTANCE, CONN)
        tris = sim.triangle_mesh(DISTANCE, 4)
        sim.simulate(params, 1)
        return edges, edges2, tris, sim.get_state()[0]

    sim = make_world()
    want = calls(sim)
    sim.close()
    sim = make_world()
    # (the step's items, counts and offsets on a grid of 20 cells a row)
    step = 16 * (N // 32 + 1 + 20 * 20) + 4 * (20 * 20 + 1)
    limit(EDGES + MESH + 12 * len(want[2]) + step)
    for g, r in zip(calls(sim), want):
        assert np.array_equal(g, r)
    sim.close()
