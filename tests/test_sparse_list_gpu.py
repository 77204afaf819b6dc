"""A grid with far more cells than particles keeps its offsets per bin of several cells of a row.
The step then gives the bits of the step on the list by cell (which a rollout takes), and
matches the oracle."""

import numpy as np
import pytest

import oracle
from cellflow_gb300 import inputs
from cellflow_gb300.world import ParticleSimulation
from tests.parity import check_step

pytestmark = pytest.mark.gpu


def scattered(n, radius, seed):
    """A third each: anywhere, in lines along x (rows of one cell's height), in clumps of about a cell
    (one at the box's corner), so that bins hold none, a few and hundreds."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, 2.0, (n, 3))
    a, b = n // 3, 2 * n // 3
    pos[a:b, 1:] = 1.0 + rng.uniform(-0.1, 0.1, (b - a, 2)) * radius
    centres = np.array([[0.0, 0.0, 0.0], [1.0, 1.0, 1.0], [1.99, 0.3, 0.7]])
    pos[b:] = centres[rng.integers(0, 3, n - b)] + rng.uniform(-1.5, 1.5, (n - b, 3)) * radius
    pos = np.mod(pos, 2.0).astype(np.float32)
    pos[pos >= 2.0] = 0.0
    return pos


# grids of 1.0 to 4.1 million cells (bins of 4 and 16 cells; too many particles for bins at the last size
# on the first grid)
@pytest.mark.parametrize("radius", [0.02, 0.0155, 0.0125])
@pytest.mark.parametrize("n", [1, 31, 33, 700, 3000, 60000])
def test_binned_list_gives_the_same_step(cflib, radius, n):
    T = 5
    w = inputs.Workload("sparse", n=n, num_types=T, radius=radius, steps=1, seed=n)
    params = w.params()
    pos, types, table = scattered(n, radius, n), w.types(), w.table()
    radio = np.zeros(T, np.float32)
    rng = np.random.default_rng(n + 1)
    vel = rng.normal(0, 0.3, (n, 3)).astype(np.float32)
    prev = rng.integers(0, 300, n).astype(np.int32)
    pos4, vel4 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos4[:, :3], vel4[:, :3] = pos, vel
    pos4[:, 3] = types.view(np.float32)
    sim = ParticleSimulation(n, T, 2.0, 2.0, 2.0)
    sim.setForceTable(table)
    sim.setRadioByType(radio)
    got = []
    for step in (lambda: sim.simulate(params, 1), lambda: sim.rollout_forward(params, 1)):
        sim.set_state(pos4, vel4, prev)
        step()
        got.append((sim.getParticleData(), sim.getNeighborCounts()))
    sim.close()
    assert got[0][0].tobytes() == got[1][0].tobytes()
    assert np.array_equal(got[0][1], got[1][1])
    if n > 5000:
        return
    po, vo, ao, co = oracle.step_f32(pos, vel, types, prev, table, radio, params)
    _, _, _, _, mag = oracle.step_f64(pos, vel, types, prev, table, radio, params)
    assert np.array_equal(got[0][1], co)
    check_step(got[0][0], po, vo, ao, mag, params.delta_t, 2.0, f"n={n}")


def test_lists_of_different_grids_in_turn(cflib):
    """Every build leaves the populations at zero for the next, whatever grid that has: steps on a grid by
    cell, on one by bins and on a generic one, with the graph's and the mesh's lists by type between
    them, give what fresh worlds give."""
    n, T = 5000, 5
    w = inputs.Workload("turns", n=n, num_types=T, radius=0.1, steps=1, seed=9)
    pos, types, table = scattered(n, 0.02, 9), w.types(), w.table()

    def world():
        sim = ParticleSimulation(n, T, 2.0, 2.0, 2.0)
        sim.setForceTable(table)
        sim.setRadioByType(np.zeros(T, np.float32))
        sim.set_particles(pos, types)
        return sim

    def step(sim, radius):
        params = inputs.Workload("turns", n=n, num_types=T, radius=radius, steps=1, seed=9).params()
        sim.set_particles(pos, types)
        sim.simulate(params, 1)
        return sim.getParticleData().tobytes(), sim.getNeighborCounts().tobytes()

    one = world()
    for radius in (0.1, 0.0125, 0.6, 0.05, 0.02, 0.1):
        one.set_particles(pos, types)
        edges = one.proximity_edges(0.03, 5)
        got = step(one, radius)
        one.set_particles(pos, types)
        fresh = world()
        assert np.array_equal(edges, fresh.proximity_edges(0.03, 5))
        fresh.close()
        fresh = world()
        want = step(fresh, radius)
        assert got[1] == want[1]
        fresh.close()
    one.close()
