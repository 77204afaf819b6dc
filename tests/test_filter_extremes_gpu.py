"""The candidate filter where its sum cancels most: pairs just inside and just outside the threshold at the
far corner of the widest stencil boxes, where the squares of both points are largest.  No pair that
the exact test keeps may be lost."""

import numpy as np
import pytest

import oracle
from cellflow_gb300.world import ParticleSimulation, SimulationParams

pytestmark = pytest.mark.gpu


# grids of 5 and 6 cells a row with items along the whole row, rows whose box starts at the
# origin (the third of them) and at the far end, and a fine grid; edge of 2 and of 8000
@pytest.mark.parametrize("extent,radius", [(2.0, 0.39), (2.0, 0.32), (2.0, 0.05), (8000.0, 1550.0)])
@pytest.mark.parametrize("row", [2, -1])
def test_pairs_at_the_threshold_are_kept(cflib, extent, radius, row):
    rng = np.random.default_rng(int(1000 * radius) + row)
    cells = int(extent / radius)
    side = extent / cells
    m = 600
    corner = np.array([cells, *([(row % cells) + 1] * 2)]) * side  # the row's far corner
    home = corner - rng.uniform(0.0, 0.3, (m, 3)) * side
    u = rng.normal(size=(m, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    # the threshold on the distance: sqrt(d^2 + 1e-4) < radius
    reach = np.sqrt(radius**2 - 1e-4) * (1.0 + rng.choice([-1e-3, -1e-5, -3e-7, 0.0, 3e-7, 1e-5], m))
    pos = np.concatenate([home, home + u * reach[:, None], [[0.01 * side, corner[1] - 0.5 * side, corner[2] - 0.5 * side]]])
    pos = np.mod(pos, extent).astype(np.float32)
    pos[pos >= extent] = 0.0
    n, T = len(pos), 2
    types = rng.integers(0, T, n).astype(np.uint32)
    table = rng.uniform(-1.0, 1.0, (T, T)).astype(np.float32)
    params = SimulationParams(radius=radius, delta_t=0.01, friction=0.51, repulsion=64.83, attraction=3.06, k=29.45,
                              balance=0.79, canvas_width=extent, canvas_height=extent, canvas_depth=extent,
                              num_particle_types=T, ratio_with_lfo=0.0, force_multiplier=2.33,
                              max_expected_neighbors=400)
    radio = np.zeros(T, np.float32)
    _, _, _, co = oracle.step_f32(pos, np.zeros_like(pos), types, np.zeros(n, np.int32), table, radio, params)
    sim = ParticleSimulation(n, T, extent, extent, extent)
    sim.set_particles(pos, types)
    sim.setForceTable(table)
    sim.setRadioByType(radio)
    sim.simulate(params, 1)
    assert np.array_equal(sim.getNeighborCounts(), co)
    sim.close()
