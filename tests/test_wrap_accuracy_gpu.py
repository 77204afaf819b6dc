"""Forces across the box's x face.  A displacement between the last cells of a row and its first is that
of the two positions one period apart, rounded at the scale of a cell and not of the box, also
where an item holds homes of both ends of the row."""

import numpy as np
import pytest

import oracle
from cellflow_gb300.world import ParticleSimulation, SimulationParams

pytestmark = pytest.mark.gpu

# of the size of the terms: displacement and square 4 roundings, square root and exponential 2^-22 each with
# an argument of at most 2 rounded three times, weight, scale and sums 6 more: less than 20 of 2^-23
TOLERANCE = 20 * 2.0**-23


def row_pairs(extent, radius, crowd, rng):
    """In every third row of cells of a plane one pair across the x face, at 1 to 40 % of the radius; with
    crowd also as many particles in the first cell as an item holds, and some along the row."""
    step = 3.3 * radius
    pos = []
    for y in np.arange(0.5 * step, extent - step, step):
        gap = radius * rng.uniform(0.01, 0.4)
        left = gap * rng.uniform(0.1, 0.9)
        yz = np.array([y, 0.5 * extent])
        pos.append([extent - (gap - left), *yz])
        pos.append([left, *(yz + rng.uniform(-0.05, 0.05, 2) * radius)])
        for _ in range(crowd):
            pos.append([rng.uniform(0.0, 0.9) * radius, *(yz + rng.uniform(-0.4, 0.4, 2) * radius)])
        for x in rng.uniform(2.2 * radius, extent, 6 if crowd else 0):
            pos.append([x, *(yz + rng.uniform(-0.4, 0.4, 2) * radius)])
    pos = np.array(pos).astype(np.float32)
    pos[pos >= extent] = 0.0
    return pos


@pytest.mark.parametrize("extent,radius", [(2.0, 0.1), (2.0, 0.3), (8000.0, 285.0), (8000.0, 60.0)])
@pytest.mark.parametrize("crowd", [0, 33])
@pytest.mark.parametrize("ratio", [0.0, 0.4])
def test_forces_across_the_face(cflib, extent, radius, crowd, ratio):
    T = 3
    rng = np.random.default_rng(int(radius * 100) + crowd)
    pos = row_pairs(extent, radius, crowd, rng)
    n = len(pos)
    types = rng.integers(0, T, n).astype(np.uint32)
    table = rng.uniform(0.3, 1.0, (T, T)).astype(np.float32)
    radio = np.array([0.0, -0.1, 0.1], np.float32)
    params = SimulationParams(radius=radius, delta_t=0.01, friction=0.51, repulsion=64.83, attraction=3.06, k=29.45,
                              balance=0.79, canvas_width=extent, canvas_height=extent, canvas_depth=extent,
                              num_particle_types=T, ratio_with_lfo=ratio, force_multiplier=2.33,
                              max_expected_neighbors=400)
    sim = ParticleSimulation(n, T, extent, extent, extent)
    sim.set_particles(pos, types)
    sim.setForceTable(table)
    sim.setRadioByType(radio)
    _, _, a64, _, mag = oracle.step_f64(pos, np.zeros_like(pos), types, np.zeros(n, np.int32), table, radio, params)
    _, _, _, co = oracle.step_f32(pos, np.zeros_like(pos), types, np.zeros(n, np.int32), table, radio, params)
    for variant in (0, 5, 12):
        sim.set_particles(pos, types)
        sim.set_force_variant(variant)
        sim.simulate(params, 1)
        assert np.array_equal(sim.getNeighborCounts(), co)
        off = np.abs(sim.getParticleData()["acc"].astype(np.float64) - a64)
        worst = (off / np.maximum(mag, 1e-30)[:, None]).max()
        assert worst <= TOLERANCE, f"variant {variant}: {worst:.2e} of the terms"
    sim.close()
