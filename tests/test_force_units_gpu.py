"""The force kernel's units: an item's candidate list is cut into units of at most 256, which
1 to 16 warps take in turn.  Around the sizes where a unit or a group of 32 begins, the step
matches the oracle and every variant gives the same bits."""

import numpy as np
import pytest

import oracle
from cellflow_gb300 import inputs
from cellflow_gb300.world import ParticleSimulation
from tests.parity import check_step

pytestmark = pytest.mark.gpu


def clump(m, centre, seed):
    """m particles within 0.04 of a point (wrapped into the box of side 2)."""
    u = np.random.default_rng(seed).uniform(-0.04, 0.04, (m, 3))
    pos = np.mod(np.asarray(centre) + u, 2.0).astype(np.float32)
    pos[pos >= 2.0] = 0.0
    return pos


def run_variants(m, T, pos, radius, ratio, radio, variants):
    """The records and counts of one step per force variant (None: the world's own), with the inputs."""
    w = inputs.Workload("units", n=m, num_types=T, radius=radius, steps=1, seed=m)
    params = w.params()
    params.ratio_with_lfo = ratio
    types, table = w.types(), w.table()
    rng = np.random.default_rng(m + 1)
    vel = rng.normal(0, 0.3, (m, 3)).astype(np.float32)
    prev = rng.integers(0, 300, m).astype(np.int32)
    pos4, vel4 = np.zeros((m, 4), np.float32), np.zeros((m, 4), np.float32)
    pos4[:, :3], vel4[:, :3] = pos, vel
    pos4[:, 3] = types.view(np.float32)
    sim = ParticleSimulation(m, T, 2.0, 2.0, 2.0)
    sim.setForceTable(table)
    sim.setRadioByType(radio)
    got = []
    for variant in variants:
        sim.set_state(pos4, vel4, prev)
        if variant is not None:
            sim.set_force_variant(variant)
        sim.simulate(params, 1)
        got.append((sim.getParticleData(), sim.getNeighborCounts()))
    sim.close()
    return got, (pos, vel, types, prev, table, radio, params)


def check_against_oracle(got, step, what):
    for rec, counts in got[1:]:
        assert rec.tobytes() == got[0][0].tobytes()
        assert np.array_equal(counts, got[0][1])
    po, vo, ao, co = oracle.step_f32(*step)
    _, _, _, _, mag = oracle.step_f64(*step)
    assert np.array_equal(got[0][1], co)
    check_step(got[0][0], po, vo, ao, mag, step[-1].delta_t, 2.0, what)


# list lengths around whole groups and units; a clump in the open, across the box's corner
# (every segment shifted), across one face, with a radius per type, and on a generic grid
@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 255, 256, 257, 288, 511, 512, 513, 1100])
@pytest.mark.parametrize("where,radius,ratio", [((1.1, 0.9, 1.3), 0.1, 0.0), ((0.0, 0.0, 0.0), 0.1, 0.0),
                                                ((0.7, 2.0, 1.0), 0.1, 0.5), ((0.0, 1.0, 2.0), 0.55, 0.3)])
def test_unit_edges_match_oracle_and_variants_agree(cflib, m, where, radius, ratio):
    T = 5
    radio = np.linspace(-0.8, 0.7, T).astype(np.float32)
    got, step = run_variants(m, T, clump(m, where, m), radius, ratio, radio, [None, *range(15)])
    check_against_oracle(got, step, f"m={m}")


# items that span the box in x, on grids of 14, 6 and 5 cells a row and on one of 3 (generic): their end
# cells are in each other's stencil across the edge
@pytest.mark.parametrize("radius", [0.138, 0.32, 0.37, 0.6])
@pytest.mark.parametrize("m", [2, 5, 22, 32, 33, 64, 300])
def test_items_across_the_whole_box(cflib, m, radius):
    rng = np.random.default_rng(m)
    pos = rng.uniform(0.0, 2.0, (m, 3))
    pos[:, 1:] = 1.0 + rng.uniform(-0.3, 0.3, (m, 2)) * radius
    pos[: m // 3, 0] = rng.choice([0.0, 0.01, 1.99, np.nextafter(np.float32(2), np.float32(0))], m // 3)
    got, step = run_variants(m, 4, pos.astype(np.float32), radius, 0.0, np.zeros(4, np.float32), [None, 0, 1, 4, 8, 12])
    check_against_oracle(got, step, f"m={m} radius={radius}")
