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


# list lengths around whole groups and units; a clump in the open, across the box's corner
# (every segment shifted), across one face, with a radius per type, and on a generic grid
@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 255, 256, 257, 288, 511, 512, 513, 1100])
@pytest.mark.parametrize("where,radius,ratio", [((1.1, 0.9, 1.3), 0.1, 0.0), ((0.0, 0.0, 0.0), 0.1, 0.0),
                                                ((0.7, 2.0, 1.0), 0.1, 0.5), ((0.0, 1.0, 2.0), 0.55, 0.3)])
def test_unit_edges_match_oracle_and_variants_agree(cflib, m, where, radius, ratio):
    T = 5
    w = inputs.Workload("units", n=m, num_types=T, radius=radius, steps=1, seed=m)
    params = w.params()
    params.ratio_with_lfo = ratio
    pos, types, table = clump(m, where, m), w.types(), w.table()
    radio = np.linspace(-0.8, 0.7, T).astype(np.float32)
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
    for variant in [None, *range(15)]:
        sim.set_state(pos4, vel4, prev)
        if variant is not None:
            sim.set_force_variant(variant)
        sim.simulate(params, 1)
        got.append((sim.getParticleData(), sim.getNeighborCounts()))
    sim.close()
    for rec, counts in got[1:]:
        assert rec.tobytes() == got[0][0].tobytes()
        assert np.array_equal(counts, got[0][1])
    po, vo, ao, co = oracle.step_f32(pos, vel, types, prev, table, radio, params)
    _, _, _, _, mag = oracle.step_f64(pos, vel, types, prev, table, radio, params)
    assert np.array_equal(got[0][1], co)
    check_step(got[0][0], po, vo, ao, mag, params.delta_t, 2.0, f"m={m}")
