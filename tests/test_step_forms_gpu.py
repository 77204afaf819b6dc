"""Forms of the force kernel that a run-time rule selects: offsets per bin of cells with a radius per type, in a
batch, under the variants and from host records; a step from one state to another with a radius per
type; all variants of one world; lists of different grids in turn."""

import numpy as np
import pytest

import oracle
from cellflow_gb300 import inputs
from cellflow_gb300.world import PARTICLE_DTYPE, Batch, ParticleSimulation
from tests.parity import check_step
from tests.test_sparse_list_gpu import scattered

pytestmark = pytest.mark.gpu

T = 5
RADIO = np.linspace(-0.8, 0.6, T).astype(np.float32)


def state(n, pos, types, seed):
    rng = np.random.default_rng(seed)
    pos4, vel4 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos4[:, :3], vel4[:, :3] = pos, rng.normal(0, 0.3, (n, 3))
    pos4[:, 3] = types.view(np.float32)
    return pos4, vel4, rng.integers(0, 300, n).astype(np.int32)


def parameters(n, radius, ratio):
    w = inputs.Workload("forms", n=n, num_types=T, radius=radius, steps=1, seed=n)
    params = w.params()
    params.ratio_with_lfo = ratio
    return params, w.types(), w.table()


def make_world(n, table, radio):
    sim = ParticleSimulation(n, T, 2.0, 2.0, 2.0)
    sim.setForceTable(table)
    sim.setRadioByType(radio)
    return sim


def result(sim):
    return sim.getParticleData().tobytes(), sim.getNeighborCounts().tobytes()


# grids of 0.8 to 2.4 million cells for the largest radius: bins of 4 and 16 cells (at 60,000 particles
# none on the first), and with a ratio of 0 one radius for all
@pytest.mark.parametrize("radius,ratio", [(0.015, 0.5), (0.0115, 0.5), (0.0115, 0.0)])
@pytest.mark.parametrize("n", [1, 33, 700, 3000, 60000])
def test_bins_with_a_radius_per_type(cflib, n, radius, ratio):
    params, types, table = parameters(n, radius, ratio)
    pos4, vel4, prev = state(n, scattered(n, radius, n), types, n + 1)
    sim = make_world(n, table, RADIO)
    sim.set_state(pos4, vel4, prev)
    sim.rollout_forward(params, 1)  # (on the list by cell)
    want = result(sim)
    for variant in (None, 0, 1, 2, 4, 8, 9, 12):
        if variant is not None:
            sim.set_force_variant(variant)
        sim.set_state(pos4, vel4, prev)
        sim.simulate(params, 1)
        assert result(sim) == want, variant
    rec, counts = sim.getParticleData(), sim.getNeighborCounts()
    sim.close()
    if n > 5000:
        return
    step = (pos4[:, :3], vel4[:, :3], types, prev, table, RADIO, params)
    po, vo, ao, co = oracle.step_f32(*step)
    _, _, _, _, mag = oracle.step_f64(*step)
    assert np.array_equal(counts, co)
    check_step(rec, po, vo, ao, mag, params.delta_t, 2.0, f"n={n}")


@pytest.mark.parametrize("pinned", [False, True])
def test_bins_from_host_records(cflib, pinned):
    n = 4000
    params, types, table = parameters(n, 0.0125, 0.4)
    pos4, vel4, _ = state(n, scattered(n, 0.0125, 3), types, 4)
    sim = make_world(n, table, RADIO)
    sim.set_state(pos4, vel4, np.zeros(n, np.int32))
    io = sim.getParticleData()
    if pinned:
        torch = pytest.importorskip("torch")
        keep = torch.empty(n * PARTICLE_DTYPE.itemsize, dtype=torch.uint8).pin_memory()
        keep.numpy().view(PARTICLE_DTYPE)[:] = io
        io = keep.numpy().view(PARTICLE_DTYPE)
    sim.rollout_forward(params, 1)
    want = result(sim)
    sim.set_state(pos4, vel4, np.zeros(n, np.int32))
    sim.step_host(params, io, io)
    assert (io.tobytes(), sim.getNeighborCounts().tobytes()) == want
    sim.close()


@pytest.mark.parametrize("captured", [False, True])
def test_bins_in_a_batch(cflib, captured):
    sizes = [3000, 1, 0, 40, 9000]
    parts, radius = [], 0.0125
    for k, n in enumerate(sizes):
        params, _, _ = parameters(1, radius, 0.0)
        types = inputs.uniform_types(n, T, 50 + k)
        parts.append((scattered(n, radius, 60 + k), types, inputs.gaussian_table(T, 0.0, 0.5, 70 + k)))
    batch = Batch(sizes, T, 2.0, 2.0, 2.0, seed=1)
    batch.set_particles(np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]))
    batch.set_force_tables(np.stack([p[2] for p in parts]))
    if captured:
        batch.capture(params, 2)
        batch.replay()
    else:
        batch.simulate(params, 2)
    got, off = batch.get_state(), batch.offsets
    batch.close()
    for k, (pos, types, table) in enumerate(parts):
        if sizes[k] == 0:
            continue
        sim = make_world(sizes[k], table, np.zeros(T, np.float32))
        sim.set_particles(pos, types)
        sim.rollout_forward(params, 2)
        for x, y in zip(got, sim.get_state()):
            assert np.array_equal(x[off[k]:off[k + 1]], y), k
        sim.close()


# a regular grid, a generic one
@pytest.mark.parametrize("radius", [0.12, 0.5])
@pytest.mark.parametrize("n", [33, 4000])
def test_from_state_to_state_with_a_radius_per_type(cflib, n, radius):
    params, types, table = parameters(n, radius, 0.4)
    pos = inputs.uniform_positions(n, n)
    pos4, vel4, prev = state(n, pos, types, n)
    sim = make_world(n, table, RADIO)
    sim.set_state(pos4, vel4, prev)
    sim.simulate(params, 4)
    want = result(sim)
    for every in (1, 3):
        sim.set_state(pos4, vel4, prev)
        sim.rollout_forward(params, 4, every)
        assert result(sim) == want, every
    sim.set_state(pos4, vel4, prev)
    sim.rollout_forward(params, 1, 1)
    rec, counts = sim.getParticleData(), sim.getNeighborCounts()
    sim.close()
    step = (pos, vel4[:, :3], types, prev, table, RADIO, params)
    po, vo, ao, co = oracle.step_f32(*step)
    _, _, _, _, mag = oracle.step_f64(*step)
    assert np.array_equal(counts, co)
    check_step(rec, po, vo, ao, mag, params.delta_t, 2.0, f"n={n}")


def test_all_variants_give_the_same_bits(cflib):
    n = 30000
    params, types, table = parameters(n, 0.12, 0.0)
    pos4, vel4, prev = state(n, inputs.uniform_positions(n, 19), types, 19)
    got = []
    for variant in range(15):
        sim = make_world(n, table, np.zeros(T, np.float32))
        sim.set_state(pos4, vel4, prev)
        sim.set_force_variant(variant)
        sim.simulate(params, 2)
        got.append(result(sim))
        sim.close()
    assert all(g == got[0] for g in got[1:])


def test_records_of_different_grids_in_turn(cflib):
    """As test_sparse_list_gpu.test_lists_of_different_grids_in_turn, the whole state set before each step."""
    n = 5000
    _, types, table = parameters(n, 0.1, 0.0)
    pos4, vel4, prev = state(n, scattered(n, 0.02, 9), types, 10)

    def step(sim, radius):
        sim.set_state(pos4, vel4, prev)
        sim.simulate(parameters(n, radius, 0.0)[0], 1)
        return result(sim)

    one = make_world(n, table, np.zeros(T, np.float32))
    for radius in (0.1, 0.0125, 0.6, 0.05, 0.02, 0.1):
        one.set_state(pos4, vel4, prev)
        one.proximity_edges(0.03, 5)
        got = step(one, radius)
        fresh = make_world(n, table, np.zeros(T, np.float32))
        assert step(fresh, radius) == got, radius
        fresh.close()
    one.close()


@pytest.mark.parametrize("sizes", [[90000, 59999], [90000, 60000]])
def test_integrator_apart_from_its_line_on(cflib, sizes):
    """From 150,000 particles the integrator is a kernel of its own: a batch of as many gives the bits of its worlds
    alone, which are below."""
    parts = []
    for k, n in enumerate(sizes):
        params, types, table = parameters(n, 0.08, 0.0)
        parts.append((inputs.uniform_positions(n, 5 + k), types, table))
    batch = Batch(sizes, T, 2.0, 2.0, 2.0, seed=1)
    batch.set_particles(np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]))
    batch.set_force_tables(np.stack([p[2] for p in parts]))
    batch.simulate(params, 2)
    got, off = batch.get_state(), batch.offsets
    batch.close()
    for k, (pos, types, table) in enumerate(parts):
        sim = make_world(sizes[k], table, np.zeros(T, np.float32))
        sim.set_particles(pos, types)
        sim.simulate(params, 2)
        for x, y in zip(got, sim.get_state()):
            assert np.array_equal(x[off[k]:off[k + 1]], y), k
        sim.close()
