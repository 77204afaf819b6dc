"""The selections where many particles of a type are in range: around the 16 that a particle's own lanes hold, the
limit of the call, and hundreds (the whole warp's), with crowded and lonely particles side by side; and their time,
which was once several times that of the same particles in many types."""

import time

import numpy as np
import pytest

import oracle
from cellflow_gb300.world import ParticleSimulation

pytestmark = pytest.mark.gpu


def clumps(sizes, seed):
    """Clumps of the given sizes, each within a tenth of the distance 0.1 of its centre, 0.3 apart in x."""
    rng = np.random.default_rng(seed)
    pos = []
    for k, m in enumerate(sizes):
        centre = np.array([0.1 + 0.3 * (k % 6), 0.1 + 0.3 * ((k // 6) % 6), 0.1 + 0.3 * (k // 36)])
        pos.append(centre + rng.uniform(-0.005, 0.005, (m, 3)))
    pos = np.concatenate(pos).astype(np.float32)
    return pos[rng.permutation(len(pos))]


# (with `others`, lonely ones in the far half of the box, the particles are too many for a warp each)
@pytest.mark.parametrize("conn,others", [(0, 0), (1, 0), (2, 0), (5, 0), (8, 0), (9, 0), (16, 0), (0, 9000), (2, 16000), (2, 3000),
                                         (5, 16000), (9, 16000), (16, 9000), (16, 3000)])
@pytest.mark.parametrize("T", [1, 3])
def test_against_the_oracle(cflib, T, conn, others):
    pos = clumps([1, 2, 3, 9, 10, 11, 16, 17, 18, 19, 31, 32, 33, 34, 65, 200, 700, 1, 17, 5], 7 + conn)
    lonely = np.random.default_rng(conn).uniform([0.0, 0.0, 0.9], 2.0, (others, 3)).astype(np.float32)
    pos = np.concatenate([pos, np.minimum(lonely, np.float32(1.9999))])[np.random.default_rng(1).permutation(len(pos) + others)]
    types = np.random.default_rng(conn).integers(0, T, len(pos)).astype(np.uint32)
    sim = ParticleSimulation(len(pos), T, 2.0, 2.0, 2.0)
    sim.set_particles(pos, types)
    want = oracle.proximity_edges(pos, types, 0.1, conn)
    assert np.array_equal(sim.proximity_edges(0.1, conn), want)
    cols = np.full((T, 3), 0.5, np.float32)
    tris, _ = oracle.triangle_mesh(pos, types, 0.08, conn, cols, T)
    assert np.array_equal(sim.triangle_mesh(0.08, conn), tris)
    torch = pytest.importorskip("torch")
    out = torch.zeros(12 * max(len(want), 1), device="cuda")
    torch.cuda.synchronize()
    assert sim.proximity_vertices_device(0.1, conn, cols, out.data_ptr(), 2 * len(want)) == 2 * len(want)
    rows = out.cpu().numpy().reshape(-1, 2, 6)[: len(want)]
    got = sorted(map(tuple, rows[:, :, :3].reshape(-1, 6)))
    assert got == sorted(map(tuple, np.concatenate([pos[want[:, 0]], pos[want[:, 1]]], 1)))
    sim.close()


def test_one_type_is_not_many_times_slower(cflib):
    n = 200_000
    rng = np.random.default_rng(1)
    pos = rng.uniform(0.0, 2.0, (n, 3)).astype(np.float32)
    pos[:, 2] = 1.0 + 0.01 * (pos[:, 2] - 1.0)
    times = []
    for T in (1, 12):
        sim = ParticleSimulation(n, T, 2.0, 2.0, 2.0)
        sim.set_particles(pos, rng.integers(0, T, n).astype(np.uint32))
        calls = []
        for _ in range(6):
            t = time.perf_counter()
            sim.triangle_mesh_device(0.05, 2, np.full((T, 3), 0.5, np.float32), 0, 0)  # (the count alone)
            calls.append(time.perf_counter() - t)
        times.append(min(calls))
        sim.close()
    # (flat world, about 390 in range: 1.1 before the lists by type, 9 then, less than 4 now)
    assert times[0] < 6.0 * times[1], times
