"""The proximity and mesh selections on the list by type: half a warp per particle, the whole warp for
one with more than 16 candidates in range or more than its limit.  Around those sizes, on grids
coarsened for the type count, with odd particle counts, against the oracle."""

import numpy as np
import pytest

import oracle
from cellflow_gb300 import inputs
from cellflow_gb300.world import ParticleSimulation

pytestmark = pytest.mark.gpu


def case(n, T, spread, seed):
    rng = np.random.default_rng(seed)
    if spread == "clumps":  # a few particles to hundreds of them within the distance
        centres = rng.uniform(0.1, 1.9, (8, 3))
        pos = centres[rng.integers(0, 8, n) ** 2 % 8] + rng.normal(0, 0.02, (n, 3))
    elif spread == "one":  # all within the distance of each other
        pos = 1.0 + rng.uniform(-0.01, 0.01, (n, 3))
    else:
        pos = rng.uniform(0, 2, (n, 3))
    pos = np.clip(pos, 0.0, 1.999).astype(np.float32)
    types = inputs.uniform_types(n, T, seed)
    sim = ParticleSimulation(n, T, 2.0, 2.0, 2.0)
    sim.set_particles(pos, types)
    return sim, pos, types


SHAPES = [(1, 1, "one"), (2, 1, "one"), (16, 1, "one"), (17, 1, "one"), (18, 1, "one"), (33, 1, "one"), (34, 1, "one"),
          (300, 2, "one"), (999, 3, "clumps"), (2001, 32, "clumps"), (5000, 8, "even"), (40001, 5, "clumps")]


@pytest.mark.parametrize("n,T,spread", SHAPES)
@pytest.mark.parametrize("max_conn", [1, 5, 8, 9, 16])
def test_edges_match_oracle(cflib, n, T, spread, max_conn):
    sim, pos, types = case(n, T, spread, n + T)
    got = sim.proximity_edges(0.05, max_conn)
    sim.close()
    assert np.array_equal(got, oracle.proximity_edges(pos, types, 0.05, max_conn))


@pytest.mark.parametrize("n,T,spread", SHAPES)
@pytest.mark.parametrize("max_conn", [1, 2, 8, 16, 17, 32, 40])
def test_mesh_matches_oracle(cflib, n, T, spread, max_conn):
    import torch

    sim, pos, types = case(n, T, spread, n + T)
    colors = ((np.arange(3 * T, dtype=np.float32) + 1) / np.float32(3 * T)).reshape(T, 3)
    tris = sim.triangle_mesh(0.04, max_conn)
    ref, verts = oracle.triangle_mesh(pos, types, 0.04, max_conn, colors, T)
    assert np.array_equal(tris, ref)
    out = torch.full((3 * len(ref) + 3, 9), -7.0, device="cuda")
    torch.cuda.synchronize()
    count = sim.triangle_mesh_device(0.04, max_conn, colors.tolist(), out.data_ptr(), 3 * len(ref))
    sim.close()
    assert count == 3 * len(ref)
    assert np.array_equal(out[:count].cpu().numpy().reshape(-1), np.asarray(verts, np.float32).reshape(-1))
    assert (out[count:] == -7.0).all()
