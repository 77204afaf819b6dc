"""The radial distribution's queue of hits: 32 are worked off, the rest moves to the front and the next
hits are stored behind it, over entries that the move left there.  A hit lost or counted
twice shows in every entry checked here: a bin holds some thirty pairs and a gradient's
largest terms are hundredths of it."""

import numpy as np
import pytest

import oracle
from cellflow_gb300.world import ParticleSimulation

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# clumps of a few times the queue's 32 and 64 entries in one cell, all in range of each other, and one
# spread over many cells (runs of a few hits each, so that the queue turns over part full)
@pytest.mark.parametrize("n,sigma", [(31, 0.03), (33, 0.03), (64, 0.03), (65, 0.03), (97, 0.03), (200, 0.03), (700, 0.3)])
def test_no_hit_is_lost_where_the_queue_turns_over(cflib, n, sigma):
    T, bins, r_max = 3, 32, 0.2
    rng = np.random.default_rng(n)
    pos = np.mod(rng.normal(1.0, sigma, (n, 3)), 2.0).astype(np.float32)
    types = rng.integers(0, T, n).astype(np.uint32)
    gh = rng.normal(size=(T, T, bins)).astype(np.float32)
    ref = oracle.rdf_f64(pos, types, T, [2.0, 2.0, 2.0], bins, r_max)
    gref = oracle.rdf_grad_f64(pos, types, T, [2.0, 2.0, 2.0], bins, r_max, gh)
    sim = ParticleSimulation(n, T, 2.0, 2.0, 2.0)
    sim.set_particles(pos, types)
    hist = torch.empty((T, T, bins), dtype=torch.float32, device="cuda")
    grad = torch.empty((n, 4), device="cuda")
    ghd = torch.from_numpy(gh).cuda()
    for _ in range(5):
        torch.cuda.synchronize()
        sim.rdf(bins, r_max, hist.data_ptr())
        sim.rdf_backward(bins, r_max, ghd.data_ptr(), grad.data_ptr())
        sim.sync()
        # 32-bit distances and weights (as test_adjoint_gpu.test_rdf_matches_oracle)
        np.testing.assert_allclose(hist.cpu().numpy(), ref, rtol=2e-4, atol=2e-4 * np.abs(ref).max())
        off = np.linalg.norm(grad[:, :3].cpu().numpy() - gref, axis=1)
        assert off.max() <= 1e-3 * np.linalg.norm(gref, axis=1).max()
    sim.close()
