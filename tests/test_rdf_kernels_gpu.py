"""The radial distribution's kernels (each pair once; hits queued 32 at a time) against the FP64
oracle where a queue, a run of cells or the type table can go wrong, through the float4 and
the three-float entry points, before and after the scratch behind their cached lists moved."""

import numpy as np
import pytest

import oracle
from cellflow_gb300 import _lib, inputs
from cellflow_gb300.world import ParticleSimulation

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# one particle, less and more than a queue, cells with hundreds (one clump), a grid of fewer than
# five cells, one bin, and a table of one type
@pytest.mark.parametrize("n,T,bins,r_max,sigma", [(1, 3, 8, 0.2, 0.0), (2, 1, 32, 0.2, 0.05), (33, 2, 16, 0.2, 0.05),
                                                  (700, 5, 32, 0.1, 0.03), (3000, 4, 1, 0.15, 0.0),
                                                  (1500, 3, 20, 0.6, 0.0), (5000, 7, 64, 0.18, 0.0)])
def test_rdf_matches_oracle(cflib, n, T, bins, r_max, sigma):
    rng = np.random.default_rng(n)
    pos = inputs.uniform_positions(n, n)
    if sigma:
        pos = np.mod(rng.normal(0.02, sigma, (n, 3)), 2.0).astype(np.float32)  # across the box's corner
        pos[pos >= 2.0] = 0.0
    types = inputs.uniform_types(n, T, n)
    gh = rng.normal(size=(T, T, bins)).astype(np.float32)
    ref = oracle.rdf_f64(pos, types, T, [2.0, 2.0, 2.0], bins, r_max)
    gref = oracle.rdf_grad_f64(pos, types, T, [2.0, 2.0, 2.0], bins, r_max, gh)
    sim = ParticleSimulation(n, T, 2.0, 2.0, 2.0)
    sim.set_particles(pos, types)
    rows = torch.from_numpy(pos).cuda()
    ghd = torch.from_numpy(gh).cuda()
    hist = torch.empty((T, T, bins), dtype=torch.float32, device="cuda")
    g4, g3 = torch.empty((n, 4), device="cuda"), torch.empty((n, 3), device="cuda")
    torch.cuda.synchronize()
    for moved in (False, True):
        if moved:
            sim.proximity_edges(0.01, 3)  # a far finer grid: the list's offsets move
            sim.rollout_forward(inputs.Workload("r", n=n, num_types=T, radius=0.1, steps=1).params(), 1, 1)
            sim.set_particles(pos, types)
        for call in (lambda: sim.rdf(bins, r_max, hist.data_ptr()),
                     lambda: _lib.check(cflib.cf_rdf_xyz(sim.handle, rows.data_ptr(), bins, r_max, hist.data_ptr()), "")):
            hist.fill_(-1.0)
            torch.cuda.synchronize()
            call()
            sim.sync()
            # as test_adjoint_gpu.test_rdf_matches_oracle
            np.testing.assert_allclose(hist.cpu().numpy(), ref, rtol=2e-4, atol=2e-4 * np.abs(ref).max() + 1e-30)
        sim.rdf_backward(bins, r_max, ghd.data_ptr(), g4.data_ptr())
        _lib.check(cflib.cf_rdf_backward_xyz(sim.handle, rows.data_ptr(), bins, r_max, ghd.data_ptr(), g3.data_ptr()), "")
        sim.sync()
        assert np.array_equal(g4[:, :3].cpu().numpy(), g3.cpu().numpy())
        assert np.linalg.norm(g3.cpu().numpy() - gref) <= 1e-4 * np.linalg.norm(gref)
    sim.close()
