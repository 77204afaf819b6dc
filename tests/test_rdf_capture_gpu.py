"""The radial distribution and its gradient recorded into a caller's CUDA graph."""

import numpy as np
import pytest

from cellflow_gb300 import autograd, inputs
from cellflow_gb300.world import ParticleSimulation

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N, T, BINS, R_MAX = 3000, 4, 16, 0.15


def positions(seed):
    rows = torch.zeros((N, 4), device="cuda")
    rows[:, :3] = torch.from_numpy(inputs.uniform_positions(N, seed)).cuda()
    return rows


def make_world():
    sim = ParticleSimulation(N, T, 2.0, 2.0, 2.0)
    sim.set_particles(inputs.uniform_positions(N, 1), inputs.uniform_types(N, T, 1))
    return sim


def test_calls_on_a_capturing_stream(cflib):
    sim = make_world()
    stream = torch.cuda.Stream()
    sim.set_stream(stream.cuda_stream)
    pos = positions(2)
    gh = torch.from_numpy(np.random.default_rng(3).normal(size=(T, T, BINS)).astype(np.float32)).cuda()
    hist, grad = torch.zeros((T, T, BINS), device="cuda"), torch.zeros((N, 4), device="cuda")

    def calls():
        sim.rdf(BINS, R_MAX, hist.data_ptr(), pos.data_ptr())
        sim.rdf_backward(BINS, R_MAX, gh.data_ptr(), grad.data_ptr(), pos.data_ptr())

    torch.cuda.synchronize()
    calls()  # (allocates)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        calls()
    for seed in (4, 5):
        pos.copy_(positions(seed))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = hist.clone(), grad.clone()
        hist.zero_()
        grad.zero_()
        torch.cuda.synchronize()
        calls()
        torch.cuda.synchronize()
        assert float(hist.abs().max()) > 0.0
        assert torch.allclose(got[0], hist, rtol=1e-6)  # (32-bit sums in any order)
        assert torch.allclose(got[1], grad, rtol=1e-5, atol=1e-6 * float(grad.abs().max()))
    sim.sync()
    sim.close()


def test_torch_function_in_a_torch_graph(cflib):
    sim = make_world()
    pos = positions(2)[:, :3].contiguous()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        autograd.radial_distribution(pos, sim, BINS, R_MAX)  # (allocates)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        hist = autograd.radial_distribution(pos, sim, BINS, R_MAX)
    pos.copy_(positions(6)[:, :3])
    graph.replay()
    torch.cuda.synchronize()
    want = autograd.radial_distribution(pos, sim, BINS, R_MAX)
    torch.cuda.synchronize()
    assert float(want.abs().max()) > 0.0
    assert torch.allclose(hist, want, rtol=1e-6)
    sim.close()
