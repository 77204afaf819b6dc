"""A rollout steps from one state to the next (checkpoints, the kept states of its last segment, the
world), and once a backward has allocated the lists the next one takes the last segment as the
forward left it.  With and without that, with the world stepped on in between and on a second
backward, the gradients are the same, and the backward leaves the world as it was."""

import numpy as np
import pytest

from tests.test_adjoint_gpu import dev4, make_world

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# one step; a last segment of one step and of several; one, two, three and more segments; an interval
# longer than the rollout
@pytest.mark.parametrize("K,every", [(1, 1), (2, 1), (3, 1), (2, 2), (3, 2), (4, 2), (6, 2), (7, 3), (3, 8)])
@pytest.mark.parametrize("own_stream", [False, True])
# (a radius of 0.55 gives a grid of 3 cells a row)
@pytest.mark.parametrize("n,radius", [(3000, 0.15), (400, 0.55)])
def test_kept_and_replayed_segments_agree(cflib, n, radius, K, every, own_stream):
    sim, params, *_ = make_world(n, 4, radius, 21, 0.03)
    stream = torch.cuda.Stream()
    if own_stream:
        sim.set_stream(stream.cuda_stream)
    start = sim.get_state()
    gx, gv = dev4(np.random.default_rng(1).normal(size=(n, 3))), dev4(np.ones((n, 3)))

    def backward():
        g0, v0 = torch.empty((n, 4), device="cuda"), torch.empty((n, 4), device="cuda")
        before = sim.getParticleData().tobytes(), sim.getNeighborCounts().tobytes()
        gF, gp = sim.rollout_backward(gx.data_ptr(), gv.data_ptr(), g0.data_ptr(), v0.data_ptr())
        torch.cuda.synchronize()
        assert before == (sim.getParticleData().tobytes(), sim.getNeighborCounts().tobytes())
        return g0[:, :3].cpu().numpy(), v0[:, :3].cpu().numpy(), gF, gp

    def forward():
        sim.set_state(*start)
        sim.rollout_forward(params, K, every)

    got = []
    forward()
    got.append(backward())  # replayed: no lists yet
    end = sim.get_state()
    got.append(backward())
    forward()
    got.append(backward())  # kept
    got.append(backward())
    forward()
    sim.simulate(params, 2)
    got.append(backward())  # kept, the world two steps on
    sim.set_state(*start)
    sim.simulate(params, K)
    for x, y in zip(sim.get_state(), end):
        assert np.array_equal(x, y)
    sim.close()
    for other in got[1:]:
        for g, r in zip(other, got[0]):  # table gradients sum double atomics: order may differ
            np.testing.assert_allclose(g, r, rtol=1e-6, atol=1e-7 * np.abs(r).max())


def test_states_with_the_integrator_apart(cflib):
    """From 500,000 particles the integrator is a kernel of its own: it reads the state before the step too."""
    n = 500_000
    sim, params, *_ = make_world(n, 4, 0.02, 5, 0.03)
    start = sim.get_state()
    sim.rollout_forward(params, 3, 2)
    end = sim.get_state()
    sim.set_state(*start)
    sim.simulate(params, 3)
    for x, y in zip(sim.get_state(), end):
        assert np.array_equal(x, y)
    sim.close()
