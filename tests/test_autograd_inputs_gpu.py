"""Forms of the inputs that the torch binding takes: rows that broadcast to (n, 3), other types."""

import numpy as np
import pytest

from cellflow_gb300 import autograd, inputs
from cellflow_gb300.world import ParticleSimulation

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N, T = 500, 3


# leading dimensions of one, one row or one number for all particles, strided rows, other types, the host
FORMS = {
    "plain": lambda x: x,
    "leading one": lambda x: x[None],
    "leading ones": lambda x: x[None, None],
    "strided": lambda x: torch.cat([x, x], 1)[:, :3],
    "double": lambda x: x.double(),
    "host": lambda x: x.cpu(),
}


@pytest.mark.parametrize("form", list(FORMS))
def test_forms_give_the_plain_rows_results(cflib, form):
    w = inputs.Workload("forms", n=N, num_types=T, radius=0.15, steps=1, seed=8)
    params = w.params()
    sim = ParticleSimulation(N, T, 2.0, 2.0, 2.0)
    sim.set_particles(w.positions(), w.types())
    sim.setRadioByType(np.zeros(T, np.float32))
    table, phys = torch.from_numpy(w.table()), autograd.phys_tensor(params)
    pos = torch.from_numpy(w.positions()).cuda()
    vel = torch.from_numpy(np.random.default_rng(9).normal(0, 0.1, (N, 3)).astype(np.float32)).cuda()
    start = sim.get_state()
    with torch.no_grad():
        want = autograd.rollout(pos, vel, table, phys, sim, params, 1)
        sim.set_state(*start)
        got = autograd.rollout(FORMS[form](pos), FORMS[form](vel), table, phys, sim, params, 1)
        for g, r in zip(got, want):
            assert g.shape == (N, 3) and torch.equal(g, r)
        hist = autograd.radial_distribution(pos, sim, 8, 0.2)
        again = autograd.radial_distribution(FORMS[form](pos), sim, 8, 0.2)
        assert torch.allclose(hist, again, rtol=1e-6)
    sim.close()


@pytest.mark.parametrize("form", [lambda v: v[0], lambda v: v[:1], lambda v: v[0, 0]])
def test_velocities_that_broadcast(cflib, form):
    w = inputs.Workload("forms", n=N, num_types=T, radius=0.15, steps=1, seed=8)
    params = w.params()
    sim = ParticleSimulation(N, T, 2.0, 2.0, 2.0)
    sim.set_particles(w.positions(), w.types())
    sim.setRadioByType(np.zeros(T, np.float32))
    table, phys = torch.from_numpy(w.table()), autograd.phys_tensor(params)
    pos = torch.from_numpy(w.positions()).cuda()
    vel = torch.from_numpy(np.random.default_rng(9).normal(0, 0.1, (N, 3)).astype(np.float32)).cuda()
    start = sim.get_state()
    want = autograd.rollout(pos, form(vel).expand(N, 3).contiguous(), table, phys, sim, params, 1)
    sim.set_state(*start)
    got = autograd.rollout(pos, form(vel), table, phys, sim, params, 1)
    for g, r in zip(got, want):
        assert torch.equal(g, r)
    sim.close()
