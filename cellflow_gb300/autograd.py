"""torch.autograd binding of the differentiable rollout and the soft radial
distribution (cf_rollout_forward / cf_rollout_backward / cf_rdf /
cf_rdf_backward).

A thin binding: torch supplies device memory and the stream, the library's
kernels do the work.  Positions and velocities are (n, 3) float32 CUDA
tensors in the world's particle order; types come from the world.  The force
table is the (T, T) table the step uses (ParticleSimulation.cu:116), and
`phys` holds the six differentiable step parameters in GRAD_PARAMS order.
No counterpart in the reference.
"""

from __future__ import annotations

import ctypes as C

import torch

from ._lib import GRAD_PARAMS, check, load
from .world import ParticleSimulation, SimulationParams


def _current_stream() -> int:
    """The caller's current stream as a handle.  torch.cuda.current_stream() builds a Stream object in about 15 us;
    where this torch has the call that gives the bare handle (which is not public), that one."""
    raw = getattr(torch._C, "_cuda_getCurrentRawStream", None)
    return raw(torch.cuda.current_device()) if raw else torch.cuda.current_stream().cuda_stream


class _Ordered:
    """Runs a block's library calls between the caller's current torch stream's earlier and
    later work: the world's stream waits for the caller's on entry and the caller's for the
    world's on exit, so tensors of the caller's stream can be handed over in both directions."""

    def __init__(self, sim: ParticleSimulation):
        self.sim = sim
        self.stream = _current_stream()

    def __enter__(self):
        check(load().cf_stream_wait(self.sim.handle, self.stream), "cf_stream_wait")

    def __exit__(self, kind, *exc):
        rc = load().cf_stream_signal(self.sim.handle, self.stream)
        if kind is None:  # (else the block's own error is the one to raise)
            check(rc, "cf_stream_signal")
        return False


def _rows(x: torch.Tensor, n: int, copy: bool = False) -> torch.Tensor:
    """x, broadcast as in an assignment (leading dimensions of one dropped), as contiguous (n, 3)
    float32 on the GPU (its own memory with copy)."""
    x = x.detach()
    while x.dim() > 2 and x.shape[0] == 1:
        x = x[0]
    return x.to("cuda", torch.float32, copy=copy).expand(n, 3).contiguous()


class Rollout(torch.autograd.Function):
    """(pos0, vel0, table, phys) -> (pos_K, vel_K) after `steps` steps."""

    @staticmethod
    def forward(ctx, pos, vel, table, phys, sim: ParticleSimulation, params: SimulationParams, steps: int,
                checkpoint_every: int = 16):
        n = sim.getParticleCount()
        p = params.to_c()
        for name, v in zip(GRAD_PARAMS, phys.detach().cpu().tolist()):
            setattr(p, name, v)
        sim.setForceTable(table.detach().to("cpu", torch.float32).numpy())
        x0, v0 = _rows(pos, n), _rows(vel, n)
        xk, vk = torch.empty_like(x0), torch.empty_like(v0)
        with _Ordered(sim):
            check(load().cf_rollout_forward_xyz(sim.handle, C.byref(p), x0.data_ptr(), v0.data_ptr(), steps,
                                                checkpoint_every, xk.data_ptr(), vk.data_ptr()), "cf_rollout_forward")
        ctx.sim = sim
        ctx.table_meta = (table.dtype, table.device)
        ctx.phys_meta = (phys.dtype, phys.device)
        return xk, vk

    @staticmethod
    def backward(ctx, gpos, gvel):
        sim = ctx.sim
        n, T = sim.getParticleCount(), sim.getNumParticleTypes()
        gxk = _rows(gpos, n) if gpos is not None else None
        gvk = _rows(gvel, n) if gvel is not None else None
        gx0, gv0 = (torch.empty((n, 3), dtype=torch.float32, device="cuda") for _ in range(2))
        gF = torch.empty((T, T), dtype=torch.float32, device="cuda")
        gp = torch.empty(len(GRAD_PARAMS), dtype=torch.float32, device="cuda")
        with _Ordered(sim):
            check(load().cf_rollout_backward_xyz(sim.handle, gxk.data_ptr() if gxk is not None else None,
                                                 gvk.data_ptr() if gvk is not None else None, gx0.data_ptr(),
                                                 gv0.data_ptr(), gF.data_ptr(), gp.data_ptr()), "cf_rollout_backward")
        tdt, tdev = ctx.table_meta
        pdt, pdev = ctx.phys_meta
        return gx0, gv0, gF.to(device=tdev, dtype=tdt), gp.to(device=pdev, dtype=pdt), None, None, None, None


class RadialDistribution(torch.autograd.Function):
    """pos (n, 3) -> soft type-resolved radial distribution (T, T, bins)."""

    @staticmethod
    def forward(ctx, pos, sim: ParticleSimulation, bins: int, r_max: float):
        n, T = sim.getParticleCount(), sim.getNumParticleTypes()
        x = _rows(pos, n, copy=True)  # (kept for the backward, whatever becomes of pos)
        hist = torch.empty((T, T, bins), dtype=torch.float32, device="cuda")
        with _Ordered(sim):
            check(load().cf_rdf_xyz(sim.handle, x.data_ptr(), bins, r_max, hist.data_ptr()), "cf_rdf")
        ctx.sim, ctx.bins, ctx.r_max = sim, bins, r_max
        ctx.save_for_backward(x)
        return hist

    @staticmethod
    def backward(ctx, ghist):
        (x,) = ctx.saved_tensors
        gh = ghist.to(torch.float32).contiguous()
        gx = torch.empty_like(x)
        with _Ordered(ctx.sim):
            check(load().cf_rdf_backward_xyz(ctx.sim.handle, x.data_ptr(), ctx.bins, ctx.r_max, gh.data_ptr(),
                                             gx.data_ptr()), "cf_rdf_backward")
        return gx, None, None, None


def rollout(pos, vel, table, phys, sim, params, steps, checkpoint_every=16):
    return Rollout.apply(pos, vel, table, phys, sim, params, steps, checkpoint_every)


def radial_distribution(pos, sim, bins=32, r_max=0.2):
    return RadialDistribution.apply(pos, sim, bins, r_max)


def phys_tensor(params: SimulationParams, dtype=torch.float64) -> torch.Tensor:
    """The differentiable step parameters of `params` in GRAD_PARAMS order."""
    return torch.tensor([float(getattr(params, name)) for name in GRAD_PARAMS], dtype=dtype)
