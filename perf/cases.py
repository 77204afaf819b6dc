"""The work that performance is measured on: what a program does with this framework.

A case is one call (or the few calls that belong together) through the public
Python entry points, on inputs made from a seed: the simulation step from the
smallest world to the largest, a batch of worlds, a step on records in host
memory, a pass of the differentiable rollout, the radial distribution, the
proximity graph and the triangle mesh.

The dynamics are chaotic, so every pass starts from the same state: a step case
copies the state back into the world and steps once (an environment that is
reset), and a rollout is a few steps long.
"""

import ctypes
import dataclasses
import math

import numpy as np
import torch

from cellflow_gb300 import _lib
from cellflow_gb300.autograd import phys_tensor, radial_distribution, rollout
from cellflow_gb300.world import PARTICLE_DTYPE, Batch, ParticleSimulation, SimulationParams

# ---- the cases -------------------------------------------------------------------

# `spread` says where the particles are: "uniform" in the box (a start), "blobs": all in a few
# Gaussian blobs, "clumps": half of them in many small clumps (what particle life grows into),
# "spawn": uniform in a central cube of a quarter of the box's side (a fresh application world).
# `ratio` != 0: every type has a radius of its own.  `tune`: the program ran the autotuner.


def listed():
    return [
        # The smallest worlds: one frame's latency, launches included.
        {"name": "step_n2048", "kind": "step", "n": 2048, "types": 6, "radius": 0.1, "extent": 2.0,
         "spread": "uniform", "ratio": 0.0, "tune": False},
        # The application with a preset of its own scale: 8 types with a radius each, canvas 8000.
        {"name": "step_app_n10000", "kind": "step", "n": 10000, "types": 8, "radius": 285.0, "extent": 8000.0,
         "spread": "spawn", "ratio": 1.0, "tune": False},
        # The application with the default parameters: a short radius in a wide, nearly empty canvas.
        {"name": "step_defaults_n10000", "kind": "step", "n": 10000, "types": 6, "radius": 42.07, "extent": 8000.0,
         "spread": "spawn", "ratio": 0.0, "tune": False},
        # The headline world, about 40 neighbours each, as a drop-in caller steps it (not tuned).
        {"name": "step_n100k", "kind": "step", "n": 100_000, "types": 8, "radius": 0.092, "extent": 2.0,
         "spread": "uniform", "ratio": 0.0, "tune": False},
        # The largest world, very uneven cells, a long run that tuned first.
        {"name": "step_blobs_n1m", "kind": "step", "n": 1_000_000, "types": 12, "radius": 0.02, "extent": 2.0,
         "spread": "blobs", "ratio": 0.0, "tune": True},
        # An ensemble of uneven worlds stepped together, its step captured in a graph.
        {"name": "batch_64w", "kind": "batch", "worlds": 64, "n_min": 2048, "n_max": 65536, "types": 6, "radius": 0.1,
         "extent": 2.0},
        # A host program that keeps the particles in its own page-locked memory.
        {"name": "host_n100k", "kind": "host", "n": 100_000, "types": 8, "radius": 0.092, "extent": 2.0,
         "spread": "clumps", "ratio": 0.0},
        # Training through the step: the rollout and its adjoint at the training configuration's
        # world size (one step), and a short one with checkpoints (at a time step that lets two
        # roundings of the first step stay close to the last).
        {"name": "rollout_n16384", "kind": "rollout", "n": 16384, "types": 6, "radius": 0.1, "extent": 2.0,
         "spread": "uniform", "dt": 0.01, "steps": 1, "every": 1},
        {"name": "rollout_n4096_k4", "kind": "rollout", "n": 4096, "types": 6, "radius": 0.1, "extent": 2.0,
         "spread": "uniform", "dt": 0.001, "steps": 4, "every": 2},
        # The training loss and its gradient.
        {"name": "rdf_n16384", "kind": "rdf", "n": 16384, "types": 6, "bins": 32, "r_max": 0.2, "extent": 2.0,
         "spread": "uniform"},
        # What is drawn each frame: the proximity graph as an edge list, the triangle mesh as vertices.
        {"name": "proximity_n100k", "kind": "proximity", "n": 100_000, "types": 8, "distance": 0.05, "max_conn": 5,
         "extent": 2.0, "spread": "clumps"},
        {"name": "mesh_n100k", "kind": "mesh", "n": 100_000, "types": 8, "distance": 0.05, "max_conn": 8,
         "extent": 2.0, "spread": "clumps"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _radius_for(neighbours, n, extent):
    return round(extent * min(0.3, (neighbours * 3.0 / (4.0 * math.pi * n)) ** (1.0 / 3.0)), 5)


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "batch", "host", "rollout", "rollout", "rdf", "proximity",
                       "mesh"])
    types = rng.randint(2, 12)
    if kind == "batch":
        return {"kind": kind, "worlds": rng.randint(3, 64), "n_min": 2048, "n_max": _log_int(rng, 4096, 65536),
                "types": rng.randint(3, 8), "radius": 0.1, "extent": 2.0}
    if kind == "step":
        world = rng.choice(["plain", "plain", "blobs", "app", "defaults"])
        tune = rng.random() < 0.3
        if world == "plain":
            n = _log_int(rng, 2048, 700_000)
            radius = _radius_for(math.exp(rng.uniform(0.7, 4.0)), n, 2.0)
            return {"kind": kind, "n": n, "types": types, "radius": radius, "extent": 2.0,
                    "spread": rng.choice(["uniform", "clumps"]), "ratio": 0.0, "tune": tune}
        if world == "blobs":
            return {"kind": kind, "n": _log_int(rng, 30_000, 900_000), "types": types, "radius": 0.02, "extent": 2.0,
                    "spread": "blobs", "ratio": 0.0, "tune": tune}
        n = _log_int(rng, 2048, 50_000)
        if world == "app":
            return {"kind": kind, "n": n, "types": types, "radius": float(rng.randint(60, 285)), "extent": 8000.0,
                    "spread": "spawn", "ratio": round(rng.uniform(0.1, 1.0), 3), "tune": tune}
        return {"kind": kind, "n": n, "types": 6, "radius": 42.07, "extent": 8000.0, "spread": "spawn", "ratio": 0.0,
                "tune": tune}
    if kind == "host":
        n = _log_int(rng, 2048, 300_000)
        return {"kind": kind, "n": n, "types": types, "radius": _radius_for(math.exp(rng.uniform(0.7, 3.7)), n, 2.0),
                "extent": 2.0, "spread": rng.choice(["uniform", "clumps"]), "ratio": rng.choice([0.0, 0.5])}
    if kind == "rollout":
        if rng.random() < 0.5:
            return {"kind": kind, "n": _log_int(rng, 2048, 65536), "types": rng.randint(2, 8), "radius": 0.1,
                    "extent": 2.0, "spread": "uniform", "dt": 0.01, "steps": 1, "every": 1}
        return {"kind": kind, "n": _log_int(rng, 1500, 4096), "types": rng.randint(2, 8), "radius": 0.1, "extent": 2.0,
                "spread": "uniform", "dt": 0.001, "steps": rng.randint(2, 4), "every": rng.randint(1, 3)}
    if kind == "rdf":
        return {"kind": kind, "n": _log_int(rng, 2048, 65536), "types": rng.randint(1, 8), "bins": rng.randint(8, 64),
                "r_max": round(rng.uniform(0.1, 0.2), 3), "extent": 2.0, "spread": rng.choice(["uniform", "clumps"])}
    return {"kind": kind, "n": _log_int(rng, 2048, 300_000), "types": types,
            "distance": round(rng.uniform(0.02, 0.05), 4), "max_conn": rng.randint(1, 12), "extent": 2.0,
            "spread": rng.choice(["uniform", "clumps"])}


# ---- inputs ----------------------------------------------------------------------

CLUMP = 40  # particles of one clump
CLUMP_SIGMA = 0.012  # of it, as a share of the box's side
BLOBS, BLOB_SIGMA = 64, 0.022  # the benchmark draws them at 0.01; within a few steps they spread to about this
SPAWN = 0.25  # side of the spawn cube, as a share of the box's


def _positions(g, n, extent, spread):
    u = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    z = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    if spread == "uniform":
        x = u
    elif spread == "spawn":
        x = 0.5 + SPAWN * (u - 0.5)
    elif spread == "blobs":
        c = torch.rand((BLOBS, 3), generator=g, device="cuda", dtype=torch.float64)
        x = c[torch.arange(n, device="cuda") % BLOBS] + BLOB_SIGMA * z
    else:
        k = max(1, n // (2 * CLUMP))
        c = torch.rand((k, 3), generator=g, device="cuda", dtype=torch.float64)
        at = torch.arange(n, device="cuda")
        x = torch.where((at % 2 == 0)[:, None], c[(at // 2) % k] + CLUMP_SIGMA * z, u)
    x = (torch.remainder(x, 1.0) * extent).float()
    x[x >= extent] = 0.0
    return x


def _world_sizes(case):
    """Particles per world, spread over the logarithm of their range; the case's alone."""
    u = np.random.default_rng(case["worlds"]).random(case["worlds"])
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return np.rint(np.exp(lo + u * (hi - lo))).astype(np.int32)


def _mesh_room(case):
    """Triangles that the caller's vertex buffer has room for."""
    return case["n"] * min(32, case["max_conn"] * (case["max_conn"] - 1) // 2 + 1)


def _inputs(case, seed):
    """Positions, velocities, types, counts of the last step, force table and radius table."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1_000_003 + 17)
    T, extent = case["types"], case["extent"]
    if case["kind"] == "batch":
        sizes = _world_sizes(case)
        n = int(sizes.sum())
        table = 0.5 * torch.randn((case["worlds"], T, T), generator=g, device="cuda")
        spread = "uniform"
    else:
        sizes, n, spread = None, case["n"], case["spread"]
        table = 0.5 * torch.randn((T, T), generator=g, device="cuda")
    pos = _positions(g, n, extent, spread)
    vel = 0.05 * extent * torch.randn((n, 3), generator=g, device="cuda")
    types = torch.randint(0, T, (n,), generator=g, device="cuda", dtype=torch.int32)
    counts = torch.randint(0, 60, (n,), generator=g, device="cuda", dtype=torch.int32)
    radio = 1.8 * torch.rand(T, generator=g, device="cuda") - 0.9
    return {"pos": pos, "vel": vel, "types": types, "counts": counts, "table": table, "radio": radio, "sizes": sizes}


def _params(case):
    app = case["extent"] > 100.0
    return SimulationParams(
        radius=case.get("radius", 0.1), delta_t=case.get("dt", 0.18 if app else 0.01), friction=0.51,
        repulsion=64.83, attraction=3.06, k=29.45, balance=0.79, canvas_width=case["extent"],
        canvas_height=case["extent"], canvas_depth=case["extent"], num_particle_types=case["types"],
        ratio_with_lfo=case.get("ratio", 0.0), force_multiplier=2.33, max_expected_neighbors=400)


class _DeviceArray:
    """A device buffer of a world, for torch.as_tensor; keeps its owner alive."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": typestr, "version": 3}


def _views(handle, owner):
    v = _lib.DeviceView()
    _lib.check(_lib.load().cf_device_buffers(handle, ctypes.byref(v)), "cf_device_buffers")

    def view(ptr, shape, typestr):
        return torch.as_tensor(_DeviceArray(ptr, shape, typestr, owner), device="cuda")

    n = int(v.n)
    return {"pos4": view(v.pos4, (n, 4), "<f4"), "vel4": view(v.vel4, (n, 4), "<f4"),
            "acc4": view(v.acc4, (n, 4), "<f4"), "counts": view(v.counts, (n,), "<i4")}


_STREAM = []


def _stream():
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def _state4(x, types=None):
    out = torch.zeros((x.shape[0], 4), device="cuda")
    out[:, :3] = x
    if types is not None:
        out[:, 3] = types.view(torch.float32)
    return out


def _world(case, inp):
    n, T, extent = case["n"], case["types"], case["extent"]
    sim = ParticleSimulation(n, T, extent, extent, extent)
    if case.get("ratio", 0.0):
        sim.setRadioByType(inp["radio"].cpu().numpy())
    else:
        sim.setRadioByType(np.zeros(T, np.float32))
    sim.setForceTable(inp["table"].cpu().numpy())
    return sim


def _reset_set(views, pos4, vel4, counts):
    """(buffers, values) of a reset, all as float32 words (one copy kernel moves them)."""
    return ([views["pos4"], views["vel4"], views["counts"].view(torch.float32)],
            [pos4, vel4, counts.view(torch.float32)])


def prepare(case, seed):
    kind = case["kind"]
    inp = _inputs(case, seed)
    params = _params(case)
    if kind == "batch":
        batch = Batch(inp["sizes"], case["types"], case["extent"], case["extent"], case["extent"])
        batch.set_stream(_stream().cuda_stream)
        batch.set_particles(inp["pos"].cpu().numpy(), inp["types"].cpu().numpy(), inp["vel"].cpu().numpy())
        batch.set_force_tables(inp["table"].cpu().numpy())
        batch.autotune(params, 2)
        batch.capture(params, 1)
        batch.sync()
        views = _views(batch.world_handle(), batch)
        s = {"batch": batch, "views": views,
             "reset": _reset_set(views, views["pos4"].clone(), views["vel4"].clone(), inp["counts"])}
        torch.cuda.synchronize()
        return s
    sim = _world(case, inp)
    if kind in ("rollout", "rdf"):
        sim.set_particles(inp["pos"].cpu().numpy(), inp["types"].cpu().numpy())
        leaf = lambda x: x.detach().clone().requires_grad_(True)  # noqa: E731
        s = {"sim": sim, "params": params, "pos": leaf(inp["pos"])}
        g = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 5)
        if kind == "rdf":
            s.update(bins=case["bins"], r_max=case["r_max"],
                     ghist=torch.randn((case["types"], case["types"], case["bins"]), generator=g, device="cuda"))
            return s
        s.update(vel=leaf(inp["vel"]), table=leaf(inp["table"]),
                 phys=phys_tensor(params, torch.float32).requires_grad_(True), steps=case["steps"],
                 every=case["every"], counts=inp["counts"], views=_views(sim.handle, sim),
                 gpos=torch.randn((case["n"], 3), generator=g, device="cuda"),
                 gvel=torch.randn((case["n"], 3), generator=g, device="cuda"))
        return s
    if kind == "host":
        rec = np.zeros(case["n"], PARTICLE_DTYPE)
        rec["pos"], rec["vel"] = inp["pos"].cpu().numpy(), inp["vel"].cpu().numpy()
        rec["ptype"] = inp["types"].cpu().numpy()
        pinned = [torch.empty(44 * case["n"], dtype=torch.uint8).pin_memory().numpy().view(PARTICLE_DTYPE)
                  for _ in range(2)]
        pinned[0][:] = rec
        return {"sim": sim, "params": params, "in": pinned[0], "out": pinned[1]}
    sim.set_stream(_stream().cuda_stream)
    sim.set_particles(inp["pos"].cpu().numpy(), inp["types"].cpu().numpy(), inp["vel"].cpu().numpy())
    if kind == "proximity":
        return {"sim": sim, "distance": case["distance"], "max_conn": case["max_conn"],
                "edges": np.zeros((case["n"] * case["max_conn"], 2), np.int32)}
    if kind == "mesh":
        colors = [tuple(c) for c in np.random.default_rng(seed).random((case["types"], 3)).astype(np.float32).tolist()]
        return {"sim": sim, "distance": case["distance"], "max_conn": case["max_conn"], "colors": colors,
                "vertices": torch.zeros((3 * _mesh_room(case), 9), device="cuda")}
    if case["tune"]:
        sim.autotune(params, 3)
    views = _views(sim.handle, sim)
    s = {"sim": sim, "params": params, "views": views,
         "reset": _reset_set(views, _state4(inp["pos"], inp["types"]), _state4(inp["vel"]), inp["counts"])}
    torch.cuda.synchronize()
    return s


# ---- one pass --------------------------------------------------------------------


def _stepped(views):
    return {"pos": views["pos4"][:, :3], "vel": views["vel4"][:, :3], "acc": views["acc4"][:, :3],
            "counts": views["counts"]}


def run(state):
    if "batch" in state:
        with torch.cuda.stream(_stream()):
            torch._foreach_copy_(*state["reset"])
        state["batch"].replay()
        return _stepped(state["views"])
    sim = state["sim"]
    if "reset" in state:
        with torch.cuda.stream(_stream()):
            torch._foreach_copy_(*state["reset"])
        sim.simulate(state["params"], 1)
        return _stepped(state["views"])
    if "in" in state:
        out = sim.step_host(state["params"], state["in"], state["out"])
        return {"pos": out["pos"], "vel": out["vel"], "acc": out["acc"], "types": out["ptype"].view(np.int32)}
    if "phys" in state:
        state["views"]["counts"].copy_(state["counts"])
        leaves = [state["pos"], state["vel"], state["table"], state["phys"]]
        pos, vel = rollout(*leaves, sim, state["params"], state["steps"], state["every"])
        grads = torch.autograd.grad([pos, vel], leaves, [state["gpos"], state["gvel"]])
        return {"pos": pos.detach(), "vel": vel.detach(), "grads": list(grads)}
    if "ghist" in state:
        hist = radial_distribution(state["pos"], sim, state["bins"], state["r_max"])
        (gpos,) = torch.autograd.grad([hist], [state["pos"]], [state["ghist"]])
        return {"hist": hist.detach(), "gpos": gpos}
    if "vertices" in state:
        v = state["vertices"]
        count = sim.triangle_mesh_device(state["distance"], state["max_conn"], state["colors"], v.data_ptr(),
                                         v.shape[0])
        return {"vertices": v, "count": count}
    edges, count = state["edges"], ctypes.c_int()
    _lib.check(_lib.load().cf_proximity_edges(sim.handle, state["distance"], state["max_conn"],
                                              ctypes.c_void_p(edges.ctypes.data), len(edges), ctypes.byref(count)),
               "cf_proximity_edges")
    return {"edges": edges, "count": count.value}


# ---- what a pass cannot do without --------------------------------------------------


def _neighbours(n, radius, extent, spread):
    """Mean number of other particles within `radius` of one."""
    ball = 4.0 / 3.0 * math.pi * radius**3 / extent**3

    def gauss(sigma):  # two points of one Gaussian blob are within the radius
        a = radius / (2.0 * sigma * extent)
        return math.erf(a) - 2.0 / math.sqrt(math.pi) * a * math.exp(-a * a)

    if spread == "uniform":
        return n * ball
    if spread == "spawn":
        return n * min(1.0, ball / SPAWN**3)
    if spread == "blobs":
        return n / BLOBS * gauss(BLOB_SIGMA) + n * ball
    return n * ball + 0.5 * CLUMP * gauss(CLUMP_SIGMA)


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: 17 for an interacting pair and 25
    for a particle of a step, 70 and 41 for its adjoint, about 30 for a pair of the radial
    distribution and of its gradient, 8 for a pair within range of the graph and the mesh."""
    kind = case["kind"]
    if kind == "batch":
        sizes = _world_sizes(case).astype(np.float64)
        n = float(sizes.sum())
        pairs = float((sizes**2).sum()) * _neighbours(1, case["radius"], case["extent"], "uniform")
        return {"bytes": 88 * n, "flops": 17 * pairs + 25 * n}
    n, T = case["n"], case["types"]
    radius = case.get("radius") or case.get("r_max") or case.get("distance")
    pairs = n * _neighbours(n, radius, case["extent"], case["spread"])
    if kind == "step":
        return {"bytes": 88 * n, "flops": 17 * pairs + 25 * n}
    if kind == "host":
        return {"bytes": (44 + 44) * n, "flops": 17 * pairs + 25 * n}
    if kind == "rollout":
        k = case["steps"]
        return {"bytes": (4 * 12 + 4 * 12 + 4) * n, "flops": k * ((17 + 70) * pairs + (25 + 41) * n)}
    if kind == "rdf":
        return {"bytes": 12 * n * 2 + 2 * 4 * T * T * case["bins"], "flops": 2 * 30 * pairs}
    same = pairs / T
    if kind == "proximity":
        return {"bytes": 16 * n + 8 * min(same / 2, n * case["max_conn"]), "flops": 8 * same}
    return {"bytes": 16 * n + 108 * min(64 * n, n * (same / n) ** 2 / 6), "flops": 8 * same}


# ---- the same in 64 bits, in plain torch -------------------------------------------


def _f32(x):
    return float(np.float32(x))


def _chunks(pos, extent, cutoff, periodic):
    """(home indices, candidate indices) so that every pair within `cutoff` is in one of them: homes
    in x order, candidates the particles whose x is near enough."""
    n = pos.shape[0]
    x, order = torch.sort(pos[:, 0].double())
    ring = torch.cat([x - extent, x, x + extent]) if periodic else x
    base = n if periodic else 0
    a = 0
    while a < n:
        b = min(n, a + 4096)
        while True:
            lo = int(torch.searchsorted(ring, x[a] - 1.001 * cutoff))
            hi = int(torch.searchsorted(ring, x[b - 1] + 1.001 * cutoff))
            lo, hi = (lo - base, hi - base) if periodic else (lo, hi)
            m = min(n, hi - lo)
            if (b - a) * m <= 2e8 or b - a <= 32:
                break
            b = a + (b - a) // 2
        yield order[a:b], order[torch.arange(lo, lo + m, device=pos.device) % n]
        a = b


def _image(d, extent):
    d = torch.where(d > extent * 0.5, d - extent, d)
    return torch.where(d < -extent * 0.5, d + extent, d)


def _square32(pos, i, j, extent, periodic):
    """The squared distance as the 32-bit definition rounds it, homes x candidates."""
    out = None
    for a in range(3):
        d = pos[j, a][None, :] - pos[i, a][:, None]
        d = _image(d, extent) if periodic else d
        d = d * d
        out = d if out is None else out + d
    return out


def _radii32(case, radio):
    r = np.float32(case["radius"])
    per = (r * (np.float32(1.0) + radio * np.float32(case.get("ratio", 0.0)))).astype(np.float32)
    return torch.from_numpy(((per[:, None] + per[None, :]) * np.float32(0.5)).astype(np.float32)).cuda()


def _pairs(pos, types, eff, extent):
    """Interacting pairs (i, j), decided by the 32-bit definition, a part at a time."""
    cutoff = float(eff.max())
    for i, j in _chunks(pos, extent, cutoff, True):
        near = torch.sqrt(_square32(pos, i, j, extent, True) + 0.0001) < eff.max()
        p, q = torch.nonzero(near & (i[:, None] != j[None, :]), as_tuple=True)
        p, q = i[p], j[q]
        d = [_image(pos[q, a] - pos[p, a], extent) for a in range(3)]
        s = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
        keep = torch.sqrt(s + 0.0001) < eff[types[p].long(), types[q].long()]
        yield p[keep], q[keep]


def _force(pos, types, table, eff, c, p, q, extent):
    d = _image(pos[q] - pos[p], extent)
    dist = torch.sqrt((d * d).sum(1) + _f32(0.0001))
    a, b = types[p].long(), types[q].long()
    r = dist / eff[a, b].double()
    net = table[a, b] * (c["repulsion"] * torch.exp(-c["k"] * r * r) - c["attraction"] * r)
    return d / dist[:, None] * net[:, None]


def _constants(params):
    return {k: _f32(v) for k, v in dataclasses.asdict(params).items()}


def _integrate(pos, vel, force, count, prev, c, extent):
    density = torch.clamp((count + prev).double() * 0.5 / c["max_expected_neighbors"], max=1.0)
    acc = force * (c["force_multiplier"] * (1.0 - (1.0 - c["balance"]) * density))[:, None]
    v = vel * c["friction"] + acc * c["delta_t"]
    return torch.fmod(pos + v * c["delta_t"] + extent, extent), v, acc


def _exact_step(case, inp, prev, sizes=None):
    pos32, types, extent = inp["pos"], inp["types"], case["extent"]
    c = _constants(_params(case))
    eff = _radii32(case, inp["radio"].cpu().numpy())
    n = pos32.shape[0]
    force = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    count = torch.zeros(n, dtype=torch.int64, device="cuda")
    starts = [0, n] if sizes is None else [0, *np.cumsum(sizes).tolist()]
    for k in range(len(starts) - 1):
        own = slice(starts[k], starts[k + 1])
        pos, ty = pos32[own], types[own]
        table = (inp["table"] if sizes is None else inp["table"][k]).double()
        pd = pos.double()
        for p, q in _pairs(pos, ty, eff, extent):
            for u in range(0, p.numel(), 1 << 24):
                a, b = p[u:u + (1 << 24)], q[u:u + (1 << 24)]
                force[own].index_add_(0, a, _force(pd, ty, table, eff, c, a, b, extent))
                count[own].index_add_(0, a, torch.ones_like(a))
    x, v, a = _integrate(pos32.double(), inp["vel"].double(), force, count, prev, c, extent)
    return {"pos": x, "vel": v, "acc": a}


def _exact_rollout(case, inp, seed):
    params, extent = _params(case), case["extent"]
    c = _constants(params)
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 5)
    gpos = torch.randn((case["n"], 3), generator=g, device="cuda")
    gvel = torch.randn((case["n"], 3), generator=g, device="cuda")
    pos = inp["pos"].double().requires_grad_(True)
    vel = inp["vel"].double().requires_grad_(True)
    table = inp["table"].double().requires_grad_(True)
    phys = phys_tensor(params, torch.float32).double().cuda().requires_grad_(True)
    for k, name in enumerate(("repulsion", "attraction", "k", "force_multiplier", "balance", "friction")):
        c[name] = phys[k]
    eff = _radii32(case, np.zeros(case["types"], np.float32))
    x, v, prev = pos, vel, inp["counts"].long()
    for _ in range(case["steps"]):
        force = torch.zeros_like(x)
        count = torch.zeros(case["n"], dtype=torch.int64, device="cuda")
        for p, q in _pairs(x.detach().float(), inp["types"], eff, extent):
            force = force.index_add(0, p, _force(x, inp["types"], table, eff, c, p, q, extent))
            count.index_add_(0, p, torch.ones_like(p))
        x, v, _ = _integrate(x, v, force, count, prev, c, extent)
        prev = count
    grads = torch.autograd.grad([x, v], [pos, vel, table, phys], [gpos.double(), gvel.double()])
    return {"pos": x.detach(), "vel": v.detach(), "grads": list(grads)}


def _exact_rdf(case, inp, seed):
    T, bins, r_max, extent = case["types"], case["bins"], case["r_max"], case["extent"]
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 5)
    ghist = torch.randn((T, T, bins), generator=g, device="cuda").double()
    width = _f32(r_max) / bins
    cut = _f32(r_max) + 1.5 * width
    pos, types = inp["pos"].double(), inp["types"].long()
    amount = torch.bincount(types, minlength=T).double()
    centre = (torch.arange(bins, device="cuda").double() + 0.5) * width
    norm = amount[:, None, None] * (amount[None, :, None] / extent**3) * 4.0 * math.pi * centre**2 * width
    weight = torch.where(norm > 0, ghist / norm, torch.zeros_like(norm))
    hist = torch.zeros(T * T * bins, dtype=torch.float64, device="cuda")
    gpos = torch.zeros_like(pos)
    for i, j in _chunks(inp["pos"], extent, cut, True):
        near = _square32(inp["pos"], i, j, extent, True) < cut * cut
        p, q = torch.nonzero(near & (i[:, None] != j[None, :]), as_tuple=True)
        p, q = i[p], j[q]
        for u in range(0, p.numel(), 1 << 22):
            a, b = p[u:u + (1 << 22)], q[u:u + (1 << 22)]
            d = _image(pos[b] - pos[a], extent)
            r = d.norm(dim=1).requires_grad_(True)
            t = r / width - 0.5
            first = torch.floor(t.detach()).long() - 1
            row = types[a] * T + types[b]
            back = types[b] * T + types[a]
            total = torch.zeros((), dtype=torch.float64, device="cuda")
            for o in range(4):
                k = first + o
                z = (t - k).abs()
                w = torch.where(z < 1, 2.0 / 3.0 - z * z + 0.5 * z**3, torch.clamp(2.0 - z, min=0.0)**3 / 6.0)
                inside = (k >= 0) & (k < bins)
                at = k.clamp(0, bins - 1)
                w = torch.where(inside, w, torch.zeros_like(w))
                hist.index_add_(0, row * bins + at, w.detach())
                flat = weight.reshape(-1)
                total = total + (w * (flat[row * bins + at] + flat[back * bins + at])).sum()
            (gr,) = torch.autograd.grad(total, r)
            gpos.index_add_(0, a, -gr[:, None] * d / r.detach()[:, None].clamp(min=1e-300))
    hist = hist.reshape(T, T, bins)
    return {"hist": torch.where(norm > 0, hist / norm, torch.zeros_like(hist)), "gpos": gpos}


def _exact_mesh(case, inp, seed):
    n, T = case["n"], case["types"]
    pos, types = inp["pos"], inp["types"]
    keep = min(case["max_conn"], 32)
    dsq = np.float32(case["distance"]) * np.float32(case["distance"]) * (np.float32(1.2) * np.float32(1.2))
    found = []
    for i, j in _chunks(pos, case["extent"], math.sqrt(float(dsq)), False):
        near = (_square32(pos, i, j, case["extent"], False) < float(dsq)) & (types[i][:, None] == types[j][None, :])
        p, q = torch.nonzero(near & (i[:, None] != j[None, :]), as_tuple=True)
        found.append(i[p] * n + j[q])
    pair = torch.sort(torch.cat(found)).values
    i, j = pair // n, pair % n
    first = torch.searchsorted(i, torch.arange(n, device="cuda"))
    rank = torch.arange(i.numel(), device="cuda") - first[i]
    i, j = i[(rank < keep) & (j > i)], j[(rank < keep) & (j > i)]
    first = torch.searchsorted(i, torch.arange(n, device="cuda"))
    lists = torch.full((n, keep), -1, dtype=torch.int64, device="cuda")
    lists[i, torch.arange(i.numel(), device="cuda") - first[i]] = j
    a, b = torch.triu_indices(keep, keep, 1, device="cuda")
    ok = (lists[:, a] >= 0) & (lists[:, b] >= 0)
    ok &= ok.cumsum(1) <= 64
    home, which = torch.nonzero(ok, as_tuple=True)
    corner = [home, lists[home, a[which]], lists[home, b[which]]]
    x = [pos[c].double() for c in corner]
    normal = torch.linalg.cross(x[1] - x[0], x[2] - x[0])
    length = normal.norm(dim=1, keepdim=True)
    normal = torch.where(length > 0.0001, normal / length.clamp(min=1e-300), normal)
    colors = torch.from_numpy(np.random.default_rng(seed).random((T, 3)).astype(np.float32)).cuda().double()
    colour = colors[types[home].long()]
    vertices = torch.zeros((3 * _mesh_room(case), 9), dtype=torch.float64, device="cuda")
    vertices[:3 * home.numel()] = torch.stack([torch.cat([v, normal, colour], 1) for v in x], 1).reshape(-1, 9)
    return {"vertices": vertices, "count": None}


def exact(case, seed):
    """What run() returns, in 64 bits.  Which pairs interact is part of the definition and is decided
    by its 32-bit test, as the whole-number outputs are."""
    inp = _inputs(case, seed)
    kind = case["kind"]
    if kind == "step":
        return {**_exact_step(case, inp, inp["counts"].long()), "counts": None}
    if kind == "batch":
        return {**_exact_step(case, inp, inp["counts"].long(), inp["sizes"]), "counts": None}
    if kind == "host":
        return {**_exact_step(case, inp, torch.zeros_like(inp["counts"]).long()), "types": None}
    if kind == "rollout":
        return _exact_rollout(case, inp, seed)
    if kind == "rdf":
        return _exact_rdf(case, inp, seed)
    if kind == "mesh":
        return _exact_mesh(case, inp, seed)
    return None
