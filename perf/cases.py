"""The work that programs have this library do, as timed cases.

Four kinds, each through the package's public entry points:

* ``step``     lattice steps of a :class:`Simulation` (dense grid or compact
               fluid-only storage), the state left on the device;
* ``sparse``   kernel steps on the caller's own compact buffers and adjacency
               list (:class:`SparseKernels`), in the reference's layout;
* ``adjoint``  loss and gradients of a checkpointed rollout through
               ``torch.autograd`` (:class:`RolloutLoss`);
* ``readout``  density and velocity to host memory and the conservation sums.

``exact`` gives the same results in 64 bits with plain torch operations: the
velocity sets, the collision and the streaming are written again below.
"""
import ctypes
import math

import numpy as np
import torch

from lbmminiapp_gb300 import Simulation, cylinder, workloads
from lbmminiapp_gb300.adjoint import RolloutLoss, new_rollout, outlet_weight
from lbmminiapp_gb300.sparse import SparseKernels, build_adjacency

ELEM = {"f64": 8, "f32": 4, "bf16": 2, "f16": 2}
TORCH = {"f64": ("<f8", torch.float64), "f32": ("<f4", torch.float32), "bf16": ("<u2", torch.bfloat16),
         "f16": ("<f2", torch.float16)}
DEVICE = "cuda"


# ------------------------------------------------------------------ cases
def _step(name, nx, ny, nz, lattice, pattern, storage, geometry, tau, arithmetic="auto", fields="none", steps=2,
          compact=False):
    case = {"kind": "step", "nx": nx, "ny": ny, "nz": nz, "lattice": lattice, "pattern": pattern, "storage": storage,
            "arithmetic": arithmetic, "geometry": geometry, "fields": fields, "tau": tau, "steps": steps,
            "compact": compact}
    return dict(case, name=name) if name else case


def _sparse(name, size, lattice, pattern, steps=2):
    case = {"kind": "sparse", "size": size, "lattice": lattice, "pattern": pattern, "steps": steps}
    return dict(case, name=name) if name else case


def _adjoint(name, nx, ny, nz, lattice, storage, adjoint, loss, steps, checkpoint):
    case = {"kind": "adjoint", "nx": nx, "ny": ny, "nz": nz, "lattice": lattice, "storage": storage,
            "adjoint": adjoint, "loss": loss, "tau": 0.7, "steps": steps, "checkpoint": checkpoint}
    return dict(case, name=name) if name else case


def _readout(name, nx, ny, nz, lattice, storage, geometry, steps):
    case = {"kind": "readout", "nx": nx, "ny": ny, "nz": nz, "lattice": lattice, "storage": storage,
            "geometry": geometry, "tau": 0.7, "steps": steps}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest box that is run in earnest (tests, parameter scans): launches and latency
        _step("box32_q19_aa_f64", 32, 32, 32, 19, "aa", "f64", "box", 0.8),
        # the headline path (FP64 storage, in-place AA, periodic Taylor-Green box) at a size far above L2
        _step("box256_q19_aa_f64", 256, 256, 256, 19, "aa", "f64", "box", 0.55),
        # D3Q27 channel between walls, two buffers: the benchmark's 256x128x128 shape, push
        _step("channel_q27_push_f64", 256, 128, 128, 27, "ab_push", "f64", "channel", 0.6),
        # the same path in its pull form, on an odd-sized channel whose rows do not fill their tiles
        _step("channel_q27_pull_f64_odd", 161, 75, 93, 27, "ab_pull", "f64", "channel", 0.6),
        # the reference's own layout, adjacency list and cylinder benchmark, size 4 (1.15 million points)
        _sparse("cylinder4_q19_aa_sparse", 4.0, 19, "aa"),
        # half-precision storage of a large periodic box, where bandwidth is the point of the format
        _step("box320_q19_aa_f16", 320, 320, 320, 19, "aa", "f16", "box", 0.55),
        # porous channel: single-precision storage, walls and a per-cell porosity field
        _step("porous_q19_aa_f32", 128, 64, 64, 19, "aa", "f32", "channel", 0.7, fields="porosity"),
        # flow through a sphere packing in the compact fluid-only storage, with a copy of the state
        # (as taken for a checkpoint) after ten steps
        _step("spheres160_q27_aa_f16", 160, 160, 160, 27, "aa", "f16", "spheres", 0.7, steps=10, compact=True),
        # the arithmetic that reproduces the reference's bits, as used to verify a run
        _step("box128_q19_aa_exact", 128, 128, 128, 19, "aa", "f64", "box", 0.55, arithmetic="f64"),
        # gradient of an outlet velocity with respect to porosity and force, single precision
        _adjoint("adjoint_q19_f32", 128, 64, 64, 19, "f32", "f32", "velocity", 20, 10),
        # the same gradient in double precision (checks, ill-conditioned losses)
        _adjoint("adjoint_q19_f64", 96, 48, 48, 19, "f64", "f64", "velocity", 10, 5),
        # what a run writes out and checks every so often: rho and u to the host, mass and momentum
        _readout("readout_q19_f64", 128, 128, 128, 19, "f64", "box", 3),
    ]


def _dims(rng, lo, hi):
    """Three edges whose product is spread over [lo^3, hi^3] by its logarithm."""
    edge = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.8, 1.2)
    d = [max(8, int(edge * a)), max(8, int(edge * b)), max(8, int(edge / (a * b)))]
    if rng.random() < 0.5:
        d[0] = max(32, d[0] // 32 * 32)
    return d


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "low", "low", "fields", "exact", "spheres", "sparse", "sparse",
                       "adjoint", "adjoint", "readout"])
    lattice = rng.choice([19, 19, 27])
    pattern = rng.choice(["aa", "ab_push", "ab_pull"])
    geometry = rng.choice(["box", "channel"])
    tau = round(rng.uniform(0.55, 1.1), 3)
    if kind == "step":
        return _step(None, *_dims(rng, 24, 210), lattice, pattern, "f64", geometry, tau)
    if kind == "low":
        return _step(None, *_dims(rng, 32, 256), lattice, pattern, rng.choice(["f32", "bf16", "f16"]), geometry, tau)
    if kind == "fields":
        return _step(None, *_dims(rng, 32, 160), lattice, pattern, "f32", "channel", tau,
                     fields=rng.choice(["porosity", "force", "both"]))
    if kind == "exact":
        return _step(None, *_dims(rng, 24, 110), lattice, pattern, "f64", geometry, tau, arithmetic="f64")
    if kind == "spheres":
        n = rng.randrange(80, 161)
        return _step(None, n, n, n, lattice, "aa", rng.choice(["f32", "bf16", "f16"]), "spheres", 0.7, steps=10,
                     compact=True)
    if kind == "sparse":
        return _sparse(None, round(rng.uniform(1.0, 4.5), 2), lattice, pattern)
    if kind == "adjoint":
        real = rng.choice(["f32", "f64"])
        dims = _dims(rng, 24, 80 if real == "f32" else 60)
        steps = rng.randrange(4, 16)
        return _adjoint(None, *dims, lattice, real, real, rng.choice(["velocity", "energy"]), steps,
                        rng.randrange(2, steps + 1))
    return _readout(None, *_dims(rng, 24, 150), lattice, rng.choice(["f64", "f32", "f16"]), geometry,
                    rng.randrange(2, 6))


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _flow(nx, ny, nz, seed, U):
    """Density and velocity of a Taylor-Green vortex of random phase with
    noise, on the device: (nz, ny, nx) and (3, nz, ny, nx)."""
    g = _rng(seed)
    phase = torch.rand(3, generator=g, device=DEVICE, dtype=torch.float64) * 2 * math.pi
    axes = [2 * math.pi / n * torch.arange(n, device=DEVICE, dtype=torch.float64) + phase[d]
            for d, n in enumerate((nx, ny, nz))]
    x, y, z = axes[0][None, None, :], axes[1][None, :, None], axes[2][:, None, None]
    u = 1e-3 * (2 * torch.rand((3, nz, ny, nx), generator=g, device=DEVICE, dtype=torch.float64) - 1)
    u[0] += U * torch.sin(x) * torch.cos(y) * torch.cos(z)
    u[1] -= U * torch.cos(x) * torch.sin(y) * torch.cos(z)
    rho = 1 + 1e-3 * (2 * torch.rand((nz, ny, nx), generator=g, device=DEVICE, dtype=torch.float64) - 1)
    return rho, u


def _field(nx, ny, nz, seed):
    """Porosity: noise smoothed over a few cells, mean 0.15, within [0, 1]."""
    noise = torch.randn((nz, ny, nx), generator=_rng(seed), device=DEVICE, dtype=torch.float64)
    k2 = sum((2 * math.pi * torch.fft.fftfreq(n, device=DEVICE, dtype=torch.float64).reshape(s)) ** 2
             for n, s in ((nz, (-1, 1, 1)), (ny, (1, -1, 1)), (nx, (1, 1, -1))))
    smooth = torch.fft.ifftn(torch.fft.fftn(noise) * torch.exp(-4.5 * k2)).real
    smooth = (smooth - smooth.mean()) / smooth.std()
    return (0.15 + 0.1 * smooth).clamp(0.0, 1.0)


def _force_field(nx, ny, nz, seed):
    return 1e-6 * torch.randn((3, nz, ny, nx), generator=_rng(seed), device=DEVICE, dtype=torch.float64)


def _force(case):
    """Body force along x: drives channels to a peak velocity of 0.03."""
    if case["geometry"] == "channel":
        return 8 * (case["tau"] - 0.5) / 3 * 0.03 / (case["ny"] - 2) ** 2
    return 1e-6 if case["geometry"] == "spheres" else 0.0


def _solid(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["geometry"] == "channel":
        return workloads.channel_mask(nx, ny, nz), (1, 0, 1)
    if case["geometry"] == "spheres":
        return workloads.sphere_packing(nx, 0.35, 6.0, 12.0, seed=seed)[0], (1, 1, 1)
    return None, (1, 1, 1)


class _Memory:
    """Device memory of the library seen as an array (no copy)."""

    def __init__(self, ptr, shape, strides, typestr, owner):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides,
                                         "typestr": typestr, "version": 3}
        self.owner = owner


def _view(sim, ptr, storage, owner):
    """[Q, ncell] tensor over a population buffer (planes are padded)."""
    typestr, dtype = TORCH[storage]
    e = ELEM[storage]
    mem = _Memory(ptr, (sim.Q, sim.ncell), (int(sim.info.plane_stride) * e, e), typestr, owner)
    return torch.as_tensor(mem, device=DEVICE).view(dtype)


def _simulation(case, seed, pattern, arithmetic="auto", compact=False):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    solid, periodic = _solid(case, seed)
    sim = Simulation(nx, ny, nz, lattice=case["lattice"], pattern=pattern, omega=1.0 / case["tau"],
                     force=(_force(case), 0.0, 0.0), periodic=periodic, storage=case["storage"],
                     arithmetic=arithmetic, compact=compact)
    if solid is not None:
        sim.set_solid(solid)
    fields = case.get("fields", "none")
    if fields in ("porosity", "both"):
        sim.set_porosity(_field(nx, ny, nz, seed + 1).cpu().numpy())
    if fields in ("force", "both"):
        sim.set_force_field(_force_field(nx, ny, nz, seed + 2).cpu().numpy())
    rho, u = _flow(nx, ny, nz, seed, 0.05 if case["geometry"] == "box" else 0.01)
    sim.init_equilibrium(rho.cpu().numpy(), u.cpu().numpy())
    return sim


def _cylinder_start(case, seed):
    (nx, ny, nz), solid = cylinder(case["size"])
    rho, u = _flow(nx, ny, nz, seed, 0.01)
    return solid, equilibrium(case["lattice"], rho, u)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        sim = _simulation(case, seed, case["pattern"], case["arithmetic"], case["compact"])
        if case["compact"]:
            # the dense copy that a program saves or post-processes
            out = torch.zeros(int(sim.info.buffer_bytes), dtype=torch.uint8, device=DEVICE)
            ptr = out.data_ptr()
        else:
            out, ptr = None, sim.population_buffer()
        return {"kind": kind, "sim": sim, "steps": case["steps"], "copy": out,
                "view": _view(sim, ptr, case["storage"], out if out is not None else sim)}
    if kind == "sparse":
        solid, f = _cylinder_start(case, seed)
        fluid, adjacency = build_adjacency(solid, (1, 1, 1), case["pattern"], case["lattice"])
        kernels = SparseKernels(adjacency, lattice=case["lattice"], pattern=case["pattern"], omega=1.0,
                                force=(1e-6, 0.0, 0.0))
        buf = raw_layout(f, case["lattice"], case["pattern"])[:, torch.from_numpy(fluid).to(DEVICE)].contiguous()
        buffers = [buf] if case["pattern"] == "aa" else [buf, buf.clone()]
        return {"kind": kind, "kernels": kernels, "buffers": buffers, "steps": case["steps"]}
    if kind == "adjoint":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        solid, weight, window = _loss_weight(case)
        _, u = _flow(nx, ny, nz, seed, 0.01)
        rollout = new_rollout(nx, ny, nz, case["lattice"], case["tau"], solid, (1, 0, 1), case["steps"],
                              case["checkpoint"], case["loss"], weight, window, storage=case["storage"],
                              adjoint=case["adjoint"], u0=u.cpu().numpy())
        porosity, force = _parameters(case, seed)
        return {"kind": kind, "rollout": rollout, "porosity": porosity.requires_grad_(),
                "force": force.requires_grad_()}
    if kind == "readout":
        sim = _simulation(case, seed, "aa")
        sim.step(case["steps"])
        nz, ny, nx = sim.shape
        rho = torch.empty((nz, ny, nx), dtype=torch.float64, pin_memory=True)
        u = torch.empty((3, nz, ny, nx), dtype=torch.float64, pin_memory=True)
        return {"kind": kind, "sim": sim, "rho": rho, "u": u, "out": (rho.numpy(), u.numpy())}
    raise ValueError(kind)


def _loss_weight(case):
    nx, ny, nz, steps = case["nx"], case["ny"], case["nz"], case["steps"]
    solid = workloads.channel_mask(nx, ny, nz)
    window = (steps - steps // 4, steps)
    span = window[1] - window[0] + 1
    if case["loss"] == "velocity":
        return solid, outlet_weight((nz, ny, nx), solid, nx - 1, span), window
    fluid = ~solid.astype(bool)
    return solid, fluid / (fluid.sum() * span), window


def _parameters(case, seed):
    """Porosity and per-cell force, in the precision of the adjoint."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dtype = torch.float32 if case["adjoint"] == "f32" else torch.float64
    force = _force_field(nx, ny, nz, seed + 2)
    force[0] += 1e-5
    return _field(nx, ny, nz, seed + 1).to(dtype), force.to(dtype)


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "step":
        sim = state["sim"]
        sim.step(state["steps"])
        if state["copy"] is not None:
            status = sim.lib.lbm_copy_state(sim.h, ctypes.c_void_p(state["copy"].data_ptr()), 0)
            if status:
                raise RuntimeError("lbm_copy_state: %d" % status)
        return state["view"]
    if kind == "sparse":
        return state["kernels"].run(state["buffers"], state["steps"])
    if kind == "adjoint":
        porosity, force = state["porosity"], state["force"]
        loss = RolloutLoss.apply(porosity.double(), force.double(), state["rollout"])
        grads = torch.autograd.grad(loss, (porosity, force))
        return {"loss": loss.detach().to(porosity.dtype), "porosity": grads[0], "force": grads[1]}
    sums = state["sim"].conserved()
    state["sim"].macros(state["out"])
    return {"rho": state["rho"], "u": state["u"], "sums": sums}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: per step the populations of the fluid cells read and written
    once in their storage format, with the per-cell fields and the
    reference's adjacency list where the step has to read them."""
    Q = case["lattice"]
    kind = case["kind"]
    if kind == "sparse":
        (nx, ny, nz), solid = cylinder(case["size"])
        n = int((solid == 0).sum())
        lists = {"aa": 0.5, "ab_push": 1.0, "ab_pull": 1.0}[case["pattern"]] * 4 * Q
        return {"bytes": n * case["steps"] * (16 * Q + lists), "flops": n * case["steps"] * 14.0 * Q}
    cells = case["nx"] * case["ny"] * case["nz"]
    e = ELEM[case["storage"]]
    if kind == "step":
        if case["geometry"] == "channel":
            cells = case["nx"] * (case["ny"] - 2) * case["nz"]
        elif case["geometry"] == "spheres":
            cells = int(0.65 * cells)
        extra = {"none": 0, "porosity": 1, "force": 3, "both": 4}[case["fields"]] * e
        nbytes = cells * case["steps"] * (2 * Q * e + extra)
        if case["compact"]:
            nbytes += 2 * cells * Q * e   # the copy that is handed out
        return {"bytes": nbytes, "flops": cells * case["steps"] * 14.0 * Q}
    if kind == "adjoint":
        cells = case["nx"] * (case["ny"] - 2) * case["nz"]
        lam = 4 if case["adjoint"] == "f32" else 8
        # forward step, then the adjoint step: state and adjoint state read, adjoint state written
        return {"bytes": cells * case["steps"] * (2 * Q * e + Q * e + 2 * Q * lam),
                "flops": cells * case["steps"] * 42.0 * Q}
    return {"bytes": cells * (2 * Q * e + 32), "flops": cells * 6.0 * Q}


# ------------------------------------------------------------------ 64-bit results
def velocities(Q):
    """Direction order of the population layout."""
    c = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
         (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (-1, 1, 0), (-1, -1, 0),
         (-1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, 1, -1), (0, -1, 1), (0, -1, -1)]
    if Q == 27:
        c += [(a, b, d) for a in (1, -1) for b in (1, -1) for d in (1, -1)]
    return c + [(0, 0, 0)]


def opposites(Q):
    c = velocities(Q)
    return [c.index((-a, -b, -d)) for a, b, d in c]


def weights(Q):
    table = {19: (1 / 3, 1 / 18, 1 / 36), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}[Q]
    return [table[a * a + b * b + d * d] for a, b, d in velocities(Q)]


def _dot(c, v):
    """c . v for a velocity with components -1, 0, 1."""
    total = 0.0
    for k in range(3):
        if c[k]:
            total = total + v[k] if c[k] > 0 else total - v[k]
    return total


def equilibrium(Q, rho, u):
    uu = 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    f = []
    for c, w in zip(velocities(Q), weights(Q)):
        cu = 3 * _dot(c, u)
        f.append(w * rho * (1 + cu + 0.5 * cu * cu - uu))
    return torch.stack(f)


def raw_layout(f, Q, pattern):
    """Slots of a stored buffer from populations by direction, flattened."""
    return (f[opposites(Q)] if pattern == "aa" else f).reshape(Q, -1)


def moments(f, Q):
    rho = f.sum(0)
    c = velocities(Q)
    j = [sum(c[s][d] * f[s] for s in range(Q) if c[s][d]) for d in range(3)]
    return rho, j


def collide(f, Q, tau, F, porosity=None):
    omega = 1.0 / tau
    rho, j = moments(f, Q)
    u = [(j[d] + 0.5 * F[d]) / rho for d in range(3)]
    uu = 3 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    fu = 3 * (F[0] * u[0] + F[1] * u[1] + F[2] * u[2])
    post = []
    for s, (c, w) in enumerate(zip(velocities(Q), weights(Q))):
        cu, cf = 3 * _dot(c, u), 3 * _dot(c, F)
        eq = w * rho * (1 + cu + 0.5 * cu * cu - 0.5 * uu)
        post.append((1 - omega) * f[s] + omega * eq + (1 - 0.5 * omega) * w * (cf - fu + cu * cf))
    if porosity is not None:
        opp = opposites(Q)
        post = [(1 - porosity) * post[s] + porosity * f[opp[s]] for s in range(Q)]
    return post


class _Walls:
    """Which neighbours bounce back, from a solid mask and open faces."""

    def __init__(self, Q, shape, solid, periodic):
        nz, ny, nx = shape
        self.Q, self.solid = Q, None if solid is None else torch.from_numpy(np.asarray(solid) != 0).to(DEVICE)
        self.blocked = [None] * Q
        if self.solid is None and all(periodic):
            return
        closed = self.solid if self.solid is not None else torch.zeros(shape, dtype=torch.bool, device=DEVICE)
        for s, c in enumerate(velocities(Q)):
            b = torch.roll(closed, (-c[2], -c[1], -c[0]), (0, 1, 2))
            for axis, (n, dim) in enumerate(((nx, 2), (ny, 1), (nz, 0))):
                if not periodic[axis] and c[axis]:
                    edge = torch.zeros(n, dtype=torch.bool, device=DEVICE)
                    edge[n - 1 if c[axis] > 0 else 0] = True
                    shape1 = [1, 1, 1]
                    shape1[dim] = n
                    b = b | edge.reshape(shape1)
            self.blocked[s] = b

    def stream(self, post, held):
        """Populations after streaming; solid cells keep ``held``."""
        opp = opposites(self.Q)
        out = []
        for s, c in enumerate(velocities(self.Q)):
            g = torch.roll(post[s], (c[2], c[1], c[0]), (0, 1, 2))
            if self.blocked[opp[s]] is not None:
                g = torch.where(self.blocked[opp[s]], post[opp[s]], g)
            if self.solid is not None:
                g = torch.where(self.solid, held[s], g)
            out.append(g)
        return torch.stack(out)


def _advance(f, Q, tau, F, porosity, walls, steps, pull=False):
    """``steps`` steps of populations by direction; pull: stored after the
    collision, before streaming."""
    held = f
    for _ in range(steps):
        if pull:
            post = torch.stack(collide(walls.stream(f, held), Q, tau, F, porosity))
            f = post if walls.solid is None else torch.where(walls.solid, held, post)
        else:
            f = walls.stream(collide(f, Q, tau, F, porosity), held)
    return f


def _shifted(f, Q, storage):
    if storage == "f64":
        return f
    w = torch.tensor(weights(Q), dtype=torch.float64, device=DEVICE).reshape(-1, 1, 1, 1)
    return (f - w) * (32768.0 if storage == "f16" else 1.0)


def exact(case, seed):
    kind, Q = case["kind"], case["lattice"]
    if kind in ("step", "readout"):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        solid, periodic = _solid(case, seed)
        walls = _Walls(Q, (nz, ny, nx), solid, periodic)
        fields = case.get("fields", "none")
        F = [_force(case), 0.0, 0.0]
        if fields in ("force", "both"):
            field = _force_field(nx, ny, nz, seed + 2)
            F = [F[d] + field[d] for d in range(3)]
        porosity = _field(nx, ny, nz, seed + 1) if fields in ("porosity", "both") else None
        f = equilibrium(Q, *_flow(nx, ny, nz, seed, 0.05 if case["geometry"] == "box" else 0.01))
        pattern = case.get("pattern", "aa")
        f = _advance(f, Q, case["tau"], F, porosity, walls, case["steps"], pattern == "ab_pull")
        if kind == "step":
            return raw_layout(_shifted(f, Q, case["storage"]), Q, pattern)
        rho, j = moments(f, Q)
        u = torch.stack([v / rho for v in j])
        keep = torch.ones_like(rho) if walls.solid is None else (~walls.solid).double()
        sums = np.array([float((v * keep).sum()) for v in (rho, *j)])
        if walls.solid is not None:
            rho = torch.where(walls.solid, math.nan, rho)
            u = torch.where(walls.solid, math.nan, u)
        return {"rho": rho, "u": u, "sums": sums}
    if kind == "sparse":
        solid, f = _cylinder_start(case, seed)
        walls = _Walls(Q, solid.shape, solid, (1, 1, 1))
        f = _advance(f, Q, 1.0, [1e-6, 0.0, 0.0], None, walls, case["steps"], case["pattern"] == "ab_pull")
        fluid = torch.from_numpy(np.flatnonzero(solid.ravel() == 0)).to(DEVICE)
        return raw_layout(f, Q, case["pattern"])[:, fluid].contiguous()
    return _exact_gradient(case, seed)


def _exact_gradient(case, seed):
    from torch.utils.checkpoint import checkpoint
    Q, tau = case["lattice"], case["tau"]
    solid, weight, window = _loss_weight(case)
    weight = torch.from_numpy(weight).to(DEVICE)
    walls = _Walls(Q, solid.shape, solid, (1, 0, 1))
    porosity, force = (p.double().requires_grad_() for p in _parameters(case, seed))
    _, u0 = _flow(case["nx"], case["ny"], case["nz"], seed, 0.01)
    f = equilibrium(Q, torch.ones_like(u0[0]), u0)
    held = f

    def term(f, force):
        rho, j = moments(f, Q)
        u = torch.stack([(j[d] + 0.5 * force[d]) / rho for d in range(3)])
        if case["loss"] == "velocity":
            return (weight * u).sum()
        return (weight * 0.5 * rho * (u * u).sum(0)).sum()

    def step(f, porosity, force):
        return walls.stream(collide(f, Q, tau, force, porosity), held)

    loss = torch.zeros((), dtype=torch.float64, device=DEVICE)
    for t in range(case["steps"] + 1):
        if window[0] <= t <= window[1]:
            loss = loss + term(f, force)
        if t < case["steps"]:
            f = checkpoint(step, f, porosity, force, use_reentrant=False)
    grads = torch.autograd.grad(loss, (porosity, force))
    return {"loss": loss.detach(), "porosity": grads[0], "force": grads[1]}
