"""lbm_loss on states far from density 1, against the same sums in FP64 with numpy.

Tolerance: each cell's term carries about (Q + 8) roundings and the sum over n
cells at most n more, relative to the terms' magnitudes; with n <= 4096 that is
below 5e-13 of sum |term|: 1e-12."""
import ctypes

import numpy as np
import pytest

from oracle import core
from lbmminiapp_gb300 import Simulation
from lbmminiapp_gb300 import _native as N

pytestmark = pytest.mark.gpu


def loss_of(f, Q, kind, weight, storage="f64"):
    import torch
    nz, ny, nx = f.shape[1:]
    with Simulation(nx, ny, nz, lattice=Q, pattern="ab_push", storage=storage) as sim:
        sim.set_populations(f)
        plane = int(sim.info.plane_stride)
        w = torch.zeros((len(weight), plane), dtype=torch.float64, device="cuda")
        w[:, :sim.ncell] = torch.as_tensor(weight.reshape(len(weight), -1), device="cuda")
        torch.cuda.synchronize()
        out = ctypes.c_double()
        N.check(sim.lib.lbm_loss(sim.h, None, kind, ctypes.c_void_p(w.data_ptr()), 1.0, ctypes.byref(out)), sim.h)
        stored = sim.get_populations()
    return out.value, stored


def terms(f, Q, kind, weight):
    c, _, _ = core.stencil(Q)
    rho = f.sum(axis=0)
    u = np.stack([sum(int(c[s][d]) * f[s] for s in range(Q)) / rho for d in range(3)])
    if kind == N.LOSS_VELOCITY:
        return weight * u
    return weight[0] * 0.5 * rho * (u * u).sum(axis=0)


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("kind", [N.LOSS_VELOCITY, N.LOSS_ENERGY])
@pytest.mark.parametrize("state", ["2.5", "4.2", "spread", "mixed"])
def test_dense_fp64_states(gpu, Q, kind, state):
    shape = (8, 8, 33)
    rng = np.random.default_rng(Q)
    if state == "spread":          # density around 9, every population below 1
        f = rng.uniform(0.05, 0.95, (Q,) + shape)
    else:
        rho = np.full(shape, float(state)) if state != "mixed" else rng.uniform(0.5, 6.0, shape)
        u = np.zeros((3,) + shape)
        u[0], u[1] = (0.45, 0.01) if state == "4.2" else (0.05, -0.02)
        f = core.equilibrium(Q, rho, u)
    weight = rng.standard_normal(((3 if kind == N.LOSS_VELOCITY else 1),) + shape)
    got, _ = loss_of(f, Q, kind, weight)
    t = terms(f, Q, kind, weight)
    assert abs(got - t.sum()) <= 1e-12 * np.abs(t).sum()
