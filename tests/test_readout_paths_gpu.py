"""lbm_get_macros into pageable memory (staged in chunks), into page-locked
memory (written by the kernel) and into one array of each: the same bits, and the
reference's for FP64 storage.
A diverged cell of shifted storage reads back as not finite."""
import numpy as np
import pytest

from oracle import core
from lbmminiapp_gb300 import Simulation, workloads

pytestmark = pytest.mark.gpu


def pinned(shape):
    import torch
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("steps", [0, 3, 4])
@pytest.mark.parametrize("dims", [(70, 40, 31), (7, 5, 3)])
def test_page_locked_and_pageable_readouts_agree(gpu, storage, steps, dims):
    nx, ny, nz = dims
    with Simulation(nx, ny, nz, storage=storage, omega=1.4, periodic=(1, 0, 1)) as sim:
        solid = workloads.channel_mask(nx, ny, nz)
        sim.set_solid(solid)
        sim.init_equilibrium(None, workloads.taylor_green(nx, ny, nz, 0.05, noise=1e-3, seed=steps))
        sim.step(steps)
        rho, u = sim.macros()
        rp, up = pinned((nz, ny, nx)), pinned((3, nz, ny, nx))
        sim.macros((rp, up))
        # rho page-locked, u not
        r2, u2 = pinned((nz, ny, nx)), np.empty((3, nz, ny, nx))
        sim.macros((r2, u2))
        raw = sim.get_populations("raw")
    for a in (rp, r2):
        assert np.array_equal(a, rho, equal_nan=True)
    for a in (up, u2):
        assert np.array_equal(a, u, equal_nan=True)
    assert np.array_equal(np.isnan(rho), solid.astype(bool))
    if storage == "f64":
        rr, ur = core.readout_macros(19, core.AA, steps, raw, solid, (1, 0, 1))
        m = solid == 0
        assert np.array_equal(rho[m], rr[m])
        assert np.abs(u - ur)[:, m].max() <= 4e-16


def test_diverged_cell_of_shifted_storage(gpu):
    f = core.equilibrium(19, np.ones((4, 4, 8)), np.zeros((3, 4, 4, 8)))
    f[3, 1, 2, 5] = 1e30           # infinite in FP16
    with Simulation(8, 4, 4, storage="f16", pattern="ab_push") as sim:
        sim.set_populations(f)
        rho, _ = sim.macros()
    assert np.isinf(rho[1, 2, 5]) and np.isfinite(rho).sum() == rho.size - 1
