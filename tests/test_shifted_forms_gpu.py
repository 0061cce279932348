"""The kernels that run the shifted-storage collision (one cell per thread, two
cells per thread, pipelined with links, compact) give the same bits for a force
along no axis: tolerance 0."""
import numpy as np
import pytest

from lbmminiapp_gb300 import Simulation, workloads

pytestmark = pytest.mark.gpu

FORCE = (1e-5, 3e-6, -2e-6)
DIMS = (34, 10, 9)


def start(sim, seed, solid=None):
    u = workloads.taylor_green(*DIMS, 0.04, noise=2e-3, seed=seed)
    if solid is not None:
        sim.set_solid(solid)
        u[:, solid.astype(bool)] = 0
    sim.init_equilibrium(1.0 + 0.01 * np.random.default_rng(seed).random(DIMS[::-1]), u)


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), FORCE])
def test_compact_equals_dense_with_an_oblique_force(gpu, Q, storage, force):
    solid = workloads.channel_mask(*DIMS)
    solid |= (np.random.default_rng(Q).random(solid.shape) < 0.1).astype(np.uint8)
    raw = []
    for compact in (False, True):
        with Simulation(*DIMS, lattice=Q, omega=1.0 / 0.7, force=force, periodic=(1, 0, 1), storage=storage,
                        compact=compact) as sim:
            start(sim, Q, solid)
            sim.step(6)
            raw.append(sim.get_populations("raw"))
    assert np.array_equal(raw[0], raw[1], equal_nan=True)


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), FORCE])
@pytest.mark.parametrize("pattern", ["aa", "ab_push", "ab_pull"])
def test_full_steps_equal_range_calls(gpu, Q, storage, force, pattern):
    import torch
    raw = []
    for ranges in (False, True):
        with Simulation(*DIMS, lattice=Q, pattern=pattern, omega=1.0 / 0.7, force=force, storage=storage) as sim:
            start(sim, Q)
            n, a = sim.ncell, sim.population_buffer()
            size = int(sim.info.buffer_bytes)
            parts = [(0, 1000), (1000, n - 1000)] if ranges else [(0, n)]
            if pattern == "aa":
                for t in range(4):
                    call = sim.timestep_even_force if t % 2 == 0 else sim.timestep_odd_force
                    for first, count in parts:
                        call(a, first, count)
            else:
                other = torch.empty(size, dtype=torch.uint8, device="cuda")
                torch.cuda.synchronize()
                b = other.data_ptr()
                for t in range(4):
                    for first, count in parts:
                        sim.timestep_force((a, b)[t % 2], (b, a)[t % 2], first, count)
            sim.synchronize()
            raw.append(sim.get_populations("raw"))
    assert np.array_equal(raw[0], raw[1])
