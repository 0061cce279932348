"""The pipelined F64X steps with the tile feed on (from 16 tiles per warp), a last
tile that is not full and, for the D3Q27 AB steps, a last group of tiles that is not
full, against the exact FP64 arithmetic.

Tolerance: a step agrees to 2e-13 of each population (the host sweeps' bound), so
two steps from the same state to 4e-13 per step, population by population."""
import numpy as np
import pytest

from lbmminiapp_gb300 import Simulation, workloads

pytestmark = pytest.mark.gpu

STEPS = 2


def run(Q, dims, pattern, arithmetic, walls, force):
    nx, ny, nz = dims
    with Simulation(nx, ny, nz, lattice=Q, pattern=pattern, omega=1.0 / 0.7, force=force,
                    periodic=(1, 0 if walls else 1, 1), arithmetic=arithmetic) as sim:
        if walls:
            sim.set_solid(workloads.channel_mask(nx, ny, nz))
        sim.init_equilibrium(None, workloads.taylor_green(nx, ny, nz, 0.04, noise=1e-3, seed=nx))
        sim.step(STEPS)
        return sim.get_populations("raw")


# 161x75x93: 35,093 tiles, the last of 31 cells; 167x89x91: 42,267, the last of 21 (D3Q19: only this one has the feed on)
@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("pattern", ["aa", "ab_push", "ab_pull"])
@pytest.mark.parametrize("dims", [(161, 75, 93), (167, 89, 91)])
@pytest.mark.parametrize("walls", [False, True])
def test_feed_with_partial_last_tiles(gpu, Q, pattern, dims, walls):
    force = (1e-6, 3e-7, 0.0) if walls else (0.0, 0.0, 0.0)
    a, b = (run(Q, dims, pattern, arithmetic, walls, force) for arithmetic in ("f64x", "f64"))
    fluid = np.isfinite(b)
    assert np.array_equal(fluid, np.isfinite(a))
    assert (np.abs(a - b)[fluid] <= 4e-13 * STEPS * np.abs(b[fluid])).all()


# small grids, population by population (no feed, blocks spread over the SMs)
@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("pattern", ["aa", "ab_push", "ab_pull"])
@pytest.mark.parametrize("dims", [(33, 9, 7), (40, 40, 31), (96, 96, 101)])
def test_small_grids_population_by_population(gpu, Q, pattern, dims):
    a, b = (run(Q, dims, pattern, arithmetic, True, (1e-6, 3e-7, 0.0)) for arithmetic in ("f64x", "f64"))
    fluid = np.isfinite(b)
    assert (np.abs(a - b)[fluid] <= 4e-13 * STEPS * np.abs(b[fluid])).all()
