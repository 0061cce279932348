"""The pipelined steps' forms at the sizes and states where their rules change.

F64X against the exact FP64 arithmetic on the GPU: a step agrees to 2e-13 per
population (the host sweeps' bound), so `steps` steps from the same state to
4e-13 * steps with the rounding of the exact one.  Exact arithmetic against the
oracle: equal bits (tolerance 0)."""
import numpy as np
import pytest

from oracle import core
from lbmminiapp_gb300 import Simulation, workloads

pytestmark = pytest.mark.gpu

PATTERNS = ["aa", "ab_push", "ab_pull"]


def run(Q, dims, pattern, arithmetic, steps, solid=None, force=(0.0, 0.0, 0.0), f0=None):
    nx, ny, nz = dims
    per = (1, 1, 1) if solid is None else (1, 0, 1)
    with Simulation(nx, ny, nz, lattice=Q, pattern=pattern, omega=1.0 / 0.7, force=force, periodic=per,
                    arithmetic=arithmetic) as sim:
        if solid is not None:
            sim.set_solid(solid)
        if f0 is None:
            sim.init_equilibrium(None, workloads.taylor_green(nx, ny, nz, 0.04, noise=1e-3, seed=nx + nz))
        else:
            sim.set_populations(f0)
        sim.step(steps)
        return sim.get_populations("raw")


def close(a, b, steps):
    m = np.isfinite(b)
    return np.array_equal(m, np.isfinite(a)) and np.abs(a - b)[m].max() <= 4e-13 * steps * np.abs(b[m]).max()


# tiles run across row ends; the last one is partial (or the only one)
@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("dims", [(1, 1, 1), (31, 1, 1), (1, 33, 2), (33, 5, 3), (161, 7, 5), (64, 4, 4)])
@pytest.mark.parametrize("walls", [False, True])
def test_tiles_across_rows(gpu, Q, pattern, dims, walls):
    if walls and dims[1] < 4:
        pytest.skip("needs fluid between the walls")
    solid = workloads.channel_mask(*dims) if walls else None
    a = run(Q, dims, pattern, "f64x", 3, solid)
    assert close(a, run(Q, dims, pattern, "f64", 3, solid), 3)


# D3Q27: below 16 tiles per warp (29,184 on 152 SMs) the rest population sits in a register
@pytest.mark.parametrize("pattern", ["aa", "ab_push"])
@pytest.mark.parametrize("nz", [101, 102])
def test_both_forms_of_the_d3q27_blocks(gpu, pattern, nz):
    a = run(27, (96, 96, nz), pattern, "f64x", 2)
    assert close(a, run(27, (96, 96, nz), pattern, "f64", 2), 2)


# no force, velocity shift, folded, added
@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("gx", [0.0, 1e-6, 1e-3, 1e-2])
def test_forcing_forms(gpu, Q, pattern, gx):
    dims = (40, 10, 9)
    solid = workloads.channel_mask(*dims)
    a = run(Q, dims, pattern, "f64x", 2, solid, (gx, 0.3 * gx, -0.2 * gx))
    assert close(a, run(Q, dims, pattern, "f64", 2, solid, (gx, 0.3 * gx, -0.2 * gx)), 2)


# cells inside and outside the ranges of the exact arithmetic's integer additions, side by side
@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("pattern,pid", [("aa", core.AA), ("ab_push", core.AB_PUSH), ("ab_pull", core.AB_PULL)])
@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), (1e-5, 0.0, 2e-6)])
def test_exact_arithmetic_outside_the_integer_ranges(gpu, Q, pattern, pid, force):
    nx, ny, nz = 33, 6, 5
    rng = np.random.default_rng(Q)
    u = workloads.taylor_green(nx, ny, nz, 0.05, noise=1e-3, seed=Q)
    f0 = core.equilibrium(Q, np.ones((nz, ny, nx)), u)
    f0[:, 0, 0, :4] = core.equilibrium(Q, np.ones((1, 1, 4)), np.full((3, 1, 1, 4), 0.12))[:, 0, 0]   # fast
    f0[:, 1, 2, 3] = core.equilibrium(Q, np.ones((1, 1, 1)), np.zeros((3, 1, 1, 1)))[:, 0, 0, 0]        # at rest
    f0[5, 2, 3, 7] = 1e-9          # far below 2^-10
    f0[3, 2, 3, 20] = 0.0
    f0[2, 3, 1, 9] = -1e-3
    f0[:, 4, 4, 11] *= 2.5         # rho above 2
    f0[:, 3, 3, :] *= 1.0 + 0.2 * rng.standard_normal((Q, nx))
    ref, _ = core.run(Q, pid, f0, 2, 1.0 / 0.7, force, (1, 1, 1), np.zeros((nz, ny, nx), np.uint8))
    out = run(Q, (nx, ny, nz), pattern, "f64", 2, None, force, f0)
    assert np.array_equal(out, ref)
