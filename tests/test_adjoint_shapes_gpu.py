"""The adjoint on grids whose rows do not fill their warps: gradients against
torch.autograd through plain FP64 operations, and the cost per cell of an adjoint
step whatever nx is.

Tolerance, relative to the largest gradient: a step is about 300 operations, each
off by half an ulp at most, and 6 steps follow one another: 1800 x 2^-53 = 2e-13
and 1800 x 2^-24 = 1.1e-4, a factor 5 above for the condition of the sums."""
import ctypes

import numpy as np
import pytest

from lbmminiapp_gb300 import _native as N

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "f32": 5e-4}


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("real", ["f64", "f32"])
@pytest.mark.parametrize("dims", [(1, 9, 7), (2, 8, 5), (8, 6, 5), (31, 5, 4), (33, 5, 4), (129, 5, 3)])
@pytest.mark.parametrize("loss", ["velocity", "energy"])
def test_gradients_on_narrow_grids(gpu, Q, real, dims, loss):
    import torch
    from perf import cases
    case = cases._adjoint(None, *dims, Q, real, real, loss, 6, 3)
    got, want = cases.run(cases.prepare(case, 5)), cases.exact(case, 5)
    torch.cuda.synchronize()
    for k in ("loss", "porosity", "force"):
        a, b = got[k].double(), want[k]
        assert float((a - b).abs().max()) <= TOL[real] * float(b.abs().max()), k


def step_time(nx, ny, nz, adjoint):
    import torch
    from lbmminiapp_gb300.adjoint import new_rollout
    r = new_rollout(nx, ny, nz, 19, 0.7, np.zeros((nz, ny, nx), np.uint8), (1, 1, 1), 2, 2, "energy",
                    np.full((nz, ny, nx), 1.0 / (nx * ny * nz)), (2, 2), storage=adjoint, adjoint=adjoint)
    real = torch.float32 if adjoint == "f32" else torch.float64
    a, b = (torch.zeros((r.Q, r.plane), dtype=real, device="cuda") for _ in range(2))
    gF = torch.zeros((3, r.plane), dtype=torch.float64, device="cuda")
    gS = torch.zeros((r.plane,), dtype=torch.float64, device="cuda")
    fn = r.lib.lbm_adjoint_step_f32 if adjoint == "f32" else r.lib.lbm_adjoint_step
    p = [ctypes.c_void_p(t.data_ptr()) for t in (r.init_state, a, b, r.weight, gF, gS)]
    torch.cuda.synchronize()
    times = []
    for _ in range(8):
        first, last = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        first.record()
        for _ in range(10):
            N.check(fn(r.h, p[0], p[1], p[2], 1, N.LOSS_ENERGY, p[3], 1.0, p[4], p[5]), r.h)
        last.record()
        last.synchronize()
        times.append(first.elapsed_time(last))
    return min(times)


@pytest.mark.parametrize("adjoint", ["f64", "f32"])
@pytest.mark.parametrize("nx", [1, 8, 129])
def test_cost_per_cell_does_not_depend_on_the_row_length(gpu, adjoint, nx):
    """The cells of a 128x64x64 grid (a little fewer for 129) in rows of nx: at most
    twice its time; with a row per block it was 3 to 20 times."""
    ny = {1: 1024, 8: 256, 129: 64}[nx]
    nz = 128 * 64 * 64 // (nx * ny)
    assert step_time(nx, ny, nz, adjoint) <= 2 * step_time(128, 64, 64, adjoint)
