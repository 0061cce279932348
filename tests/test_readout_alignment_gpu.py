"""lbm_get_macros into page-locked arrays that do not start on an 8-byte boundary,
or that reach past their allocation: the same bits as into aligned ones
(tolerance 0)."""
import numpy as np
import pytest

from lbmminiapp_gb300 import Simulation, workloads

pytestmark = pytest.mark.gpu

DIMS = (70, 9, 7)


def page_locked(shape, offset):
    """A float64 array `offset` bytes into a page-locked allocation that ends with it."""
    import torch
    n = int(np.prod(shape))
    raw = torch.zeros(8 * n + offset, dtype=torch.uint8, pin_memory=True)
    a = np.frombuffer(raw.numpy(), dtype=np.float64, count=n, offset=offset).reshape(shape)
    return a, raw


@pytest.mark.parametrize("storage", ["f64", "f16"])
@pytest.mark.parametrize("offsets", [(0, 0), (4, 0), (0, 4), (1, 7), (8, 16)])
def test_page_locked_arrays_at_any_offset(gpu, storage, offsets):
    nx, ny, nz = DIMS
    with Simulation(nx, ny, nz, storage=storage, omega=1.4) as sim:
        sim.init_equilibrium(None, workloads.taylor_green(nx, ny, nz, 0.05, noise=1e-3, seed=1))
        sim.step(3)
        rho, u = sim.macros()
        (r, keep_r), (v, keep_v) = page_locked(rho.shape, offsets[0]), page_locked(u.shape, offsets[1])
        assert r.flags.aligned == (offsets[0] % 8 == 0) and v.flags.aligned == (offsets[1] % 8 == 0)
        sim.macros((r, v))
    assert np.array_equal(r, rho) and np.array_equal(v, u)
