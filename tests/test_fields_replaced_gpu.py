"""Per-cell fields set from device memory and then again from the host: steps, loss
and both gradients are those of a handle that only ever had the second ones, bit
for bit (the same kernels on the same values)."""
import ctypes

import numpy as np
import pytest

from lbmminiapp_gb300 import workloads

pytestmark = pytest.mark.gpu

NX, NY, NZ = 24, 10, 9


def fields(seed):
    rng = np.random.default_rng(seed)
    return 1e-5 * rng.standard_normal((3, NZ, NY, NX)), rng.uniform(0.0, 0.3, (NZ, NY, NX))


def rollout(storage, adjoint):
    from lbmminiapp_gb300.adjoint import new_rollout
    solid = workloads.channel_mask(NX, NY, NZ)
    weight = (~solid.astype(bool)).astype(float)
    u0 = workloads.taylor_green(NX, NY, NZ, 0.03, noise=1e-3, seed=2)
    return new_rollout(NX, NY, NZ, 19, 0.7, solid, (1, 0, 1), 6, 3, "energy", weight, (5, 6), storage=storage, u0=u0,
                       adjoint=adjoint)


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("adjoint", ["f64", "f32"])
def test_host_fields_replace_device_fields(gpu, storage, adjoint):
    import torch
    f1, p1 = fields(1)
    f2, p2 = fields(2)
    results = []
    for first in (True, False):
        r = rollout(storage, adjoint)
        if first:
            r.set_fields(torch.as_tensor(f1, device="cuda"), torch.as_tensor(p1, device="cuda"))
            r.sim.set_porosity(p2)
            r.sim.set_force_field(f2)
        else:
            r.set_fields(torch.as_tensor(f2, device="cuda"), torch.as_tensor(p2, device="cuda"))
        loss = r.run_forward(store=True)
        gF, gS = r.run_backward()
        results.append((loss, r.from_plane(gF).cpu().numpy(), r.from_plane(gS).cpu().numpy()))
        r.release()
    (la, fa, sa), (lb, fb, sb) = results
    assert la == lb
    assert np.array_equal(fa, fb) and np.array_equal(sa, sb)
