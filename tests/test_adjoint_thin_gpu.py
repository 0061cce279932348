"""The FP64 adjoint of states of small density, against torch.autograd through
plain FP64 operations.

Tolerance: 3 steps of about 300 operations at half an ulp each are 1e-13 of the
largest gradient; 1e-12 leaves a factor 10 for the condition of the sums."""
import numpy as np
import pytest

from oracle import core
from lbmminiapp_gb300 import Simulation, workloads

pytestmark = pytest.mark.gpu

NX, NY, NZ, TAU, STEPS = 20, 7, 6, 0.7, 3


def autograd(Q, f0, porosity, force, weight):
    import torch
    from perf import cases
    dev = torch.device("cuda")
    f = torch.as_tensor(f0, device=dev)
    p, F = (torch.as_tensor(v, device=dev).requires_grad_() for v in (porosity, force))
    walls = cases._Walls(Q, (NZ, NY, NX), None, (1, 1, 1))
    for _ in range(STEPS):
        f = walls.stream(cases.collide(f, Q, TAU, F, p), f)
    rho, j = cases.moments(f, Q)
    u = torch.stack([(j[d] + 0.5 * F[d]) / rho for d in range(3)])
    loss = (torch.as_tensor(weight, device=dev) * 0.5 * rho * (u * u).sum(0)).sum()
    return [g.cpu().numpy() for g in torch.autograd.grad(loss, (p, F))]


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("density", [1.0, 1e-2, 1e-4, 1e-6])
def test_thin_states(gpu, Q, density):
    import torch
    from lbmminiapp_gb300.adjoint import Rollout
    rng = np.random.default_rng(Q)
    u = workloads.taylor_green(NX, NY, NZ, 0.03, noise=1e-3, seed=Q)
    f0 = core.equilibrium(Q, density * (1 + 0.01 * rng.random((NZ, NY, NX))), u)
    porosity = rng.uniform(0.0, 0.3, (NZ, NY, NX))
    force = density * 1e-5 * rng.standard_normal((3, NZ, NY, NX))
    weight = rng.random((NZ, NY, NX))
    sim = Simulation(NX, NY, NZ, lattice=Q, pattern="ab_push", omega=1.0 / TAU, arithmetic="f64")
    sim.set_populations(f0)
    r = Rollout(sim, STEPS, STEPS, "energy", weight, (STEPS, STEPS))
    r.set_fields(torch.as_tensor(force, device="cuda"), torch.as_tensor(porosity, device="cuda"))
    r.run_forward(store=True)
    gF, gS = r.run_backward()
    got = [r.from_plane(gS).cpu().numpy(), r.from_plane(gF).cpu().numpy()]
    for a, b in zip(got, autograd(Q, f0, porosity, force, weight)):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
