"""What a uniform force adds to a step of a periodic box in the D3Q19 16-bit
storages: a quarter at most (measured: 18 %; 32 % where the forcing spills registers)."""
import pytest

from lbmminiapp_gb300 import Simulation

pytestmark = pytest.mark.gpu


def step_time(storage, pattern, force):
    import torch
    with Simulation(256, 256, 128, pattern=pattern, omega=1.25, force=force, storage=storage) as sim:
        sim.step(4)
        times = []
        for _ in range(6):
            first, last = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            sim.synchronize()
            first.record()
            sim.step(20)
            last.record()
            last.synchronize()
            times.append(first.elapsed_time(last))
        return min(times)


@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("pattern", ["ab_push", "ab_pull", "aa"])
def test_a_force_costs_little(gpu, storage, pattern):
    assert step_time(storage, pattern, (1e-6, 0.0, 0.0)) <= 1.25 * step_time(storage, pattern, (0.0, 0.0, 0.0))
