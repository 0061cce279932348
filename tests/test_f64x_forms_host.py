"""F64X with a small force, on the host: the velocity-shift form is no further from
the collision in extended precision than the form that it replaces, whose forcing
terms are float pairs.

Tolerance: the two errors are rms values over 76,000 populations or more of
independent roundings, so each is known to better than 2 %: the shift form's is
below 1.02 times the other's."""
import numpy as np
import pytest

from oracle import core
from test_f64x_host import f64x, random_cells, run as run_form  # noqa: F401 (fixture)
from test_f64x_shift_host import lib, run as run_library        # noqa: F401 (fixture)

LD = np.longdouble


def collide_extended(Q, f, omega, F):
    c = core.stencil(Q)[0].astype(LD)
    table = {19: [LD(1) / 3, LD(1) / 18, LD(1) / 36], 27: [LD(8) / 27, LD(2) / 27, LD(1) / 54, LD(1) / 216]}[Q]
    w = np.array([table[int(k)] for k in (c * c).sum(axis=1)], dtype=LD)
    f, F, om = f.astype(LD), np.asarray(F).astype(LD), LD(omega)
    rho = f.sum(axis=1)
    v = np.stack([(f * c[:, d]).sum(axis=1) + F[d] / 2 for d in range(3)], axis=1) / rho[:, None]
    cu = 3 * sum(v[:, d:d + 1] * c[None, :, d] for d in range(3))
    cf = 3 * (c * F).sum(axis=1)
    vv, fv = 3 * (v * v).sum(axis=1)[:, None], 3 * (v * F).sum(axis=1)[:, None]
    eq = w * rho[:, None] * (1 + cu + cu * cu / 2 - vv / 2)
    return (1 - om) * f + om * eq + (1 - om / 2) * w * (cf - fv + cu * cf)


@pytest.mark.skipif(np.finfo(LD).nmant <= 60, reason="needs an extended format")
@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("omega", [1.0 / 0.55, 1.0, 0.5])
@pytest.mark.parametrize("share", [0.01, 0.999])
@pytest.mark.parametrize("direction", [(1.0, 0.0, 0.0), (1.0, 1.0, 1.0)])
def test_velocity_shift_is_as_accurate(f64x, lib, Q, omega, share, direction):  # noqa: F811
    limit = 1e-5 * omega / (1.0 - 0.5 * omega)
    F = share * limit * np.array(direction) / np.sum(direction)
    f = random_cells(Q, 4000, 0.05, 0.01, seed=Q)
    form, shift, fast = run_library(lib, Q, f, omega, F)
    assert form == 3 and fast.all()
    folded, fast2 = run_form(f64x, Q, f, omega, F, force_mode=2)
    assert fast2.all()
    want = collide_extended(Q, f, omega, F)
    rms = [float(np.sqrt((((out.astype(LD) - want) / want) ** 2).mean())) for out in (shift, folded)]
    assert rms[0] <= 1.02 * rms[1]
