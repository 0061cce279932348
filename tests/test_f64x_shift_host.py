"""The F64X forcing form that shifts the velocity, compiled for the host: which
forces take it, and its precision against the exact IEEE double collision.

Tolerance: the double-float terms agree with the exact collision to 2e-13 per
population in every form; the velocity shift adds one single-precision term,
omega w rho k^2 E with k |F| <= 1e-5 / rho.  Its rounding is below
2^-24 k^2 4.5 F^2 <= 4.3e-16 of w (rho >= 1/4), so the same bound holds."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from test_f64x_host import collide_exact, random_cells

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    out = tmp_path_factory.mktemp("f64x") / "libf64x_shift.so"
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC",
                    "-I", str(ROOT / "lbmminiapp_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "f64x_shift_check.cu"), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


def run(lib, Q, f, omega, F, compat=0):
    f = np.ascontiguousarray(f)
    out = np.empty_like(f)
    fast = np.empty(f.shape[0], np.int32)
    Fa = np.asarray(F, dtype=np.float64)
    P = ctypes.c_void_p
    form = lib.f64x_library_collide(Q, P(f.ctypes.data), P(out.ctypes.data), f.shape[0], ctypes.c_double(omega),
                                    P(Fa.ctypes.data), compat, P(fast.ctypes.data))
    return form, out, fast.astype(bool)


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("omega", [1.0 / 0.55, 1.0, 0.3])
@pytest.mark.parametrize("direction", [(1.0, 0.0, 0.0), (0.0, -1.0, 0.0), (0.5, -0.3, 0.2)])
@pytest.mark.parametrize("share", [1e-8, 0.1, 0.999])
def test_velocity_shift_matches_exact_collision(lib, Q, omega, direction, share):
    """Forces from far below the form's limit to its edge."""
    limit = 1e-5 * omega / (1.0 - 0.5 * omega)
    F = share * limit * np.array(direction) / np.abs(direction).sum()
    f = random_cells(Q, 3000, 0.08, 0.02, seed=Q)
    form, out, fast = run(lib, Q, f, omega, F)
    assert form == 3
    assert fast.mean() > 0.99
    ref = collide_exact(Q, f, omega, F)
    err = np.abs(out[fast] - ref[fast]) / np.abs(ref[fast])
    assert err.max() < 2e-13, err.max()


def test_which_forces_shift_the_velocity(lib):
    f = random_cells(19, 4, 0.05, 0.01, seed=1)
    omega = 1.25
    limit = 1e-5 * omega / (1.0 - 0.5 * omega)
    assert run(lib, 19, f, omega, (0.0, 0.0, 0.0))[0] == 0
    assert run(lib, 19, f, omega, (0.999 * limit, 0.0, 0.0))[0] == 3
    assert run(lib, 19, f, omega, (0.4 * limit, -0.4 * limit, 0.4 * limit))[0] == 2
    assert run(lib, 19, f, omega, (0.01, 0.0, 0.0))[0] == 1
    # the Unroll kernels' rest weight breaks the identity
    assert run(lib, 19, f, omega, (0.1 * limit, 0.0, 0.0), compat=1)[0] == 2
