"""The cell moments of the readouts and the loss, compiled for the host, against
sums in exact rational arithmetic.

Tolerance: a sum of Q doubles added one after another is within (Q - 1) half ulps
of the largest partial sum of the true value: (Q - 1) 2^-53 sum |f|.  Cells the
integer sums take are held to the same."""
import ctypes
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

from oracle import core

ROOT = Path(__file__).resolve().parents[1]
P = ctypes.c_void_p


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    out = tmp_path_factory.mktemp("moments") / "libmoments.so"
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", "-I", str(ROOT / "lbmminiapp_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "moments_check.cu"), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


def moments_f64(lib, Q, f):
    f = np.ascontiguousarray(f)
    out, regular = np.empty((len(f), 4)), np.empty(len(f), np.uint8)
    lib.moments_f64(Q, P(f.ctypes.data), len(f), P(out.ctypes.data), P(regular.ctypes.data))
    return out, regular.astype(bool)


def exact(Q, f):
    """Sums as fractions, [n][4]."""
    c, _, _ = core.stencil(Q)
    rows = []
    for cell in f:
        v = [Fraction(x) for x in cell.tolist()]
        rows.append([sum(v)] + [sum(int(c[s][d]) * v[s] for s in range(Q)) for d in range(3)])
    return rows


def largest_error(Q, f, out):
    """Largest error over the tolerance of its cell."""
    worst = 0.0
    for cell, got, want in zip(f, out, exact(Q, f)):
        tol = (Q - 1) * 2.0 ** -53 * float(np.abs(cell).sum())
        worst = max(worst, *(abs(float(Fraction(g) - w)) / tol for g, w in zip(got.tolist(), want)))
    return worst


def equilibrium(Q, rho, u):
    n = len(rho)
    return core.equilibrium(Q, np.asarray(rho), np.broadcast_to(np.asarray(u)[:, None], (3, n)).copy()).T.copy()


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("u", [(0.0, 0.0, 0.0), (0.05, -0.02, 0.01), (0.45, 0.0, 0.0)])
def test_dense_cells(lib, Q, u):
    """Densities around and above 2, 4 and 8 with every population below 1."""
    rho = np.concatenate([np.linspace(0.3, 9.0, 120), [2.0, np.nextafter(2.0, 0), 4.0, 4.2, 8.0]])
    f = equilibrium(Q, rho, u)
    f = f[(f.max(axis=1) < 1) & (f.min(axis=1) > 0)]
    assert largest_error(Q, f, moments_f64(lib, Q, f)[0]) <= 1


@pytest.mark.parametrize("Q", [19, 27])
def test_any_populations_below_one(lib, Q):
    rng = np.random.default_rng(Q)
    f = rng.uniform(1e-3, 1.0, (400, Q))
    f[:200] *= np.exp2(-rng.uniform(0, 6, (200, 1)))
    f[-1] = 0.23
    f[-2] = np.nextafter(1.0, 0)
    out, regular = moments_f64(lib, Q, f)
    assert regular.any() and not regular.all()
    assert largest_error(Q, f, out) <= 1


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("scale", [1e-1, 1e-3, 1e-5, 1e-7])
def test_thin_cells(lib, Q, scale):
    """Populations down to 2^-31 and below, all of them small or one alone."""
    rng = np.random.default_rng(Q)
    f = equilibrium(Q, np.ones(200), (0.05, -0.02, 0.01)) * (1 + 1e-3 * rng.standard_normal((200, Q)))
    f[:100] *= scale
    f[np.arange(100, 200), rng.integers(0, Q, 100)] *= scale
    assert largest_error(Q, f, moments_f64(lib, Q, f)[0]) <= 1
