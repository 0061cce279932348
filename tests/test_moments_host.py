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


def moments_shifted(lib, Q, g, f16=False):
    g = np.ascontiguousarray(g)
    out, regular = np.empty((len(g), 4)), np.empty(len(g), np.uint8)
    lib.moments_shifted(Q, int(f16), P(g.ctypes.data), len(g), P(out.ctypes.data), P(regular.ctypes.data))
    return out, regular.astype(bool)


def errors_shifted(Q, g, out):
    """|out - exact| of rho = 1 + sum g and j = sum c g, [n][4]."""
    rows = exact(Q, g.astype(np.float64))
    return np.array([[abs(float(Fraction(a) - (b + (k == 0)))) for k, (a, b) in enumerate(zip(got.tolist(), want))]
                     for got, want in zip(out, rows)])


def sums_fp64(Q, g):
    """rho and j of f = g + w, added up in FP64 one after another."""
    c, _, w = core.stencil(Q)
    out = np.zeros((len(g), 4))
    for s in range(Q):
        f = g[:, s].astype(np.float64) + w[s]
        out[:, 0] += f
        for d in range(3):
            out[:, 1 + d] += c[s][d] * f
    return out


def as_stored(g, f16):
    """Deviations as the storage holds them (FP16: scaled by 2^15)."""
    return (np.float16(g * 32768) / np.float32(32768)).astype(np.float32) if f16 else g


def assert_as_accurate_as_fp64(lib, Q, g, f16=False):
    """The largest and the mean error over the cells, of rho and of j, are no larger
    than those of sums in FP64."""
    out, regular = moments_shifted(lib, Q, g, f16)
    e, ref = errors_shifted(Q, g, out), errors_shifted(Q, g, sums_fp64(Q, g))
    if f16:
        assert (regular == (g.sum(axis=1) > -0.5)).all()   # any state above density 1/2
    for k in (slice(0, 1), slice(1, 4)):
        assert e[:, k].max() <= ref[:, k].max()
        assert e[:, k].mean() <= ref[:, k].mean()
    return regular


# spread of the deviations, density, velocity
@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("noise,rho,U", [(1e-3, 1.0, 0.05), (1e-6, 1.0, 1e-4), (1e-2, 1.1, 0.15), (1e-2, 0.8, 0.1),
                                         (3e-2, 1.25, 0.2), (1e-2, 2.5, 0.1), (1e-2, 5.0, 0.1)])
@pytest.mark.parametrize("f16", [False, True])
def test_shifted_sums_of_flow_cells(lib, Q, noise, rho, U, f16):
    rng = np.random.default_rng(Q)
    n = 300
    u = rng.uniform(-U, U, (3, n))
    f = core.equilibrium(Q, rho * (1 + 0.01 * rng.standard_normal(n)), u).T
    g = as_stored((f - core.stencil(Q)[2] + f * noise * rng.standard_normal(f.shape)).astype(np.float32), f16)
    regular = assert_as_accurate_as_fp64(lib, Q, g, f16)
    if abs(rho - 1) <= 0.2:
        assert regular.all()


# exponents of the smallest and the largest deviation of a cell
@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("least,most", [(-10, -6), (-20, -4), (-30, -4), (-45, -4), (-30, 0), (-20, 6), (-6, 20)])
@pytest.mark.parametrize("f16", [False, True])
def test_shifted_sums_of_spread_deviations(lib, Q, least, most, f16):
    if f16 and most > 0:
        pytest.skip("FP16 storage holds deviations below 2")
    rng = np.random.default_rng(Q)
    g = (np.exp2(rng.uniform(least, most, (300, Q))) * rng.choice([-1.0, 1.0], (300, Q))).astype(np.float32)
    assert_as_accurate_as_fp64(lib, Q, as_stored(np.abs(g) if most >= 0 else g, f16), f16)


@pytest.mark.parametrize("Q", [19, 27])
def test_shifted_sums_at_the_edges(lib, Q):
    """Zeros, subnormals, the smallest and largest deviations the integers take,
    and the values that they leave to FP64."""
    edges = np.float32([0.0, 1e-45, 2.0 ** -126, 2.0 ** -62, 2.0 ** -61, 2.0 ** -60, 2.0 ** -38, 2.0 ** -30, 0.01,
                        np.nextafter(np.float32(0.125), np.float32(0)), 0.125, 0.3, 1e30, 3e38])
    rows = [np.where(np.arange(Q) == k, sign * e, np.float32(0)) for e in edges for sign in (1, -1) for k in (0, 5, Q - 1)]
    rows += [np.full(Q, sign * e) for e in edges[:-2] for sign in (1, -1)]
    g = np.float32(rows)
    out, regular = moments_shifted(lib, Q, g)
    assert regular[np.abs(g).max(axis=1) < 0.02].all() and not regular[np.abs(g).max(axis=1) >= 0.125].any()
    # per population: what a rounding of g + w in FP64 loses (half an ulp of 1/2 at most), and the sum's own rounding
    tol = 2 * Q * 2.0 ** -53 * (1 + np.abs(g.astype(np.float64)).sum(axis=1))
    assert (errors_shifted(Q, g, out).max(axis=1) <= tol).all()
    for bad in (np.inf, -np.inf, np.nan):
        g = np.zeros((1, Q), np.float32)
        g[0, 3] = bad
        out, regular = moments_shifted(lib, Q, g)
        assert not regular[0] and not np.isfinite(out[0, 0])
