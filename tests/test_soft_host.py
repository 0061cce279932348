"""The integer double additions of the exact FP64 collision, compiled for the
host, against the machine's own: equal bits (tolerance 0) over their ranges and
at the edges of them, where rounding can go wrong: ties, sticky bits, powers of
two, zeros and sums that cancel."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
N = 200000


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    out = tmp_path_factory.mktemp("soft") / "libsoft.so"
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", "-I", str(ROOT / "lbmminiapp_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "soft_check.cu"), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


def p(a):
    return ctypes.c_void_p(a.ctypes.data)


def same(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


def populations(rng, shape, short):
    """Values in [2^-10, 1/4); short: few significant bits, so that sums tie."""
    d = np.exp2(rng.uniform(-10, -2, shape))
    if short:
        bits = rng.integers(1, 54, shape)
        e = np.floor(np.log2(d))
        d = np.ldexp(np.floor(np.ldexp(d, (bits - e).astype(int))), -(bits - e).astype(int))
    return np.clip(d, 2.0 ** -10, np.nextafter(0.25, 0))


@pytest.mark.parametrize("short", [False, True])
@pytest.mark.parametrize("m", [2, 10, 19])
def test_signed_running_sums(lib, m, short):
    rng = np.random.default_rng(m)
    d = populations(rng, (N // m, m), short)
    sign = np.where(rng.random(d.shape) < 0.5, 1, -1).astype(np.int8)
    d[:5] = 2.0 ** -10                      # sums that cancel to zero
    ref = np.zeros(len(d))
    ok = np.ones(len(d), bool)
    for k in range(m):
        ref = ref + sign[:, k] * d[:, k]
        ok &= np.abs(ref) < 2
    out = np.empty(len(d))
    lib.soft_sums(p(d), p(sign), len(d), m, p(out))
    assert same(out[ok], ref[ok])


@pytest.mark.parametrize("short", [False, True])
def test_positive_running_sums(lib, short):
    rng = np.random.default_rng(3)
    m = 7
    d = populations(rng, (N // m, m), short)
    ref = d[:, 0].copy()
    for k in range(1, m):
        ref = ref + d[:, k]
    out = np.empty(len(d))
    lib.soft_positive_sums(p(d), len(d), m, p(out))
    assert same(out, ref)


@pytest.mark.parametrize("least", [-3, -12, -40, -80, -1070])
def test_polynomial(lib, least):
    rng = np.random.default_rng(-least)
    c = np.exp2(rng.uniform(least, -0.16, N)) * np.where(rng.random(N) < 0.5, 1, -1)
    c[::7] = np.ldexp(rng.integers(1, 8, len(c[::7])).astype(float), -rng.integers(4, 70, len(c[::7])))
    c[::11] = 0.0
    c[5] = -0.0
    q = 0.5 * c * c
    h = np.exp2(rng.uniform(min(least, -8), -4.5, N))
    h[::13] = np.ldexp(1.0, -rng.integers(6, 80, len(h[::13])))
    h[::17] = 0.0
    out = np.empty(N)
    lib.soft_polynomial(p(c), p(q), p(h), N, p(out))
    assert same(out, ((1.0 + c) + q) - h)


def test_addition(lib):
    """Inside the range, at its edges and outside (where it is the machine's)."""
    rng = np.random.default_rng(11)
    b = np.exp2(rng.uniform(-13, -1.5, N))
    a = np.exp2(rng.uniform(-60, -1.5, N)) * np.where(rng.random(N) < 0.5, 1, -1)
    a[::5] = -b[::5] * rng.choice([1.0, 0.5, 0.999, 1.0 - 2.0 ** -50, 2.0 ** -20], len(b[::5]))   # cancellation
    a[::7] = np.ldexp(rng.integers(1, 16, len(a[::7])).astype(float), -rng.integers(4, 75, len(a[::7])))
    a[::11] = 0.0
    a[3], b[3] = -0.0, 2.0 ** -12
    edges = [2.0 ** -12, np.nextafter(2.0 ** -12, 0), 0.25, np.nextafter(0.25, 0), 2.0 ** -10, 2.0 ** -62, 2.0 ** -64,
             5e-324, 2.2250738585072014e-308, 1e300, np.inf]
    k = 100
    for x in edges:
        for y in edges:
            a[k], b[k] = x, y
            a[k + 1], b[k + 1] = -x, y
            k += 2
    out = np.empty(N)
    lib.soft_add(p(a), p(b), N, p(out))
    with np.errstate(all="ignore"):
        ref = a + b
    fine = ~np.isnan(ref)
    assert same(out[fine], ref[fine]) and np.isnan(out[~fine]).all()


def test_fixed_point_to_double(lib):
    rng = np.random.default_rng(5)
    v = rng.integers(-2 ** 62, 2 ** 62, N) >> rng.integers(0, 62, N)
    v[::3] = (v[::3] & ~0x7FF) | 0x400      # ties
    v[:3] = [0, 1, -1]
    out = np.empty(N)
    lib.fixed62(p(v), N, p(out))
    assert same(out, np.ldexp(v.astype(np.float64), -62))
