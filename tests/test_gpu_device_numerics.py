"""The sweeps' own reciprocal, inverse square root, wave speed and half-space functions as the device runs
them, against CUDA's operations and extended precision.  u = 2^-53 below.

Bounds.  recip and rsqrt_t: the ones they state.  Wave speed up to Mach 1: 7.5 u for the form with one
reciprocal and one inverse root (velocities 2 u each, |u|^2 7.1 u, c^2 7.6 u with the cancellation of the
kinetic energy, halved by the root) and 6 u for the reference's form.  gauss_small: coefficients rounded
to double and Horner's rule on them, at most 5.2 u (exp) and 5 u (erf), together below 8 u."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53
TINY = np.finfo(np.float64).tiny


@pytest.fixture(scope="module")
def run():
    out = os.path.join(tempfile.mkdtemp(), "libdevnum.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC,-ffp-contract=off", "-ccbin", "g++", "-cudart", "static",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "dns_gkm_lpt_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "devnum.cu"), "-o", out], check=True)
    L = C.CDLL(out)
    L.dn_run.argtypes = [C.c_int, C.c_void_p, C.c_long, C.c_void_p, C.c_void_p]

    def call(which, x):
        d = torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).cuda()
        a = torch.empty(len(x), dtype=torch.float64, device="cuda")
        b = torch.empty_like(a)
        torch.cuda.synchronize()
        assert L.dn_run(which, d.data_ptr(), len(x), a.data_ptr(), b.data_ptr()) == 0
        return a.cpu().numpy(), b.cpu().numpy()
    return call


def _normals(lo, hi):
    """Random mantissas, powers of two and their neighbours, for every exponent in [lo, hi)."""
    e = np.arange(lo, hi)
    rng = np.random.default_rng(11)
    m = np.concatenate([rng.uniform(1.0, 2.0, (200, len(e))), np.full((1, len(e)), 1.0), np.full((1, len(e)), 1.0 + 2 * U),
                        np.full((1, len(e)), 2.0 - 2 * U), np.full((1, len(e)), 1.5)])
    return np.ldexp(m, e).ravel()


def _ulps(a, b):
    """Steps between doubles of the same sign."""
    return np.abs(a.view(np.int64) - b.view(np.int64))


def test_reciprocal_within_one_step_of_the_division(run):
    x = _normals(-1022, 1021)
    x = np.concatenate([x, -x])
    mine, cuda = run(0, x)
    assert np.array_equal(cuda, 1.0 / x)
    assert _ulps(mine, cuda).max() <= 1
    mine, _ = run(0, np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 0.5 * TINY]))
    assert np.isnan(mine).all()


def test_inverse_root_within_two_ulp(run):
    x = _normals(-1022, 1024)
    mine, cuda = run(1, x)
    exact = 1 / np.sqrt(x.astype(np.longdouble))
    for got in (mine, cuda):
        assert (np.abs(got - exact) / np.spacing(exact.astype(np.float64))).max() <= 2.0
    mine, _ = run(1, np.array([0.0, -1.0, np.inf, np.nan]))
    assert np.isnan(mine).all()
    assert not np.isfinite(run(1, np.array([5e-324, 0.5 * TINY]))[0]).any()


def _states(rho, u, c):
    """Conserved states (n, 5) of speed u in a random direction and sound speed c, gamma = 1.4."""
    d = np.random.default_rng(12).normal(size=(len(rho), 3))
    v = d / np.linalg.norm(d, axis=1)[:, None] * u[:, None]
    p = rho * c * c / 1.4
    return np.column_stack([rho, rho[:, None] * v, p / 0.4 + 0.5 * rho * (v * v).sum(axis=1)])


def test_wave_speed_of_the_sweeps(run):
    rng = np.random.default_rng(13)
    n = 200_000
    rho, c = 10.0 ** rng.uniform(-6, 6, n), 10.0 ** rng.uniform(-2, 4, n)
    mach = np.concatenate([rng.uniform(0, 1, n // 2), 10.0 ** rng.uniform(-12, 0, n // 4), 10.0 ** rng.uniform(-160, -100, n // 4)])
    w = _states(rho, mach * c, c)
    w[:100, 1:4] = 0.0                       # gas at rest
    w[:100, 4] = rho[:100] * c[:100] ** 2 / 1.4 / 0.4
    mine, cuda = run(2, w)
    assert (np.abs(mine - cuda) / cuda).max() <= 13.5 * U
    bad = _states(np.ones(4), np.array([0.0, 1.0, 100.0, 1e-200]), np.ones(4))
    bad[:, 4] *= -1.0                        # pressure below zero
    bad = np.concatenate([bad, np.array([[0.0, 1, 1, 1, 1], [np.nan, 0, 0, 0, 1], [1, np.inf, 0, 0, 1], [1, 0, 0, 0, np.nan]])])
    assert not np.isfinite(run(2, bad)[0]).any()


def _half_erf(x):
    """erf(x / sqrt(2)) / 2 in extended precision by its power series."""
    t = x * x / 2
    term, total = np.ones_like(x), np.ones_like(x)
    for k in range(1, 40):
        term = -term * t / k
        total += term / (2 * k + 1)
    return x * total / np.sqrt(2 * np.longdouble("3.14159265358979323846264338327950288"))


@pytest.mark.parametrize("which,real,bound", [(3, np.float64, 8 * U), (4, np.float32, 8 * 2.0 ** -24)])
def test_half_space_polynomials(run, which, real, bound):
    r = np.sqrt(2.0)
    x = np.concatenate([np.linspace(-r, r, 100_001), 10.0 ** np.linspace(-300 if real is np.float64 else -30, 0, 3001)])
    x = x[x * x <= 2.0].astype(real).astype(np.float64)
    x = x[x != 0.0]
    ex, herf = run(which, x)
    X = x.astype(np.longdouble)
    assert (np.abs(ex - np.exp(-X * X / 2)) / np.exp(-X * X / 2)).max() <= bound
    ref = _half_erf(X)
    assert (np.abs(herf - ref) / np.abs(ref)).max() <= bound
