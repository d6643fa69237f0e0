"""The kernels' flux (moments in the peculiar frames) against the reference's moment algebra where
the two could part: ratios of specific heats whose internal degrees of freedom are not whole, and
normal velocities on both sides of the bound between the polynomials and the library functions of
the half-space moments (sqrt(lam) |U| = 1), up to supersonic.

Tolerance 1e-11 of each face's largest component, the bar of the golden faces: either form sums about
10^3 rounded products, none above some twenty times the largest component (2e-12)."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_dp = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(tempfile.mkdtemp(), "libhostnum.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "dns_gkm_lpt_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "hostnum.cpp"), "-o", out], check=True)
    L = C.CDLL(out)
    for f in (L.hn_flux_double, L.hn_flux_double_mcal):
        f.argtypes = [_dp, C.c_double, C.c_double, C.c_double, _dp]
    return L


@pytest.mark.parametrize("gam", [1.4, 1.3, 5.0 / 3.0, 1.2])
@pytest.mark.parametrize("x", [0.0, 1e-9, 0.3, -0.6, 1.0 - 1e-9, 1.0 + 1e-9, -1.0, 1.4, -2.0])
def test_peculiar_form_equals_mcal_form(lib, gam, x):
    rng = np.random.default_rng(int(1000 * (x + 3)))
    dx = 0.05
    for _ in range(40):
        rho, p = rng.uniform(0.5, 2.0), 1e5 * rng.uniform(0.5, 2.0)
        c = np.sqrt(p / rho)
        # sqrt(lam) U = x for both states (lam = rho / 2p) but for small jumps
        U = np.array([x * np.sqrt(2.0) * c, *rng.normal(0.0, 0.4 * c, 2)])

        def state(e):
            r, q, v = rho * (1 + e * rng.normal()), p * (1 + e * rng.normal()), U + e * c * rng.normal(size=3)
            return np.array([r, *(r * v), q / (gam - 1) + 0.5 * r * v @ v])

        scale = np.array([rho, rho * c, rho * c, rho * c, p])
        f = np.concatenate([state(0.02), state(0.02), state(1e-3), state(1e-3),
                            (0.1 / dx * scale * rng.normal(size=(6, 5))).ravel(), [1e-5 * 10 ** rng.uniform(-2, 1)]])
        a, b = np.zeros(5), np.zeros(5)
        dt = 0.3 * dx / (c * (2.0 + abs(x)))
        lib.hn_flux_double(f.ctypes.data_as(_dp), gam, dt, dx, a.ctypes.data_as(_dp))
        lib.hn_flux_double_mcal(f.ctypes.data_as(_dp), gam, dt, dx, b.ctypes.data_as(_dp))
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max(), (np.abs(a - b) / np.abs(b).max()).tolist()
