"""The division by a spline pivot through its tabled reciprocal (csrc/pivot_div.cuh) against IEEE
division, bit for bit: every pivot that a line of any length and end condition has, on the
numerators whose quotients lie nearest to a midpoint of two doubles (the only ones a wrong last
digit could come from: with q within 1.5 ulp of a/d and r rounded, the corrected quotient is within 3 2^-54
ulp of a/d before its rounding, and a quotient of 53-bit numbers that is no midpoint is at least 2^-54 ulp
away from one, rho 2^-54 for a remainder rho), and on random ones."""
import ctypes as C
import math
import os
import subprocess
import tempfile

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_dp = C.POINTER(C.c_double)


def _pivots():
    seen = set()
    for N in range(4, 64):
        d = 4.0   # natural ends
        for _ in range(2, N - 1):
            seen.add(d)
            d = 4.0 - 1.0 / d
        seen.add(d)
        d = 8.0   # periodic
        for i in range(1, N):
            seen.add(d)
            d = (4.25 if i == N - 1 else 4.0) - 1.0 / d
    return sorted(seen)


def _hard(d):
    """Numerators A 2^0 with A 2^k = M D + rho, M an odd 54-bit number (a midpoint), |rho| <= 8."""
    m, _ = math.frexp(d)
    D = int(m * 2 ** 53)
    D >>= (D & -D).bit_length() - 1
    out = []
    for k in range(48, 60):
        mod = 1 << k
        inv = pow(D, -1, mod)
        for rho in [r for r in range(-8, 9) if r]:
            M = (-rho * inv) % mod
            while M.bit_length() <= 54:
                if M.bit_length() == 54 and M % 2 and (M * D + rho) % mod == 0:
                    A = (M * D + rho) >> k
                    if 0 < A < 1 << 53:
                        out.append(float(A))
                M += mod
    return out


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(tempfile.mkdtemp(), "libpivot.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "dns_gkm_lpt_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "pivotnum.cpp"), "-o", out], check=True)
    L = C.CDLL(out)
    L.pn_in_range.argtypes = [C.c_double]
    L.pn_quotients.argtypes = [_dp, C.c_long, C.c_double, C.c_double, _dp]
    return L


@pytest.mark.parametrize("d", _pivots())
def test_quotient_is_the_rounded_division(lib, d):
    rng = np.random.default_rng(7)
    a = np.concatenate([_hard(d), rng.normal(size=20000) * 10.0 ** rng.uniform(-12, 12, 20000)])
    a = np.concatenate([a, -a, a * 2.0 ** 700, a * 2.0 ** -700])
    q = np.empty_like(a)
    lib.pn_quotients(a.ctypes.data_as(_dp), len(a), d, 1.0 / d, q.ctypes.data_as(_dp))
    assert np.array_equal(q, a / d)


def test_range_of_the_short_division(lib):
    for a in (0.0, -0.0, 1e-308, 5e-324, 2.0 ** -896, 2.0 ** 898, math.inf, -math.inf, math.nan):
        assert not lib.pn_in_range(a), a
    for a in (1.0, -1.0, 2.0 ** -895, 1.5 * 2.0 ** 896, 1e-200, -1e200):
        assert lib.pn_in_range(a), a
