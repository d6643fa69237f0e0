"""The line solves of the velocity splines at the lengths where their paths change, against the oracle bit
for bit: lines resident in shared memory and streamed ones (three components per launch up to 200
points, one per launch up to 264), batches and their remainders, the rows before the pivots' fixed
point, and numerators that take the division instead of the short quotient (zeros, 1e-290)."""
import numpy as np
import pytest

from dns_gkm_lpt_b200 import ic
from dns_gkm_lpt_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,build", [(4, 2), (10, 1), (24, 2), (25, 1), (26, 2), (27, 1), (28, 2), (34, 2), (200, 2), (201, 2),
                                     (264, 1), (265, 1)])
@pytest.mark.parametrize("mode", [0, 1])
def test_coefficients_at_the_edges_of_the_line_kernels(oracle, mode, N, build):
    n = N if mode == 1 else N - 6
    if n < 4:
        pytest.skip("no natural grid has lines this short")
    rng = np.random.default_rng(N + mode)
    P = ic.Params(n=n, gam=1.4, den0=1.0, Mt=0.3, Re=30.0, mu0=0.9, p0=86100.0, t0=0.01)
    u = rng.normal(0.0, 100.0, (n, n, n))
    u[: n // 2, : n // 3] = 0.0                       # whole stretches of zeros
    v = rng.normal(size=(n, n, n)) * np.where(rng.random((n, n, n)) < 0.5, 1e-290, 1.0)
    W0 = ic.embed_ghost(np.stack([np.ones_like(u), u, v, np.zeros_like(u), np.full_like(u, 1e6)]))
    start, dinv = oracle.grid(oracle.params(P, 0.5), mode)
    with Solver(P, cfl=0.5, spline_mode=mode, spline_build=build) as s:
        s.upload_state(W0)
        s.generate_splines()
        for c in range(3 if N < 100 else 2):
            data = W0[1 + c]
            if mode == 1:
                data = np.ascontiguousarray(data[3:-3, 3:-3, 3:-3])
            _, ref = oracle.spline3d(data, mode, start, dinv)
            assert np.array_equal(s.spline_coefs(c), ref), c
