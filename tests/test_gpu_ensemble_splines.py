"""Ensembles whose members' spline lines differ in length: resident lines, several groups of them in a block, and
streamed lines give every member the coefficients of a single cube, bit for bit."""
import numpy as np
import pytest

from dns_gkm_lpt_b200.solver import Ensemble, Solver
from tests.gpu_helpers import analytic_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("sizes", [[12], [4, 12], [33, 4, 20, 9], [90, 9, 10, 21, 22, 23, 24, 25], [120] + [33] * 12,
                                   [194] + [40] * 8, [204, 7, 16]])
def test_members_splines_equal_single_cubes(sizes, mode):
    """One size; two to eight, packed or not by the largest; the longest resident lines (200 points) and longer."""
    cases = {n: analytic_case(n, 20 + n) for n in sizes}
    pos = np.random.default_rng(5).uniform(0, 2 * np.pi, (37, 3))
    with Ensemble([dict(params=cases[n][0], cfl=0.5, spline_mode=mode, max_particles=len(pos)) for n in sizes]) as E:
        for m, n in enumerate(sizes):
            E[m].upload_state(cases[n][1])
            E[m].particles_upload(pos)
        E.step(1)
        E.synchronize()
        for m, n in enumerate(sizes):
            s = E[m]
            built = [s.spline_coefs(c) for c in range(3)]   # of the stepped state, by the ensemble's launch
            W = s.download_state()
            with Solver(cases[n][0], cfl=0.5, spline_mode=mode) as one:
                one.upload_state(W)
                one.generate_splines()
                for c in range(3):
                    assert np.array_equal(built[c], one.spline_coefs(c)), (n, c)
