"""Odd grids, whose device rows have a pitch: states pass through uploads, downloads, the pipelined plug
point and outputs unchanged, and a step of the tensor-copy sweeps matches the oracle."""
import numpy as np
import pytest
import torch

from dns_gkm_lpt_b200.solver import Solver
from tests.gpu_helpers import analytic_case, rel_l2

pytestmark = pytest.mark.gpu

FIELD_TOL = 1e-12   # as in the parity tests


@pytest.mark.parametrize("n,variant,segment", [(9, 0, 9), (15, 0, 4), (17, 1, 5), (33, 2, 16), (47, 1, 47)])
def test_odd_rows_round_trip_and_step(oracle, n, variant, segment):
    P, W0 = analytic_case(n, 70 + n)
    p = oracle.params(P, 0.5)
    ref = W0.copy()
    oracle.run(p, ref, 2, 0, None, stats=False)
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W0)
        assert np.array_equal(s.download_state(), W0)
        assert np.array_equal(s.download_state(), W0)      # the copy made for it leaves the state alone
        s.set_sweep_config([(variant, segment)] * 3)
        dt = s.timestep()
        s.evolve_eulerian(1)
        one = s.download_state()
        s.evolve_eulerian(1)
        assert rel_l2(s.download_state(), ref).max() <= FIELD_TOL
    pinned = torch.from_numpy(W0.copy()).pin_memory()
    with Solver(P, cfl=0.5) as s:
        s.evolve(pinned.numpy(), dt)
        kept = s.download_state()
    assert rel_l2(pinned.numpy(), one).max() <= 1e-13
    assert np.array_equal(kept, pinned.numpy())
