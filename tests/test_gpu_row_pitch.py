"""Odd grids, whose device rows have a pitch: states pass through uploads, downloads, the pipelined plug
point and outputs unchanged, and a step of the tensor-copy sweeps matches the oracle."""
import numpy as np
import pytest
import torch

from dns_gkm_lpt_b200.solver import Ensemble, Solver
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


@pytest.mark.parametrize("n", [9, 10, 15])
def test_device_state_is_the_state_until_the_next_step(n):
    """Reads of the view give the state, writes to it are the state for everything that follows, and
    uploads show in it; members of an ensemble likewise."""
    P, W0 = analytic_case(n, 90 + n)
    W1 = W0 * 1.0
    W1[0] *= 1.01
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W1)
        dt = s.timestep()
        stats = s.print_stats()
        s.step(1)
        want = s.download_state()
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W0)
        view = s.device_state()
        assert np.array_equal(view.cpu().numpy(), W0)
        view[0] *= 1.01
        torch.cuda.synchronize()
        assert np.array_equal(s.download_state(), W1)
        s.upload_state(W0)
        s.synchronize()
        assert np.array_equal(view.cpu().numpy(), W0)
        view[0] *= 1.01
        torch.cuda.synchronize()
        assert s.timestep() == dt
        assert s.print_stats() == stats
        s.step(1)
        assert np.array_equal(s.device_state().cpu().numpy(), want)
        assert np.array_equal(s.download_state(), want)
    with Ensemble([dict(params=P, cfl=0.5)] * 2) as E:
        for m in range(2):
            E[m].upload_state(W0)
            view = E[m].device_state()
            view[0] *= 1.01
        torch.cuda.synchronize()
        for m in range(2):
            E[m].timestep()
        E.step(1)
        E.synchronize()
        for m in range(2):
            assert rel_l2(E[m].device_state().cpu().numpy(), want).max() <= FIELD_TOL
