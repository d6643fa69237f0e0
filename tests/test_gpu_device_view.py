"""The device state handed to callers: uploads wrap the ghosts of a live view, and the call needs no memory."""
import numpy as np
import pytest
import torch

from dns_gkm_lpt_b200.solver import Ensemble, Solver
from tests.gpu_helpers import analytic_case, rel_l2

pytestmark = pytest.mark.gpu


def _stale_ghosts(W0):
    """W0's interior inside ghosts of another gas (uploads wrap them, whatever they hold)."""
    W = W0 * 1.25
    sl = (slice(None),) + (slice(3, -3),) * 3
    W[sl] = W0[sl]
    return W


@pytest.mark.parametrize("n", [9, 10, 15])
def test_upload_wraps_the_ghosts_of_a_live_view(n):
    P, W0 = analytic_case(n, 40 + n)
    W1 = _stale_ghosts(W0)
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W1)
        dt, stats = s.timestep(), s.print_stats()
        s.evolve_eulerian(1)
        want = s.download_state()
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W0)
        view = s.device_state()
        s.upload_state(W1)
        s.synchronize()
        assert np.array_equal(view.cpu().numpy(), W0)
        assert np.array_equal(s.download_state(), W0)
        assert s.timestep() == dt
        assert s.print_stats() == stats
        s.evolve_eulerian(1)
        assert np.array_equal(s.download_state(), want)
    with Ensemble([dict(params=P, cfl=0.5)] * 2) as E:
        finals = []
        for live in (False, True):
            for m in range(2):
                E[m].upload_state(W0)
                if live:
                    E[m].device_state()
                E[m].upload_state(W1)
            E.step(2)
            E.synchronize()
            finals.append([E[m].download_state() for m in range(2)])
    for m in range(2):
        assert np.array_equal(finals[0][m], finals[1][m])


def test_device_state_of_an_odd_grid_allocates_nothing():
    P, W0 = analytic_case(65, 4)
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W0)
        s.evolve_eulerian(1)
        s.synchronize()
        before = torch.cuda.mem_get_info()[0]
        view = s.device_state()
        assert torch.cuda.mem_get_info()[0] == before   # 5 x 71^3 doubles: 14 MB
        assert np.array_equal(view.cpu().numpy(), s.download_state())


@pytest.mark.parametrize("n", [9, 10])
def test_a_live_view_outlasts_the_tuner(n):
    P, W0 = analytic_case(n, 60 + n)
    W1 = W0 * 1.0
    W1[0] *= 1.01
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W1)
        s.set_sweep_config([(0, 4)] * 3)
        s.evolve_eulerian(2)
        want = s.download_state()
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W0)
        view = s.device_state()
        s.autotune(1)
        assert np.array_equal(view.cpu().numpy(), W0)
        view[0] *= 1.01
        torch.cuda.synchronize()
        s.autotune(1)
        assert np.array_equal(view.cpu().numpy(), W1)
        s.timestep()
        s.set_sweep_config([(0, 4)] * 3)
        s.evolve_eulerian(2)
        assert np.array_equal(s.download_state(), want)
    with Ensemble([dict(params=P, cfl=0.5)] * 2) as E:
        views = []
        for m in range(2):
            E[m].upload_state(W0)
            views.append(E[m].device_state())
            views[m][0] *= 1.01
        torch.cuda.synchronize()
        E.autotune(1)
        for m in range(2):
            assert np.array_equal(views[m].cpu().numpy(), W1)
            assert np.array_equal(E[m].download_state(), W1)
            E[m].timestep()
        E.set_sweep_config([(0, 4)] * 3)
        E.step(2)
        E.synchronize()
        for m in range(2):
            assert rel_l2(E[m].download_state(), want).max() <= 1e-12   # as in the parity tests
