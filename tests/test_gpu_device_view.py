"""The device state handed to callers: uploads wrap the ghosts of a live view, and the call needs no memory of its own."""
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


@pytest.fixture
def no_memory():
    """A call that takes the device's free memory but for a few MB, until the test ends."""
    held = []

    def take(leave=6 << 20):
        for _ in range(20):
            free = torch.cuda.mem_get_info()[0]
            if free <= 2 * leave:
                return
            try:
                held.append(torch.empty(free - leave, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                leave += 2 << 20
    yield take
    held.clear()
    torch.cuda.empty_cache()


def _view_round(s, W0, before_view=lambda: None):
    """States seen and left by a view, writes to it, a download, the tuner and two steps."""
    s.upload_state(W0)
    s.synchronize()
    before_view()
    view = s.device_state()
    seen = [view.cpu().numpy()]
    view[0] *= 1.01
    torch.cuda.synchronize()
    seen.append(s.download_state())
    s.autotune(1)
    seen.append(view.cpu().numpy())
    s.timestep()
    s.set_sweep_config([(0, 13)] * 3)
    s.evolve_eulerian(2)
    s.synchronize()
    return seen + [s.device_state().cpu().numpy(), s.download_state()]


def test_view_without_memory_for_its_buffer(no_memory):
    P, W0 = analytic_case(65, 4)   # its view takes 14 MB
    with Solver(P, cfl=0.5) as s:
        want = _view_round(s, W0)
    W1 = W0 * 1.0
    W1[0] *= 1.01
    assert np.array_equal(want[0], W0) and np.array_equal(want[1], W1) and np.array_equal(want[2], W1)
    with Solver(P, cfl=0.5) as s:
        got = _view_round(s, W0, no_memory)
        assert torch.cuda.mem_get_info()[0] < 5 * 71 ** 3 * 8
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_a_step_leaves_the_last_view_alone():
    """For callers whose streams still read it: its buffer is not the step's."""
    for n in (14, 15):
        P, W0 = analytic_case(n, 3)
        with Solver(P, cfl=0.5) as s:
            s.upload_state(W0)
            view = s.device_state()
            s.evolve_eulerian(1)
            s.synchronize()
            assert np.array_equal(view.cpu().numpy(), W0)


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
