"""Steps recorded into a caller's own CUDA graph: they order their particles each, as a replay does not know how
many steps have passed since the last ordering, and take in a live device view when they are recorded."""
import numpy as np
import pytest
import torch

from dns_gkm_lpt_b200.solver import Solver
from tests.gpu_helpers import analytic_case, case

pytestmark = pytest.mark.gpu


def test_captured_steps_order_their_particles():
    P, W0 = case(16, 0.3, 30.0, 8)
    pos = np.random.default_rng(8).uniform(0, 2 * np.pi, (60_000, 3))
    with Solver(P, cfl=0.5, max_particles=len(pos)) as s:
        s.upload_state(W0)
        s.particles_upload(pos)
        s.step(5)
        want, want_pos = s.download_state(), s.particles_download()
    with Solver(P, cfl=0.5, max_particles=len(pos), use_graphs=False) as s:
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        s.upload_state(W0)
        s.particles_upload(pos)
        before = s.launch_count()
        s.step(1)   # the first step after an upload orders the particles
        ordered = s.launch_count() - before
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        before = s.launch_count()
        with torch.cuda.graph(g, stream=stream):
            s.step(2)
        assert s.launch_count() - before == 2 * ordered
        with torch.cuda.stream(stream):
            g.replay()
            g.replay()
        s.synchronize()
        assert np.array_equal(s.download_state(), want)
        for a, b in zip(s.particles_download(), want_pos):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("n", [14, 15])
def test_captured_steps_and_the_device_state(n, late):
    """Writes to the device state before the recording, or between it and the first replay, count; replays after the
    first step on from their own result, and every later call sees it."""
    P, W0 = analytic_case(n, 30 + n)
    W1 = W0 * 1.0
    W1[0] *= 1.01
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W1)
        dt = s.timestep()
        s.set_dt(dt)
        s.evolve_eulerian(2)
        half = s.download_state()
        s.evolve_eulerian(2)
        want = s.download_state()
    with Solver(P, cfl=0.5, use_graphs=False) as s:
        s.set_dt(dt)
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        s.upload_state(W0)
        if not late:
            s.device_state()[0] *= 1.01
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            view = s.device_state()
            s.evolve_eulerian(2)
        if late:
            view[0] *= 1.01
            torch.cuda.synchronize()
            assert np.array_equal(s.download_state(), W1)
        with torch.cuda.stream(stream):
            g.replay()
            if late:
                assert np.array_equal(s.download_state(), half)
            g.replay()
        s.synchronize()
        assert np.array_equal(s.device_state().cpu().numpy(), want)
        assert np.array_equal(s.download_state(), want)
        s.upload_state(W1)
        s.evolve_eulerian(2)
        s.synchronize()
        assert np.array_equal(s.device_state().cpu().numpy(), half)


@pytest.mark.parametrize("n", [14, 15])
def test_recorded_splines_leave_later_states_alone(n):
    """Splines recorded while a device view was live, replayed after steps of the host: no old view comes back."""
    P, W0 = analytic_case(n, 60 + n)
    with Solver(P, cfl=0.5) as s:
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        s.upload_state(W0)
        s.device_state()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            s.generate_splines()
        s.evolve_eulerian(2)
        want = s.download_state()
        with torch.cuda.stream(stream):
            g.replay()
        s.synchronize()
        assert np.array_equal(s.download_state(), want)
