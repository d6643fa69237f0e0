"""Steps recorded into a caller's own CUDA graph order their particles each, as a replay does not know how
many steps have passed since the last ordering."""
import numpy as np
import pytest
import torch

from dns_gkm_lpt_b200.solver import Solver
from tests.gpu_helpers import case

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
