"""The pipelined plug point with the five component arrays lying in every way: one allocation, one with
room between the components, reversed, five allocations, and device memory."""
import ctypes as C

import numpy as np
import pytest
import torch

from dns_gkm_lpt_b200.solver import Solver
from tests.gpu_helpers import analytic_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["one", "gaps", "reversed", "separate", "device"])
@pytest.mark.parametrize("n", [20, 21, 48])
def test_component_arrays_of_the_plug_point(n, layout):
    P, W0 = analytic_case(n, 50 + n)
    cells = W0[0].size
    with Solver(P, cfl=0.5) as s:
        s.upload_state(W0)
        dt = s.timestep()
    want = torch.from_numpy(W0.copy()).pin_memory()
    with Solver(P, cfl=0.5) as s:
        s.set_pipeline(16, 2)
        s.evolve(want.numpy(), dt)
    if layout == "separate":
        parts = [torch.empty(cells, dtype=torch.float64, pin_memory=True) for _ in range(5)]
    else:
        step = cells + (10 if layout == "gaps" else 0)
        kind = dict(device="cuda") if layout == "device" else dict(pin_memory=True)
        whole = torch.full((5 * step,), -7.0, dtype=torch.float64, **kind)
        parts = [whole[q * step:q * step + cells] for q in range(5)]
        if layout == "reversed":
            parts.reverse()
    for q in range(5):
        parts[q].copy_(torch.from_numpy(W0[q].reshape(-1)))
    torch.cuda.synchronize()
    dp = C.POINTER(C.c_double)
    with Solver(P, cfl=0.5) as s:
        s._check(s.L.gkm_evolve(s.h, (dp * 5)(*[C.cast(C.c_void_p(x.data_ptr()), dp) for x in parts]), dt))
    torch.cuda.synchronize()
    for q in range(5):
        assert np.array_equal(parts[q].cpu().numpy().reshape(W0[q].shape), want.numpy()[q])
    if layout == "gaps":
        assert all((whole[(q + 1) * step - 10:(q + 1) * step] == -7.0).all() for q in range(5))
