"""Uploads from and downloads to the device's own arrays, which odd grids read and write without staging."""
import ctypes as C

import numpy as np
import pytest
import torch

from dns_gkm_lpt_b200.solver import GkmError, Solver, _dp
from tests.gpu_helpers import analytic_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 9, 10, 31])
def test_device_arrays_round_trip(n):
    P, W0 = analytic_case(n, 50 + n)
    W1 = W0 * 1.25
    W1[:, 3:-3, 3:-3, 3:-3] = W0[:, 3:-3, 3:-3, 3:-3]   # ghosts that the upload has to wrap
    d = torch.from_numpy(W1).cuda()
    parts = [torch.full((W0[0].size + 2,), 7.0, dtype=torch.float64, device="cuda") for _ in range(5)]
    ptrs = (_dp * 5)(*[C.cast(C.c_void_p(p.data_ptr() + 8), _dp) for p in parts])   # 8 bytes off, apart
    with Solver(P, cfl=0.5) as s:
        s.upload_state(d)
        s.synchronize()
        assert np.array_equal(d.cpu().numpy(), W1)
        assert np.array_equal(s.download_state(), W0)
        out = torch.zeros_like(d)
        assert np.array_equal(s.download_state(out).cpu().numpy(), W0)
        s._check(s.L.gkm_download_state(s.h, ptrs))
        for q in range(5):
            got = parts[q].cpu().numpy()
            assert np.array_equal(got[1:-1], W0[q].ravel()) and got[0] == got[-1] == 7.0
        s.upload_state(W0 * 2.0)
        s._check(s.L.gkm_upload_state(s.h, ptrs))
        assert np.array_equal(s.download_state(), W0)
        view = s.device_state()
        view[0] *= 1.01
        torch.cuda.synchronize()
        W2 = view.cpu().numpy()
        assert np.array_equal(s.download_state(out).cpu().numpy(), W2)   # through the view
        s.upload_state(d)
        s.synchronize()
        assert np.array_equal(view.cpu().numpy(), W0)
        s.upload_state(view)   # the state's own view
        s.synchronize()
        assert np.array_equal(s.download_state(), W0)
        missing = (_dp * 5)(*[ptrs[q] for q in range(4)], None)
        for call in (s.L.gkm_download_state, s.L.gkm_upload_state):
            with pytest.raises(GkmError):
                s._check(call(s.h, missing))
