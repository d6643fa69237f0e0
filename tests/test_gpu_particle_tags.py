"""Damaged particle tags are reported by every call that needs them, until particles are uploaded again."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest
import torch

from dns_gkm_lpt_b200 import _capi
from dns_gkm_lpt_b200.solver import GkmError, Solver
from tests.gpu_helpers import case

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _tags(s):
    out = os.path.join(tempfile.mkdtemp(), "libhandleptr.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-arch=sm_100a", "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-ccbin", "g++",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "dns_gkm_lpt_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "handleptr.cu"), "-o", out], check=True)
    L = C.CDLL(out)
    L.hp_tags.argtypes, L.hp_tags.restype = [C.c_void_p], C.c_void_p
    view = type("Tags", (), {})()
    view.__cuda_array_interface__ = {"shape": (s.np,), "typestr": "<i8", "data": (L.hp_tags(s.h), False), "version": 2}
    return torch.as_tensor(view, device="cuda:0")


@pytest.mark.parametrize("bad", [-1, 500])
def test_a_new_upload_ends_the_report_of_damaged_tags(bad):
    P, W0 = case(16, 0.3, 30.0, 3)
    rng = np.random.default_rng(3)
    pos = rng.uniform(0, 2 * np.pi, (500, 3))
    with Solver(P, cfl=0.5, max_particles=500) as s:
        s.upload_state(W0)
        s.particles_upload(pos)
        s.synchronize()
        tags = _tags(s)
        tags[7] = bad
        torch.cuda.synchronize()
        for call in (s.particles_download, s.particle_props, s.particles_download):
            with pytest.raises(GkmError) as ei:
                call()
            assert ei.value.status == _capi.GKM_ERR_STATE
        s.particles_upload(pos[:0])
        s.clock()
        s.particles_upload(pos)
        assert np.array_equal(s.particles_download()[0], pos)
        s.step(1)
        assert s.clock()[2] == 1
        s.particle_props()
