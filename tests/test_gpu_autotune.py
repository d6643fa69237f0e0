"""The tuner keeps the shape in use unless another one is faster."""
import pytest

from dns_gkm_lpt_b200.solver import Solver
from tests.gpu_helpers import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_short_segments_of_small_cubes_survive(precision):
    """A 16^3 cube starts with segments of a few faces, several times faster than the eight or more of the
    tuner's list; set by hand to one segment it gets them back."""
    P, W0 = case(16, 0.3, 30.0, 9)
    with Solver(P, cfl=0.5, precision=precision) as s:
        s.upload_state(W0)
        assert all(d["segment"] < 8 for d in s.sweep_config())
        assert all(d["segment"] < 8 for d in s.autotune(5))
        s.set_sweep_config([(0, 16)] * 3)
        assert all(d["segment"] < 8 for d in s.autotune(5))
