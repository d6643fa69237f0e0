"""The tuner keeps the shape in use unless another one of its range is faster."""
import pytest

from dns_gkm_lpt_b200.solver import Solver
from tests.gpu_helpers import analytic_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_the_shape_in_use_is_a_candidate(precision):
    """13 faces in segments of 9 and 4: not one of the lengths n / k of the tuner's list, of which only 13 has 8
    faces or more, and faster than that one (each launch is one round of few CTAs that march their segments)."""
    P, W0 = analytic_case(13, 9)
    with Solver(P, cfl=0.5, precision=precision) as s:
        s.upload_state(W0)
        s.set_sweep_config([(0, 9)] * 3)
        assert [d["segment"] for d in s.autotune(10)] == [9, 9, 9]
