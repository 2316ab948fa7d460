"""A swimmer whose 6 x 6 body matrix cannot be inverted: the step reports it and leaves the solved-for quantities, the
rates that the next step would advance with among them, as they were."""
import numpy as np
import pytest

from cufcm_fil_b200 import _lib

from .test_gpu_swim import make_swimmer

pytestmark = pytest.mark.gpu


def test_singular_body_matrix_keeps_the_rates():
    with make_swimmer(body_x0=[np.nan, 0.0, 0.0]) as s:
        before = s.state()
        with pytest.raises(_lib.CufilError) as e:
            s.step(0)
        assert e.value.code == _lib.CF_NONFINITE and "singular" in str(e.value)
        after = s.state()
    assert (before["phase_dot"] == 2 * np.pi).all()
    for key in ("phase_dot", "angle_dot", "body_q", "body_v"):
        np.testing.assert_array_equal(after[key], before[key])
