"""exp_tang over every argument a weight's exponent can have: exactly 0 from
-1024 down to -infinity (cycles with a particle thrown far out reach -1e15 and
beyond; the table index has room to -4.6e7), NaN for NaN.
"""
import numpy as np
import pytest

from tests.gpu_cases import pk

pytestmark = pytest.mark.gpu


def test_exp_tang_far_below_its_range():
    x = -np.concatenate([np.geomspace(1024.0, 1.7e308, 200001), [np.inf]])
    assert (pk.math_check(x)[:, 1] == 0.0).all()


def test_exp_tang_of_nan():
    x = np.array([np.nan, -np.nan])
    assert np.isnan(pk.math_check(x)[:, 1]).all()
