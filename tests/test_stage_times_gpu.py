"""Stage times of an evaluation: four stages that add up to the total, also where
one launch does all of them."""

import math

import numpy as np
import pytest

import gprx_b200 as gx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 40, 128, 129, 300])
def test_stages_add_up(n):
    rs = np.random.RandomState(n)
    x = rs.standard_normal(n * 2)
    m = gx.Gpr(gx.RbfKernel(0.8), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(
        x, n, 2, np.sin(x[:n]))
    m.value_and_gradient([math.log(0.8), math.log(0.05)])
    t = m.stage_times_ms()
    stages = [t[k] for k in ("fill", "factor", "inverse", "gradient")]
    assert all(s > 0.0 for s in stages)
    # the events' differences are single-precision milliseconds in steps of half a microsecond
    assert abs(sum(stages) - t["total"]) <= 4 * 0.0005 + 1e-6 * t["total"]
