"""The first evaluation of a batch launches no tuning for problems whose tile shape
decides nothing."""

import math

import numpy as np
import pytest

import gprx_b200 as gx

pytestmark = pytest.mark.gpu


def test_small_problems_are_not_tuned():
    d, sizes = 7, [5, 64, 65, 128]
    ls = [1.0 + 0.1 * k for k in range(d)]
    rs = np.random.RandomState(1)
    xs = [rs.standard_normal(n * d) for n in sizes]
    b = gx.GprBatch(gx.ConstantKernel(1.5) * gx.RbfArdKernel(ls), xs, [np.sin(x[:n]) for x, n in zip(xs, sizes)], d)
    p = np.tile([math.log(v) for v in [1.5] + ls + [0.1]], (len(sizes), 1))
    count = gx._lib.lib().gprx_launch_count
    at = [count()]
    for _ in range(2):
        _, _, st = b.value_and_gradient(p)
        assert np.all(st == 0)
        at.append(count())
    assert at[1] - at[0] == at[2] - at[1]
