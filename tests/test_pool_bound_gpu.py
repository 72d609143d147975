"""What the pool keeps: more than its bound is held by several models at once, and
after they are gone no more than the bound stays with the process."""

import math

import numpy as np
import pytest

import gprx_b200 as gx

pytestmark = pytest.mark.gpu


def test_pooled_buffers_beyond_the_bound_go_back():
    torch = pytest.importorskip("torch")
    gx.Gpr(gx.RbfKernel(0.5), gx.GaussianLikelihood(0.1)).with_optimizer(gx.Fixed()).factor(
        np.arange(40.0), 20, 2, np.zeros(20))
    free0 = torch.cuda.mem_get_info()[0]
    n, d = 5600, 2  # matrices of 251 MB, the largest that are pooled: A and its inverse a model
    x = np.random.RandomState(1).standard_normal(n * d)
    models = []
    for _ in range(4):
        m = gx.Gpr(gx.RbfKernel(0.5), gx.GaussianLikelihood(0.1)).with_optimizer(gx.Fixed()).factor(x, n, d, x[:n])
        m.value_and_gradient([math.log(0.5), math.log(0.1)])
        models.append(m)
    # (what the pool kept from before may be among it)
    assert free0 - torch.cuda.mem_get_info()[0] >= 8 * 250e6 - (1 << 30)
    del m, models
    assert free0 - torch.cuda.mem_get_info()[0] <= (1 << 30) + (64 << 20)
