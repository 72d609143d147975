"""Predictions of more points than one pinned block's results: the chunks' edge,
against the same points asked for in two calls of the same solve class."""

import numpy as np
import pytest

import gprx_b200 as gx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [65535, 65536, 65537, 131073])
def test_chunks_meet(q):
    n, d = 40, 2
    rs = np.random.RandomState(4)
    x, xs = rs.standard_normal(n * d), rs.standard_normal((d, q))
    m = gx.Gpr(gx.RbfKernel(0.8), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(
        x, n, d, np.sin(x[:n]))
    p = m.predict(xs.reshape(-1), q, d)
    at = 33000
    a = m.predict(xs[:, :at].reshape(-1).copy(), at, d)
    b = m.predict(xs[:, at:].reshape(-1).copy(), q - at, d)
    assert np.array_equal(p.mean, np.concatenate([a.mean, b.mean]))
    assert np.array_equal(p.variance, np.concatenate([a.variance, b.variance]))
