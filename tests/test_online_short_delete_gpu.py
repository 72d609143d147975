"""Online deletes near the last point: at most 32 trailing rows take the one-warp
update, more the blocked one; both against the model without the point."""

import math

import numpy as np
import pytest

import gprx_b200 as gx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 34, 64, 130, 160])
def test_deletes_near_the_end_match_the_model_without_the_point(n):
    d = 2
    rs = np.random.RandomState(n)
    x = rs.standard_normal((d, n))
    y = np.sin(x[0]) + 0.1 * rs.standard_normal(n)
    xs = rs.standard_normal(3 * d)

    def factored(keep):
        return gx.Gpr(gx.RbfKernel(0.8), gx.GaussianLikelihood(0.1)).with_optimizer(gx.Fixed()).factor(
            x[:, keep].reshape(-1).copy(), len(keep), d, y[keep].copy())

    for idx in sorted({0, max(0, n - 34), max(0, n - 33), max(0, n - 32), n - 2, n - 1}):
        m = factored(list(range(n))).into_online()
        m.delete(int(m.point_ids()[idx]))
        e = factored([i for i in range(n) if i != idx])
        p, q = m.predict(xs, 3, d), e.predict(xs, 3, d)
        assert np.all(np.abs(p.mean - q.mean) <= 1e-10 * np.maximum(np.abs(q.mean), 1.0))
        assert np.all(np.abs(p.variance - q.variance) <= 1e-10 * np.maximum(np.abs(q.variance), 1.0))
        assert math.isclose(m.neg_log_marginal_likelihood(), e.neg_log_marginal_likelihood(), rel_tol=1e-10)
