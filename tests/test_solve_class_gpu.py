"""The line between one cluster launch and the recursion: on both sides of it, by the
clusters that the device holds and by the blocks a CTA owns, against the oracle."""

import math

import numpy as np
import pytest

import gprx_b200 as gx
import oracle_lib as O

pytestmark = pytest.mark.gpu

TOL = 1e-10  # |a − e| / max(|e|, 1) against the oracle: the suite's FP64 bound
PARAMS = np.array([math.log(v) for v in (0.7, 1.1, 1.6, 0.05)])


# strips of 16 columns a cluster of 16, of 8, of 4, of 2; the last that one launch takes and the first that it does not
@pytest.mark.parametrize("n,q", [(2000, 112), (2000, 113), (2000, 240), (2000, 257), (1500, 528), (1500, 700),
                                 (3000, 112), (3000, 144), (513, 1200), (512, 390), (512, 391), (900, 1100),
                                 (1, 6001), (77, 6001), (128, 6000), (128, 6001), (129, 6001)])
def test_both_sides_match_oracle(n, q):
    d = 3
    rs = np.random.RandomState(n + q)
    x, xs = rs.standard_normal(n * d), rs.standard_normal(q * d)
    y = np.sin(x[:n]) + 0.1 * rs.standard_normal(n)
    m = gx.Gpr(gx.RbfArdKernel([0.7, 1.1, 1.6]), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(
        x, n, d, y)
    mo, vo = O.exact_predict([[11, 3]], PARAMS, x, n, d, y, xs, q, 1)
    p = m.predict(xs, q, d)
    assert np.all(O.rel_err(p.mean, mo) <= TOL) and np.all(O.rel_err(p.variance, vo) <= TOL)
