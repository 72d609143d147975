"""The diagonal-block step (16-wide leaves, 128-wide blocks) at the sizes where
a leaf or a block ends, through one evaluation and one factor."""

import math

import numpy as np
import pytest

import gprx_b200 as gx
import oracle_lib as O

pytestmark = pytest.mark.gpu

# |a − e| / max(|e|, 1) against the oracle: the suite's FP64 bound
TOL = 1e-10


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 47, 95, 111, 112, 113, 127, 128, 129, 143, 145, 250])
def test_leaf_edges_match_oracle(n):
    d = 2
    rs = np.random.RandomState(n)
    x = rs.standard_normal(n * d)
    y = np.sin(x[:n]) + 0.1 * rs.standard_normal(n)
    params = np.array([math.log(0.9), math.log(0.02)])
    m = gx.Gpr(gx.RbfKernel(0.9), gx.GaussianLikelihood(0.02)).with_optimizer(gx.Fixed()).factor(x, n, d, y)
    nl_o, g_o, a_o, _ = O.exact_eval([[10, 0]], params, x, n, d, y)
    assert O.rel_err(m.neg_log_marginal_likelihood(), nl_o) <= TOL
    nl, g = m.value_and_gradient(params)
    assert O.rel_err(nl, nl_o) <= TOL and np.all(O.rel_err(g, g_o) <= TOL)


@pytest.mark.parametrize("n,dup", [(20, 3), (40, 17), (130, 127), (130, 129)])
def test_a_repeated_point_in_any_leaf(n, dup):
    # a pivot of about twice the noise among pivots of one: the leaf's longest
    # cancellation, in its first, a middle and its last column
    rs = np.random.RandomState(n + dup)
    x = 3.0 * np.arange(n, dtype=float)
    x[dup] = x[0]
    y = rs.standard_normal(n)
    params = np.array([math.log(0.5), math.log(0.01)])
    m = gx.Gpr(gx.RbfKernel(0.5), gx.GaussianLikelihood(0.01)).with_optimizer(gx.Fixed()).factor(x, n, 1, y)
    nl_o, g_o, _, _ = O.exact_eval([[10, 0]], params, x, n, 1, y)
    nl, g = m.value_and_gradient(params)
    assert O.rel_err(nl, nl_o) <= TOL and np.all(O.rel_err(g, g_o) <= TOL)
