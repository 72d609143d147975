"""Evaluations of at most 128 points with more than 16 ARD dimensions: one launch
up to one 64x64 tile, separate ones from there on, against the oracle on both
sides of the line."""

import math

import numpy as np
import pytest

import gprx_b200 as gx
import oracle_lib as O

pytestmark = pytest.mark.gpu

TOL = 1e-10  # |a − e| / max(|e|, 1) against the oracle: the suite's FP64 bound


@pytest.mark.parametrize("d", [17, 32])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129])
def test_wide_trees_match_oracle(d, n):
    ls = [2.0 + 0.1 * k for k in range(d)]
    rs = np.random.RandomState(n)
    x = rs.standard_normal(n * d)
    y = np.sin(x[:n]) + 0.1 * rs.standard_normal(n)
    params = np.array([math.log(v) for v in ls + [0.05]])
    m = gx.Gpr(gx.RbfArdKernel(ls), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(x, n, d, y)
    nl, g = m.value_and_gradient(params)
    nl_o, g_o, a_o, _ = O.exact_eval([[11, d]], params, x, n, d, y)
    assert O.rel_err(nl, nl_o) <= TOL and np.all(O.rel_err(g, g_o) <= TOL)
    assert np.all(O.rel_err(m.alpha(), a_o) <= 1e-9)  # α: the suite's bound
