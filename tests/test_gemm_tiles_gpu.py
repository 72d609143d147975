"""The FP64 products of one evaluation and one Hessian at sizes on both sides of
the tile rule (32×64 below four 64×64 tiles a SM, 64×64 from there on), ragged
ones included, against the oracle."""

import math

import numpy as np
import pytest

import gprx_b200 as gx
import oracle_lib as O

pytestmark = pytest.mark.gpu

TOL = 1e-10  # |a − e| / max(|e|, 1): the suite's FP64 bound


@pytest.mark.parametrize("n", [257, 513, 1025, 2111, 2300])
def test_evaluation_on_both_sides_of_the_tile_rule(n):
    d = 4
    rs = np.random.RandomState(n)
    x = rs.standard_normal(n * d)
    y = np.sin(x[:n]) + 0.1 * rs.standard_normal(n)
    ls = [0.6, 0.9, 1.4, 2.0]
    params = np.array([math.log(v) for v in ls] + [math.log(0.05)])
    m = gx.Gpr(gx.RbfArdKernel(ls), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(x, n, d, y)
    nl_o, g_o, _, _ = O.exact_eval([[11, d]], params, x, n, d, y)
    nl, g = m.value_and_gradient(params)
    assert O.rel_err(nl, nl_o) <= TOL and np.all(O.rel_err(g, g_o) <= TOL)


def test_hessian_on_the_small_tile():
    n, d = 333, 2
    rs = np.random.RandomState(n)
    x = rs.standard_normal(n * d)
    y = np.sin(x[:n]) + 0.1 * rs.standard_normal(n)
    params = np.array([math.log(0.8), math.log(1.3), math.log(0.05)])
    m = gx.Gpr(gx.RbfArdKernel([0.8, 1.3]), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(x, n, d, y)
    h = m.hessian(params)
    h_o = O.exact_hessian([[11, d]], params, x, n, d, y)
    assert np.max(np.abs(h - h_o)) <= 1e-9 * max(np.max(np.abs(h_o)), 1.0)
