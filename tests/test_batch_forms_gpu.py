"""Every compiled form of the batched evaluation (width of the ARD leaf, bound of
the leaves) at the edges of its one-block and several-block paths."""

import math

import numpy as np
import pytest

import gprx_b200 as gx
import oracle_lib as O

pytestmark = pytest.mark.gpu

TOL = 1e-10  # |a − e| / max(|e|, 1) against the oracle: the suite's FP64 bound


def tree(d, leaves):
    """ARD trees of two or of four leaves; d = 0: isotropic ones."""
    ls = [1.0 + 0.1 * k for k in range(d)]
    lead = gx.RbfArdKernel(ls) if d else gx.RbfKernel(0.8)
    node, theta = ([11, d], ls) if d else ([10, 0], [0.8])
    if leaves == 2:
        return [[2, 2], [12, 0], node], [2.0] + theta, gx.ConstantKernel(2.0) * lead
    return ([[1, 2], [2, 2], [12, 0], node, [2, 2], [12, 0], [10, 0]], [2.0] + theta + [0.5, 1.3],
            gx.ConstantKernel(2.0) * lead + gx.ConstantKernel(0.5) * gx.RbfKernel(1.3))


@pytest.mark.parametrize("leaves", [2, 4])
@pytest.mark.parametrize("d", [0, 4, 8, 11])
def test_every_form_matches_oracle(d, leaves):
    nodes, theta, kernel = tree(d, leaves)
    dim = d or 2
    params = np.array([math.log(v) for v in theta + [0.05]])
    rs = np.random.RandomState(10 * d + leaves)
    sizes = [1, 64, 65, 128, 129, 200, 257]
    xs = [rs.standard_normal(n * dim) for n in sizes]
    ys = [np.sin(x[:n]) + 0.1 * rs.standard_normal(n) for x, n in zip(xs, sizes)]
    nl, g, st = gx.GprBatch(kernel, xs, ys, dim).value_and_gradient(np.tile(params, (len(sizes), 1)))
    assert np.all(st == 0)
    for i, n in enumerate(sizes):
        nl_o, g_o, _, _ = O.exact_eval(nodes, params, xs[i], n, dim, ys[i])
        assert O.rel_err(nl[i], nl_o) <= TOL and np.all(O.rel_err(g[i], g_o) <= TOL), n
