"""The one-launch evaluation of at most 128 points (single models and batches):
every width of the kernel tree at the edges of the leaf and of the block, and
the state it leaves."""

import math

import numpy as np
import pytest

import gprx_b200 as gx
import oracle_lib as O

pytestmark = pytest.mark.gpu

TOL = 1e-10  # |a − e| / max(|e|, 1) against the oracle: the suite's FP64 bound

TREES = {
    "rbf": (2, [[10, 0]], [0.8], lambda: gx.RbfKernel(0.8)),
    "ard3": (3, [[11, 3]], [0.7, 1.1, 1.6], lambda: gx.RbfArdKernel([0.7, 1.1, 1.6])),
    "const_ard8": (8, [[2, 2], [12, 0], [11, 8]], [2.0] + [1.0 + 0.1 * k for k in range(8)],
                   lambda: gx.ConstantKernel(2.0) * gx.RbfArdKernel([1.0 + 0.1 * k for k in range(8)])),
    "ard12": (12, [[11, 12]], [1.5 + 0.1 * k for k in range(12)],
              lambda: gx.RbfArdKernel([1.5 + 0.1 * k for k in range(12)])),
    "sum3": (1, [[1, 3], [10, 0], [13, 0], [12, 0]], [0.8, 1.1, 2.0, 0.5],
             lambda: gx.RbfKernel(0.8) + gx.PeriodicKernel(1.1, 2.0) + gx.ConstantKernel(0.5)),
}


@pytest.mark.parametrize("tree", sorted(TREES))
@pytest.mark.parametrize("n", [1, 2, 16, 17, 63, 65, 112, 127, 128, 129])
def test_evaluation_alone_and_in_a_batch_matches_oracle(tree, n):
    d, nodes, theta, kernel = TREES[tree]
    rs = np.random.RandomState(n)
    x = rs.standard_normal(n * d)
    y = np.sin(x[:n]) + 0.1 * rs.standard_normal(n)
    params = np.array([math.log(v) for v in theta + [0.05]])
    nl_o, g_o, a_o, _ = O.exact_eval(nodes, params, x, n, d, y)
    m = gx.Gpr(kernel(), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(x, n, d, y)
    nl, g = m.value_and_gradient(params)
    assert O.rel_err(nl, nl_o) <= TOL and np.all(O.rel_err(g, g_o) <= TOL)
    assert np.all(O.rel_err(m.alpha(), a_o) <= 1e-9)  # α: the suite's bound
    assert m.stage_times_ms()["total"] > 0.0
    p = m.predict(x[:d].copy() if n == 1 else rs.standard_normal(3 * d), 1 if n == 1 else 3, d)
    assert np.all(np.isfinite(p.mean)) and np.all(p.variance > 0.0)
    nlb, gb, st = gx.GprBatch(kernel(), [x, x], [y, y], d).value_and_gradient(np.stack([params, params]))
    assert np.all(st == 0) and nlb[0] == nlb[1] and np.array_equal(gb[0], gb[1])
    assert O.rel_err(nlb[0], nl_o) <= TOL and np.all(O.rel_err(gb[0], g_o) <= TOL)
