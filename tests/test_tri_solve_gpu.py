"""The one-launch triangular solves (few right-hand sides) and the online
delete built on them, at the sizes where a block, a strip or a route ends."""

import math

import numpy as np
import pytest

import gprx_b200 as gx
import oracle_lib as O

pytestmark = pytest.mark.gpu

# |a − e| / max(|e|, 1) against the oracle: the suite's FP64 bound
TOL = 1e-10
ARD = [[11, 3]]


def data(n, d, seed):
    rs = np.random.RandomState(seed)
    x = rs.standard_normal(n * d)
    return x, np.sin(x[:n]) + 0.1 * rs.standard_normal(n), rs


def model(x, n, d, y):
    return gx.Gpr(gx.RbfArdKernel([0.7, 1.1, 1.6]), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(
        x, n, d, y)


PARAMS = np.array([math.log(v) for v in (0.7, 1.1, 1.6, 0.05)])


@pytest.mark.parametrize("n", [1, 15, 128, 129, 255, 257, 640, 1153, 2049])
@pytest.mark.parametrize("q", [1, 8, 9, 17, 150, 1200, 1201])
def test_predict_matches_oracle_in_every_class(n, q):
    d = 3
    x, y, rs = data(n, d, n + q)
    xs = rs.standard_normal(q * d)
    m = model(x, n, d, y)
    mo, vo = O.exact_predict(ARD, PARAMS, x, n, d, y, xs, q, 1)
    p = m.predict(xs, q, d)
    assert np.all(O.rel_err(p.mean, mo) <= TOL) and np.all(O.rel_err(p.variance, vo) <= TOL)


@pytest.mark.parametrize("n,few,many", [(700, 1, 150), (700, 290, 1100), (700, 1201, 3000), (1500, 1, 130)])
def test_queries_of_one_class_give_the_same_bits(n, few, many):
    # solves of few, mid and wide classes: the first `few` queries alone and
    # among `many` of the same class
    d = 3
    x, y, rs = data(n, d, 5)
    xs = rs.standard_normal((d, many))
    m = model(x, n, d, y)
    p = m.predict(xs.reshape(-1), many, d)
    one = m.predict(xs[:, :few].copy().reshape(-1), few, d)
    assert np.array_equal(one.mean, p.mean[:few]) and np.array_equal(one.variance, p.variance[:few])


def test_server_merges_predicts_of_one_class_only():
    # 20, 700 and 20 queries against 1500 points: the second is of another
    # class than the first, so each keeps the bits it has alone
    n, d = 1500, 3
    x, y, rs = data(n, d, 6)
    srv = gx.Server(workers=1)
    mid = srv.submit_fit(gx.RbfArdKernel([0.7, 1.1, 1.6]), gx.GaussianLikelihood(0.05), x, n, d, y,
                         optimizer=gx.Fixed())
    xs = [rs.standard_normal(q * d) for q in (20, 700, 20)]
    reqs = [srv.submit_predict(mid, v, v.size // d) for v in xs]
    for r in reqs:
        assert srv.wait(r[0])[0] == 0
    m = model(x, n, d, y)
    for (_, mean, var), v in zip(reqs, xs):
        p = m.predict(v, v.size // d, d)
        assert np.array_equal(mean, p.mean) and np.array_equal(var, p.variance)
    srv.close()


@pytest.mark.parametrize("n", [2, 128, 129, 300, 513])
def test_online_delete_anywhere_matches_oracle(n):
    d = 3
    x, y, rs = data(n, d, n)
    xs = rs.standard_normal(5 * d)
    for idx in sorted({0, n // 2, min(n - 1, 127), min(n - 1, 128), n - 1}):
        on = model(x, n, d, y).into_online()
        on.delete(on.point_ids()[idx])
        keep = np.delete(np.arange(n), idx)
        xk, yk = x.reshape(d, n)[:, keep].reshape(-1), y[keep]
        mo, vo = O.exact_predict(ARD, PARAMS, xk, n - 1, d, yk, xs, 5, 1)
        p = on.predict(xs, 5, d)
        assert np.all(O.rel_err(p.mean, mo) <= TOL) and np.all(O.rel_err(p.variance, vo) <= TOL)
