"""Memory and streams that outlive a model: models made and dropped from several
threads at once give the bits they give one after another, and what stays with
the process after they are gone is bounded."""

import math
import threading

import numpy as np
import pytest

import gprx_b200 as gx

pytestmark = pytest.mark.gpu


def one(seed):
    rs = np.random.RandomState(seed)
    n, d = 150 + 61 * (seed % 7), 3
    x = rs.standard_normal(n * d)
    y = np.sin(x[:n]) + 0.1 * rs.standard_normal(n)
    g = gx.Gpr(gx.RbfArdKernel([0.7, 1.1, 1.6]), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed())
    m = g.factor(x, n, d, y)
    p = m.predict(x[:6 * d], 6, d)
    v, gr = m.value_and_gradient([math.log(0.8), math.log(1.0), math.log(1.5), math.log(0.06)])
    return np.concatenate([p.mean, p.variance, gr, [v]])


def test_models_from_several_threads_give_the_same_bits():
    seeds = list(range(24))
    expect = [one(s) for s in seeds]
    got = [None] * len(seeds)

    def work(k):
        for s in seeds[k::4]:
            got[s] = one(s)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(expect, got):
        assert np.array_equal(a, b)


def test_memory_kept_after_the_models_is_bounded():
    torch = pytest.importorskip("torch")
    one(0)
    free0 = torch.cuda.mem_get_info()[0]
    n, d = 6000, 2
    x = np.random.RandomState(1).standard_normal(n * d)
    for _ in range(3):  # 2 × 288 MB and more each
        m = gx.Gpr(gx.RbfKernel(0.5), gx.GaussianLikelihood(0.1)).with_optimizer(gx.Fixed()).factor(x, n, d, x[:n])
        m.value_and_gradient([math.log(0.5), math.log(0.1)])
        del m
    assert free0 - torch.cuda.mem_get_info()[0] <= (1 << 30) + (64 << 20)
