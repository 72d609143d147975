"""What a free waits for: models dropped in one thread leave another thread's
batched fits (which capture their rounds into a graph) alone, and neither side
sees an error that is not its own."""

import math
import threading

import numpy as np
import pytest

import gprx_b200 as gx

pytestmark = pytest.mark.gpu


def fits(count, out, errors):
    try:
        rs = np.random.RandomState(3)
        xs = [rs.standard_normal(n * 2) for n in (20, 33, 40, 27)]
        b = gx.GprBatch(gx.RbfKernel(0.8), xs, [np.sin(x[:x.size // 2]) for x in xs], 2)
        p = np.tile([math.log(0.8), math.log(0.1)], (len(xs), 1))
        for _ in range(count):
            out.append(b.fit(p, gx.Lbfgs(max_iterations=2)).params)
    except Exception as e:  # noqa: BLE001
        errors.append(e)


def test_models_dropped_beside_batched_fits():
    expect, errors = [], []
    fits(1, expect, errors)
    done = threading.Event()
    values = []

    def drop(n):
        rs = np.random.RandomState(n)
        x = rs.standard_normal(n * 2)
        try:
            while not done.is_set():
                m = gx.Gpr(gx.RbfKernel(0.7), gx.GaussianLikelihood(0.05)).with_optimizer(gx.Fixed()).factor(
                    x, n, 2, np.sin(x[:n]))
                for q in (3, 50):  # the second regrows the prediction's buffers
                    m.predict(x[:2 * q], q, 2)
                values.append((n, m.value_and_gradient([math.log(0.8), math.log(0.06)])[0]))
                del m
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    droppers = [threading.Thread(target=drop, args=(n,)) for n in (60, 150)]
    got = []
    fitter = threading.Thread(target=fits, args=(200, got, errors))
    for t in droppers + [fitter]:
        t.start()
    fitter.join()
    done.set()
    for t in droppers:
        t.join()
    assert not errors, errors[0]
    assert len(got) == 200 and all(np.array_equal(g, expect[0]) for g in got)
    for n in (60, 150):
        assert len({v for k, v in values if k == n}) == 1
