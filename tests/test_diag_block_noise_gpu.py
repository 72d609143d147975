"""The diagonal block's error where noise is small: a model of at most one block
against 80-bit arithmetic, next to what LAPACK's factor and solves lose on the same
inputs."""

import math

import numpy as np
import pytest

import gprx_b200 as gx
import oracle_lib as O

pytestmark = pytest.mark.gpu

WIDE = np.longdouble
SEEDS = 8


def kernel_matrix(x, ell, noise):
    xl = x.astype(WIDE)
    r2 = (xl[:, None] - xl[None, :]) ** 2
    return np.exp(-r2 / (2 * np.exp(WIDE(math.log(ell))) ** 2)) + np.exp(WIDE(math.log(noise))) * np.eye(x.size, dtype=WIDE)


def wide_solution(k, y):
    """NLML and α in 80 bits."""
    n = y.size
    c = k.copy()
    for j in range(n):
        c[j:, j] -= c[j:, :j] @ c[j, :j]
        c[j:, j] /= np.sqrt(c[j, j])
    z = y.astype(WIDE)
    for i in range(n):
        z[i] = (z[i] - c[i, :i] @ z[:i]) / c[i, i]
    a = z.copy()
    for i in range(n - 1, -1, -1):
        a[i] = (a[i] - c[i + 1:, i] @ a[i + 1:]) / c[i, i]
    return (y @ a + 2 * np.log(np.diag(c)).sum() + n * np.log(2 * WIDE(np.pi))) / 2, a


def lapack_solution(k, y):
    c = np.linalg.cholesky(k.astype(np.float64))
    a = np.linalg.solve(c.T, np.linalg.solve(c, y))
    return (y @ a + 2 * np.log(np.diag(c)).sum() + y.size * math.log(2 * math.pi)) / 2, a


# both factors are backward stable with the same constants up to the order of the sums:
# three times LAPACK's root-mean-square error over eight draws leaves room for that order
@pytest.mark.parametrize("noise", [1e-3, 1e-4, 1.1e-5])
@pytest.mark.parametrize("n", [17, 64, 100, 128])
def test_error_is_that_of_a_substitution(n, noise):
    ell, ours, theirs = 0.9, [], []
    for seed in range(SEEDS):
        rs = np.random.RandomState(1000 * seed + n)
        x = rs.uniform(0.0, 10.0, n)
        y = np.sin(x) + 0.1 * rs.standard_normal(n)
        k = kernel_matrix(x, ell, noise)
        nl, a = wide_solution(k, y)
        m = gx.Gpr(gx.RbfKernel(ell), gx.GaussianLikelihood(noise)).with_optimizer(gx.Fixed()).factor(x, n, 1, y)
        v, _ = m.value_and_gradient([math.log(ell), math.log(noise)])
        vb, _, st = gx.GprBatch(gx.RbfKernel(ell), [x], [y], 1).value_and_gradient(
            np.array([[math.log(ell), math.log(noise)]]))
        assert st[0] == 0
        lv, la = lapack_solution(k, y)
        scale = np.max(np.abs(a))
        ours.append([abs(v - nl) / abs(nl), abs(vb[0] - nl) / abs(nl), np.max(np.abs(m.alpha() - a)) / scale])
        theirs.append([abs(lv - nl) / abs(nl)] * 2 + [np.max(np.abs(la - a)) / scale])
    rms = [np.sqrt(np.mean(np.square(np.array(e, dtype=np.float64)), axis=0)) for e in (ours, theirs)]
    assert np.all(rms[0] <= 3.0 * rms[1]), rms


@pytest.mark.parametrize("n", [64, 128, 200])
def test_small_noise_matches_oracle(n):
    """κ(K) is 1e7 here: both sides carry κ·2^-53 = 1e-9 of the values they solve for."""
    rs = np.random.RandomState(n)
    x = rs.uniform(0.0, 10.0, n)
    y = np.sin(x) + 0.1 * rs.standard_normal(n)
    params = np.array([math.log(0.9), math.log(1.1e-5)])
    nl_o, g_o, a_o, _ = O.exact_eval([[10, 0]], params, x, n, 1, y)
    m = gx.Gpr(gx.RbfKernel(0.9), gx.GaussianLikelihood(1.1e-5)).with_optimizer(gx.Fixed()).factor(x, n, 1, y)
    nl, g = m.value_and_gradient(params)
    assert abs(nl - nl_o) <= 1e-9 * abs(nl_o)
    assert np.max(np.abs(g - g_o)) <= 1e-9 * np.max(np.abs(g_o))
    assert np.max(np.abs(m.alpha() - a_o)) <= 1e-8 * np.max(np.abs(a_o))
