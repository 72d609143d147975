"""What an online model holds beyond its factor: the buffer that its deletes write to
is there for whoever asks for memory, and its results do not depend on it."""

import numpy as np
import pytest

import gprx_b200 as gx

pytestmark = pytest.mark.gpu


def model(n, d=2):
    x = np.random.RandomState(2).standard_normal(n * d)
    return gx.Gpr(gx.RbfKernel(0.5), gx.GaussianLikelihood(0.1)).with_optimizer(gx.Fixed()).factor(
        x, n, d, np.sin(x[:n]))


def test_a_deletes_buffer_goes_when_memory_is_asked_for():
    torch = pytest.importorskip("torch")
    n = 16000  # a factor of 2 GB, more than a pool keeps
    m = model(n).into_online()
    for at in (0, 17, n - 3):
        m.delete(int(m.point_ids()[at]))
    xs = np.linspace(-1.0, 1.0, 8)
    before = m.predict(xs, 4, 2)
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
    try:
        other = model(n)  # room for its factor is only there once the buffer has gone
        del other
        m.delete(int(m.point_ids()[5]))  # without one, a delete makes its own
        after = m.predict(xs, 4, 2)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.all(np.abs(after.mean - before.mean) < 0.1)
