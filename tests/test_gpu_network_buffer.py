"""Device memory of network calls on host arrays: kept, grown and given back without waiting
for work on other streams."""
import numpy as np
import pytest
import torch

from retainwall_code_b200.closure import Mlp

pytestmark = pytest.mark.gpu


def _samples(n):
    rng = np.random.default_rng(n)
    return (rng.uniform(-1, 1, (n, 16)).astype(np.float32), rng.uniform(-1, 1, (n, 6)).astype(np.float32))


def test_calls_do_not_wait_for_other_streams():
    a, b = Mlp(seed=7), Mlp(seed=7)
    b.set_params(a.params())
    sizes = [100, 300, 5000, 800_000, 20_000, 800_000]  # the buffer grows; too large to keep
    data = {n: _samples(n) for n in sizes}
    x, t = data[100]
    b.forward(x), b.grad(x, t)  # the kernels are loaded
    side, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(3_000_000_000)  # about 1.5 s on one SM
        done.record(side)
    got = {n: (a.forward(data[n][0]), a.grad(*data[n])) for n in sizes}
    waited = done.query()
    torch.cuda.synchronize()
    assert not waited
    for n in sizes:  # in a fresh network with the same parameters, smallest last
        y, (loss, g) = got[n]
        np.testing.assert_array_equal(y, b.forward(data[n][0]))
        loss2, g2 = b.grad(*data[n])
        assert abs(loss - loss2) <= 1e-12 * loss2  # float atomics leave the gradient's order open
        np.testing.assert_allclose(g, g2, rtol=0, atol=1e-5 * np.abs(g2).max())
    a.close()
    b.close()
