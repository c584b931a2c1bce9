"""Closure training kernel at the edges of its tiles (128 samples a tile, a tile or more a
block): the gradient against the emulated arithmetic, and one update's direction."""
import numpy as np
import pytest

from oracle import mlp_oracle as M
from tests.test_mlp import _block_errors, _features, _params, _target

pytestmark = pytest.mark.gpu

# Five layers, each rounding its values to BF16 (spacing 2^-8 of a value): a value near a tie
# may round the other way once a layer.
TOL = 5 * 2.0 ** -8


@pytest.mark.parametrize("n", [1, 127, 128, 129, 148 * 128, 148 * 128 + 1])
def test_gradient_at_tile_edges(n):
    from retainwall_code_b200.closure import Mlp

    net = Mlp(seed=41)
    p = _params(42)
    net.set_params(p)
    x = _features(n, 43)
    t = _target(x)
    loss, g = net.grad(x, t)
    le, ge = M.loss_grad(p, x, t, emulate=True)
    assert abs(loss - le) <= TOL * le
    for off, e in _block_errors(g, ge).items():
        assert e < TOL, (off, e)
    net.close()


@pytest.mark.parametrize("n", [128, 1000])
def test_first_update_follows_the_gradient(n):
    """From zero moments an update moves each parameter by its rate against its gradient's sign,
    where the sign is certain (above the bound on its block's error).  A call's last update,
    here its only one, has a twentieth of the rate."""
    from retainwall_code_b200.closure import Mlp

    net = Mlp(seed=51, sample_capacity=n)
    p = _params(52)
    net.set_params(p)
    x = _features(n, 53)
    t = _target(x)
    net.add_samples(x, t)
    lr = 1e-2
    net.train(epochs=1, batch=n, lr=lr, seed=1)
    _, ge = M.loss_grad(p, x, t, emulate=True)
    d = net.params() - p
    for off, shp in M.SHAPES:
        k = int(np.prod(shp))
        gb, db = ge[off:off + k], d[off:off + k]
        sure = np.abs(gb) > 2 * TOL * np.linalg.norm(gb)
        np.testing.assert_allclose(db[sure], -lr / 20 * np.sign(gb[sure]), rtol=1e-3)
    net.close()
