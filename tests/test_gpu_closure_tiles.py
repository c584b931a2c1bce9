"""The closure's integrators at the edges of their tiles (128 rows, one or two tiles a block at
a time, every block more than once): with a network whose outputs are never trusted each row
takes the exact rate, so the state is the plain method's."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, cases as C
from retainwall_code_b200.closure import Mlp, training_run
from tests._util import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (4, 4, 8), (5, 5, 10), (8, 8, 16), (40, 40, 75)])
def test_untrusted_rows_take_the_exact_rate(nx, ny, nz, precision):
    c = C.column_collapse(nx=nx, ny=ny, nz=nz, runout=1.0)
    net = Mlp(seed=3, sample_capacity=10_000)
    training_run(net, C.column_collapse(nx=8, ny=8, nz=16, runout=1.0), steps=4, every=2)
    p = net.params()
    p[-6:] = 1e6  # output biases far beyond every stored target
    net.set_params(p)
    clo, plain = LoquatSph(case=c, precision=precision), LoquatSph(case=c, precision=precision)
    clo.set_closure(net, margin=0.0)
    steps = 3
    clo.step(steps)
    plain.step(steps)
    st = clo.closure_stats()
    assert 0 < st["offered"] <= 2 * steps * c.npm and st["used"] == 0
    np.testing.assert_array_equal(clo.get("cellpos"), plain.get("cellpos"))
    for key in ("pospres", "velrhop", "str", "stn"):
        assert rel(clo.get(key), plain.get(key)) < 1e-6, key
    assert clo.info().device_err == 0
