"""The boundary extrapolation with one thread per particle (a case beside so many boundary
particles that eight lanes each would cost more) through carried and updated lists: bit for
bit the scan of the cells, which reads no boundary row's velocity or stress."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, _abi, cases as C
from retainwall_code_b200.sph import Batch

pytestmark = pytest.mark.gpu

KEYS = ["pospres", "velrhop", "str", "contact_mag", "contact_var"]


def _column():
    c = C.column_collapse(11, 9, 13, seed=11)
    c.velrhop[c.npb:, 0] = 0.5
    return c


def _wall():
    """Contact walls list their own boundary rows beside the soil."""
    c = C.retaining_wall(nx=13, ny=7, nz=11, mode="passive", wall_speed=0.05, seed=8)
    c.velrhop[c.npb:, 0] = 0.5
    return c


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("make", [_column, _wall])
def test_thread_per_particle_through_list_updates(make, precision):
    a, b = LoquatSph(case=make(), precision=precision), LoquatSph(case=make(), precision=precision)
    big = C.retaining_wall(nx=150, ny=80, nz=4, seed=1)
    assert big.npb > 40960
    beside = LoquatSph(case=big, precision=precision)
    b.set_option(_abi.OPT_LIST_SKIN, 0.0)
    batch = Batch([a, beside])
    for _ in range(3):
        batch.step(20)
        batch.synchronize()
        b.step(20)
        for key in KEYS:
            np.testing.assert_array_equal(a.get(key), b.get(key), err_msg=key)
    assert a.info().n_list_updates > 0 and a.info().device_err == 0
    batch.close()
