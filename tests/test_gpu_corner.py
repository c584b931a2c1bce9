"""The corner search takes its contact-wall candidates from the kept lists in two passes
(collect, then visit); scanning the boundary cells visits the same ones in the same order, so
the contact state agrees bit for bit."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, _abi, cases as C

pytestmark = pytest.mark.gpu

KEYS = ["contact_var", "contact_mag", "pospres", "velrhop", "str"]


def _dense_wall(layers):
    """A wall of `layers` times as many particles per layer: candidates past the capacity
    of one collection (32), and lists that overflow and scan."""
    c = C.retaining_wall(nx=9, ny=6, nz=7, mode="passive", wall_speed=0.02, seed=3)
    wall = np.flatnonzero(c.codes[:c.npb, 0] >= 10)
    extra = np.concatenate([wall] * (layers - 1)) if layers > 1 else wall[:0]
    shift = np.repeat(np.arange(1, layers), len(wall))[:, None] * c.params["dr"] * np.array([0.0, 0.23, 0.31])
    ins = lambda a, b: np.concatenate([a[:c.npb], b, a[c.npb:]])  # noqa: E731
    pos = c.pospres[extra].copy()
    pos[:, :3] += shift
    c.pospres, c.codes = ins(c.pospres, pos), ins(c.codes, c.codes[extra])
    c.velrhop, c.idmassidx = ins(c.velrhop, c.velrhop[extra]), ins(c.idmassidx, c.idmassidx[extra])
    c.stress, c.strain = ins(c.stress, c.stress[extra]), ins(c.strain, c.strain[extra])
    c.normal = np.concatenate([c.normal, c.normal[extra]])
    c.idmassidx[:, 2] = np.arange(len(c.idmassidx))
    c.params.update(np=len(c.codes), npb=len(c.normal))
    return c


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("layers", [1, 2, 3])
def test_collected_candidates_equal_the_scan(layers, precision):
    a, b = LoquatSph(case=_dense_wall(layers), precision=precision), LoquatSph(case=_dense_wall(layers), precision=precision)
    b.set_option(_abi.OPT_LIST_SKIN, 0.0)
    a.step(8)
    b.step(8)
    for key in KEYS:
        np.testing.assert_array_equal(a.get(key), b.get(key), err_msg=key)
    assert (a.get("contact_var")[a.info().npb:, 1] < 999).any()  # some particles met the wall
