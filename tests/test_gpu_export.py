"""rw_get_array: every array, small (one piece) and in several pieces of the device's export
buffer, against the fields it is put together from."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("n", [1, 9, 50])
def test_exported_rows(n, precision):
    c = C.column_collapse(n, n, 2 * n if n > 1 else 1, seed=2)
    s = LoquatSph(case=c, precision=precision)
    inf, idx = s.info(), s.get("idmassidx")[:, 2].astype(np.int64)
    f = np.float32 if precision == 4 else np.float64
    np.testing.assert_array_equal(s.get("str"), c.stress[idx].astype(f))
    np.testing.assert_array_equal(s.get("velrhop"), c.velrhop[idx].astype(f))
    cell, pos = s.get("cellpos"), s.get("pospres")
    two_h = f(2.0 * inf.h)
    want = pos.copy()
    want[:, :3] += cell[:, :3].astype(f) * two_h
    np.testing.assert_array_equal(s.get("pos_abs"), want)
    key, beg, end = cell[:, 3], s.get("cell_beg"), s.get("cell_end")
    np.testing.assert_array_equal(beg[key] <= np.arange(inf.np), True)
    np.testing.assert_array_equal(end[key] > np.arange(inf.np), True)
    assert (end - beg)[beg >= 0].sum() == inf.np and len(beg) == inf.ncell
    s.step(2)
    mag, var = s.get("contact_mag"), s.get("contact_var")
    assert mag.shape == (inf.np, 9) and var.shape == (inf.np, 4)
    mag2 = np.random.default_rng(1).normal(size=mag.shape).astype(f)
    s.set("contact_mag", mag2)
    np.testing.assert_array_equal(s.get("contact_mag"), mag2)
