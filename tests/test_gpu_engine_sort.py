"""The cell sort of a context in sparse, enlarged domains: digits of up to 11 bits, plans of two
and three passes, each tile size.  Particles are strewn over the grid, so the first search sorts;
the permutation is numpy's stable argsort of the keys."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, cases as C

pytestmark = pytest.mark.gpu


def _strewn(nx, ny, nz, cells):
    c = C.column_collapse(nx, ny, nz, seed=6)
    two_h = 2.0 * c.params["hdr"] * c.params["dr"]
    for ax in "xyz":  # `cells` per edge
        c.params[f"domain_size_{ax}"] = float(np.float32((cells - 0.5) * two_h))
    rng = np.random.default_rng(nx + cells)
    at = rng.uniform(two_h, (cells - 1.5) * two_h, (c.npb + c.npm, 3))
    at[::7] = at[0]  # a cell of many
    c.pospres[:, :3] = at.astype(np.float32)
    return c


# key bits: twice the cells and the deleted cell
@pytest.mark.parametrize("cells,bits", [(79, 20), (90, 21), (120, 22), (150, 23)])
@pytest.mark.parametrize("dims", [(9, 7, 11), (40, 40, 90), (82, 82, 80)])
def test_first_search_sorts_stably(dims, cells, bits):
    c = _strewn(*dims, cells)
    s = LoquatSph(case=c)
    inf = s.info()
    assert (inf.ncell - 1).bit_length() == bits and inf.np == c.npb + c.npm and inf.n_sorts == 1
    perm, key = s.get("part_idx"), s.get("cellpos")[:, 3]
    assert (np.sort(perm) == np.arange(inf.np)).all()
    before = np.empty_like(key)
    before[perm] = key
    np.testing.assert_array_equal(perm, np.argsort(before, kind="stable"))
    np.testing.assert_array_equal(s.get("idmassidx")[:, 2].astype(np.int64), perm)
    beg, end = s.get("cell_beg"), s.get("cell_end")
    occupied, first, count = np.unique(key, return_index=True, return_counts=True)
    np.testing.assert_array_equal(beg[occupied], first)
    np.testing.assert_array_equal(end[occupied], first + count)
    assert (beg >= 0).sum() == len(occupied)
    s.close()
