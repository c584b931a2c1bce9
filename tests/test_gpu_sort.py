"""The cell-key sort at the edges of its tiles, digits and runs of equal keys: stable, so the
permutation is numpy's stable argsort."""
import numpy as np
import pytest
import torch

from retainwall_code_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def _keys(n, max_key, kind, rng):
    if kind == "random":
        return rng.integers(0, max_key + 1, n)
    if kind == "equal":
        return np.full(n, max_key)
    k = np.sort(rng.integers(0, max_key + 1, n))  # sorted but for a few (a moving case's cells)
    at = rng.integers(0, n, max(1, n // 200))
    k[at] = rng.integers(0, max_key + 1, len(at))
    return k


@pytest.mark.parametrize("kind", ["random", "equal", "nearly sorted"])
@pytest.mark.parametrize("max_key", [0, 1, 255, 256, 65_535, 65_536, (1 << 24) - 1])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 131_072, 131_073, 524_289, 1 << 20])
def test_sort_is_numpys_stable_argsort(n, max_key, kind):
    keys = _keys(n, max_key, kind, np.random.default_rng(n + max_key)).astype(np.int32)
    d = torch.from_numpy(keys).cuda()
    s, p = torch.full_like(d, -1), torch.full_like(d, -1)
    check(lib().rw_cell_sort_noalloc(d.data_ptr(), n, max_key, s.data_ptr(), p.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream), "rw_cell_sort_noalloc")
    want = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(p.cpu().numpy(), want)
    np.testing.assert_array_equal(s.cpu().numpy(), keys[want])
