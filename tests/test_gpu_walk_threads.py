"""The walk's block size: the one a caller sets is the one in use, in small cases too; without
one the library decides by size and reports what it takes."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, _abi, cases as C

pytestmark = pytest.mark.gpu

# soil particles: eight lanes each, a thread each at up to two blocks of 128 per SM, and more
SIZES = {693: (9, 7, 11), 17280: (24, 24, 30), 54000: (30, 30, 60)}


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("n", SIZES)
def test_block_in_use(n, precision):
    make = lambda: LoquatSph(case=C.column_collapse(*SIZES[n], seed=3), precision=precision)  # noqa: E731
    default, narrow, wide = make(), make(), make()
    assert default.info().walk_threads == (64 if precision == 8 and n == 17280 else 128)
    for s, threads in ((narrow, 64), (wide, 128)):
        s.set_option(_abi.OPT_WALK_THREADS, threads)
        assert s.info().walk_threads == threads
    for s in (default, narrow, wide):
        s.step(3)
    for key in ("pospres", "velrhop", "str"):
        for s in (narrow, wide):
            np.testing.assert_array_equal(default.get(key), s.get(key), err_msg=key)
