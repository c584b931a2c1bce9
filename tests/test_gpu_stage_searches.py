"""Searches of stage calls, run as captured graphs of their own, and what they share with the
rest of a host program: its captures and its option changes."""
import numpy as np
import pytest
import torch

from retainwall_code_b200 import LoquatSph, cases as C

pytestmark = pytest.mark.gpu

KEYS = ["pospres", "velrhop", "str", "cellpos"]


def _column():
    c = C.column_collapse(8, 7, 9, seed=12)
    c.velrhop[c.npb:, 0] = 5.0  # cells change from the third step on
    return c


def _stages(s, n):
    for _ in range(n):
        s.step_calculation()
        s.predictor_section()
        s.corrector_section()
        s.end_step()


@pytest.mark.parametrize("mode", ["global", "thread_local"])
def test_stage_calls_beside_a_capture(mode):
    """The host program captures a graph of its own on another stream meanwhile."""
    a, b = LoquatSph(case=_column()), LoquatSph(case=_column())
    x = torch.zeros(16, device="cuda")
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode=mode)
        x.add_(1)
        _stages(a, 8)
        x.add_(2)
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 3).all()
    b.step(8)
    for key in KEYS:
        np.testing.assert_array_equal(a.get(key), b.get(key), err_msg=key)
    assert a.info().n_search_skipped > 0  # gated searches ran
