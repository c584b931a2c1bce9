"""Searches of stage calls, run as captured graphs of their own, and what they share with the
rest of a host program: its captures and its option changes."""
import numpy as np
import pytest
import torch

from retainwall_code_b200 import LoquatSph, _abi, cases as C

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


@pytest.mark.parametrize("every", [1, 2, 3, 5])
def test_options_set_between_steps(every):
    """A program that sets an option every few steps: captured searches are dropped each time,
    and made again after twice as many plain ones (2, 4, 8, ... steps), so soon not at all.
    Plain searches count none as skipped."""
    c = C.column_collapse(8, 7, 9, seed=12)  # at rest: every search is skipped once gated
    a, b = LoquatSph(case=c), LoquatSph(case=c)
    skipped = []
    for k in range(48):
        if k % every == 0:
            a.set_option(_abi.OPT_WALL_FRICTION, 0.5)
        _stages(a, 1)
        skipped.append(a.info().n_search_skipped)
    b.set_option(_abi.OPT_WALL_FRICTION, 0.5)
    b.step(48)
    for key in KEYS:
        np.testing.assert_array_equal(a.get(key), b.get(key), err_msg=key)
    made = sum(n > m for m, n in zip([0] + skipped, skipped))  # steps that ran gated searches
    assert made == sum(max(0, every - 2 ** k) for k in range(1, 10)), skipped
    _stages(a, 40)  # left alone, they come back
    assert a.info().n_search_skipped > skipped[-1] + 20
