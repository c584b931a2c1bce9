"""The walks of the interaction against the chunked kernel, which evaluates every pair by
itself: eight lanes per particle (a small case alone), and the packed walk of one thread per
particle (the same case beside a large one in a batch: two list entries at a time, predicated
sums).  Every sum is the same, so the states agree bit for bit."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, _abi, cases as C
from retainwall_code_b200.sph import Batch

pytestmark = pytest.mark.gpu

KEYS = ["pospres", "velrhop", "str", "accad", "acestn", "spin", "contact_mag", "contact_var"]


def _tension():
    """Stresses in tension: the artificial stress of both particles of a pair."""
    c = C.column_collapse(5, 4, 6, seed=3, model="dp")
    c.stress[c.npb:] *= np.where(np.arange(c.npm) % 3, 1.0, -0.5)[:, None]
    c.velrhop[c.npb:, :3] = np.random.default_rng(3).uniform(-0.05, 0.05, (c.npm, 3))
    return c


def _coincident():
    """Two pairs of particles at one place (r = 0), and one particle a rounding apart."""
    c = C.column_collapse(6, 5, 7, seed=4)
    p = c.pospres[c.npb:]
    p[11, :3] = p[10, :3]
    p[40, :3] = p[41, :3]
    p[40, 0] = np.nextafter(np.float32(p[41, 0]), np.float32(1.0))
    return c


def _not_finite():
    """A velocity and a stress that are not finite reach their neighbours within 2h only."""
    c = C.column_collapse(9, 9, 9, seed=5)
    c.velrhop[c.npb + 100, 0] = np.nan
    c.stress[c.npb + 620, 2] = -np.inf
    return c


def _no_viscosity():
    c = C.column_collapse(5, 5, 6, seed=6)
    c.params["viscosity_type"] = 0
    c.velrhop[c.npb:, :3] = np.random.default_rng(6).uniform(-0.05, 0.05, (c.npm, 3))
    return c


def _lone():
    """Particles out of every other's reach beside a small column: lists of one entry."""
    c = C.column_collapse(4, 4, 4, seed=7)
    c.pospres[c.npb + 63, 2] += 0.02
    c.pospres[c.npb + 60, 0] += 0.03
    return c


CASES = {
    "tension": (_tension, 3), "coincident": (_coincident, 2), "not finite": (_not_finite, 1),
    "no viscosity": (_no_viscosity, 5), "lone": (_lone, 5),
    # contact against a wall that moves in (slide flags), lists of every length mod 4
    "contact": (lambda: C.retaining_wall(nx=13, ny=7, nz=11, mode="passive", wall_speed=0.05, seed=8), 60),
    "one": (lambda: C.column_collapse(1, 1, 1, seed=9), 4),
}


def _step(sim, steps, beside):
    if not beside:
        sim.step(steps)
        return
    big = LoquatSph(case=C.retaining_wall(nx=40, ny=25, nz=20, seed=1), precision=sim.precision)
    batch = Batch([sim, big])
    batch.step(steps)
    batch.synchronize()
    batch.close()


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("skin", [0.02, 0.4])
@pytest.mark.parametrize("name", CASES)
def test_packed_walk_equals_single_pairs(name, skin, beside):
    make, steps = CASES[name]
    a, b = LoquatSph(case=make()), LoquatSph(case=make())
    a.set_option(_abi.OPT_LIST_SKIN, skin)
    b.set_option(_abi.OPT_INTERACTION_KERNEL, 1)
    _step(a, steps, beside)
    b.step(steps)
    for key in KEYS:
        np.testing.assert_array_equal(a.get(key), b.get(key), err_msg=key)
    assert a.list_stats()[1] == a.info().npm  # every particle walked a list


@pytest.mark.parametrize("beside", [False, True])
def test_walks_in_fp64(beside):
    """FP64 through cell changes (lists rebuilt, carried and updated), against the scan."""
    c = C.column_collapse(11, 9, 13, seed=11)
    c.velrhop[c.npb:, 0] = 0.5
    a, b = LoquatSph(case=c, precision=8), LoquatSph(case=c, precision=8)
    b.set_option(_abi.OPT_LIST_SKIN, 0.0)
    _step(a, 60, beside)
    b.step(60)
    for key in KEYS:
        np.testing.assert_array_equal(a.get(key), b.get(key), err_msg=key)
    assert a.info().n_list_updates > 0


@pytest.mark.parametrize("when", ["search", "write"])
def test_lists_dropped_between_stages(when):
    """Stage calls with the interaction kernel changed, or an array written, between the
    search and the boundary stage: no stale list is walked."""
    c = C.retaining_wall(nx=9, ny=6, nz=7, mode="passive", wall_speed=0.02, seed=3)
    a, b = LoquatSph(case=c), LoquatSph(case=c)
    a.step(3)
    b.step(3)
    for s in (a, b):
        s.set_option(_abi.OPT_LIST_SKIN, 0.0 if s is b else 0.02)
        if when == "search":
            s.set_option(_abi.OPT_INTERACTION_KERNEL, 1)
        s.step_calculation()
        s.neighbor_search(0)
        if when == "search":
            s.set_option(_abi.OPT_INTERACTION_KERNEL, 0)
        else:
            s.set("velrhop", s.get("velrhop"))
        s.rigid_body_update()
        s.adami_boundary()
        s.find_corner_particle()
    for key in KEYS:
        np.testing.assert_array_equal(a.get(key), b.get(key), err_msg=key)


def test_stage_calls_equal_steps_across_an_option():
    """Stage calls whose searches run as captured graphs (from the third step on), through
    cell changes and an option that drops the captures, against whole steps."""
    c = C.column_collapse(8, 7, 9, seed=12)
    c.velrhop[c.npb:, 0] = 5.0  # about 0.03 dx a step: the first cell changes after two steps
    a, b = LoquatSph(case=c), LoquatSph(case=c)

    def stages(n):
        for _ in range(n):
            a.step_calculation()
            a.predictor_section()
            a.corrector_section()
            a.end_step()

    stages(12)
    b.step(12)
    for s in (a, b):
        s.set_option(_abi.OPT_LIST_SKIN, 0.3)
    stages(12)
    b.step(12)
    for key in KEYS + ["cellpos", "codes"]:
        np.testing.assert_array_equal(a.get(key), b.get(key), err_msg=key)
    assert a.info().n_sorts > 3 and a.info().device_err == 0
