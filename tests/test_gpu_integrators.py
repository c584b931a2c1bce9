"""The integrators row by row: blocks that read their rows directly (boundary, the first and
last soil rows), staged predictor rows, and a state large enough for staged corrector rows.
Each update is a product and a sum of values read back, so it holds to a few roundings."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, _abi, cases as C

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _near(a, b, *terms):
    """a == b up to four roundings of the terms summed."""
    size = sum(np.abs(t.astype(np.float64)) for t in terms)
    assert np.all(np.abs(a.astype(np.float64) - b) <= 4 * EPS * size)


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("size", ["few", "blocks", "staged corrector"])
def test_rows(size, threads, mixed):
    c = {"few": lambda: C.column_collapse(5, 4, 6, seed=3),
         "blocks": lambda: C.column_collapse(15, 15, 24, seed=4),
         "staged corrector": lambda: C.retaining_wall(140, 60, 90, seed=4)}[size]()
    assert (c.npb + c.npm >= 800000) == (size == "staged corrector")
    soil = slice(c.npb, None)
    c.velrhop[soil, :3] = np.random.default_rng(5).uniform(-0.05, 0.05, (c.npm, 3))
    s = LoquatSph(case=c)
    s.set_option(_abi.OPT_INTEGRATOR_THREADS, threads)
    s.set_option(_abi.OPT_MIXED_PRECISION, mixed)
    dt, two_h = s.info().dt, 2 * s.info().h
    get = lambda *names: [s.get(n)[soil].astype(np.float64) for n in names]  # noqa: E731
    start = {n: s.get(n) for n in ("pospres", "velrhop", "str", "stn", "cellpos")}
    s.step_calculation()
    s.predictor_section()
    for n in ("pospres", "velrhop", "str", "stn"):  # soil as it was, boundary rows as they are
        ini, now = s.get(n + "_ini"), s.get(n)
        np.testing.assert_array_equal(ini[soil], start[n][soil])
        np.testing.assert_array_equal(ini[:c.npb], now[:c.npb])
    p0, v0, e0, acc, D, p, v, e = get("pospres_ini", "velrhop_ini", "stn_ini", "accad", "acestn", "pospres",
                                      "velrhop", "stn")
    _near(v[:, :3], (v0 + acc * dt / 2)[:, :3], v0[:, :3], acc[:, :3] * dt)
    _near(p[:, :3], (p0 + v * dt / 2)[:, :3], p0[:, :3], v[:, :3] * dt)
    _near(e, e0 + D * dt / 2, e0, D * dt)
    s.corrector_section()
    D, p, v, e = get("acestn", "pospres", "velrhop", "stn")
    moved = (s.get("cellpos")[soil, :3].astype(np.float64) - start["cellpos"][soil, :3]) * two_h
    _near(p[:, :3] + moved, (p0 + (v0 + v) * dt / 2)[:, :3], p0[:, :3], (v0 + v)[:, :3] * dt, moved)
    _near(e, e0 + D * dt, e0, D * dt)
    s.close()
