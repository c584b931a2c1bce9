"""FP32 walks on velocities so small that the viscous quotient is subnormal (below 1.2e-38):
eight lanes per particle, the packed walk of one thread per particle and the chunked kernel
keep it alike."""
import numpy as np
import pytest

from retainwall_code_b200 import LoquatSph, _abi, cases as C

pytestmark = pytest.mark.gpu


def _drifting(nx, ny, nz, size):
    """Weightless, stressless soil with velocities of up to size: viscous forces only."""
    c = C.column_collapse(nx, ny, nz, seed=13)
    c.params.update(gravity_x=0.0, gravity_y=0.0, gravity_z=0.0)
    c.stress[:] = 0.0
    c.velrhop[c.npb:, :3] = np.random.default_rng(13).uniform(-size, size, (c.npm, 3))
    return c


@pytest.mark.parametrize("size", [1e-38, 1e-36, 1e-34])
@pytest.mark.parametrize("dims", [(6, 5, 7), (26, 26, 26)])  # eight lanes; one thread per particle
def test_subnormal_viscous_terms(dims, size):
    sims = [LoquatSph(case=_drifting(*dims, size)) for _ in range(2)]
    sims[1].set_option(_abi.OPT_INTERACTION_KERNEL, 1)
    for s in sims:
        s.step_calculation()
        s.neighbor_search(0)
        s.rigid_body_update()
        s.adami_boundary()
        s.find_corner_particle()
        s.particle_interaction()
    want = sims[1].get("accad")[sims[1].info().npb:, :3]
    assert (want != 0).any()
    np.testing.assert_array_equal(sims[0].get("accad"), sims[1].get("accad"))
