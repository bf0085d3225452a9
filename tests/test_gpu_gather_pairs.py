"""The FP64 step's gather, where two lanes share a particle: counts that leave part of a warp empty,
particles at the faces and outside (clamped), against the FP64 oracle.  Tolerance 1e-10 of the largest
component, as for every FP64 step."""
import numpy as np
import pytest

import openspacecharge_b200 as osc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npart", [1, 2, 15, 16, 17, 31, 32, 33, 257])
@pytest.mark.parametrize("cathode", [False, True])
def test_fp64_step_matches_oracle(ctx, oracle, npart, cathode):
    n = (6, 9, 16)
    rng = np.random.default_rng(npart)
    umin, delta = np.array([-1e-3, -2e-3, 0.5e-3]), np.array([4e-4, 5e-4, 2e-4])
    umax = umin + (np.array(n) - 1) * delta
    x, y, z = (rng.uniform(umin[d] + 0.01 * delta[d], umax[d] - 0.01 * delta[d], npart) for d in range(3))
    x[-1], y[0] = umax[0] + 0.2 * delta[0], umin[1]
    om = oracle.make_mesh((1, 1, 1), n, (1, 1, 1), umin, umax, delta, 2.0)
    rho, _ = oracle.deposit_particles(x, y, z, om, total_charge=1e-10, resize_mesh=False)
    e_ref, _ = oracle.space_charge_3d(om, rho, at_cathode=cathode)
    E0, _, _ = oracle.interpolate_field(om, e_ref, x, y, z)
    m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=umin.copy(), max=umax.copy(), delta=delta.copy(), gamma=2.0)
    E, _ = osc.space_charge_step(ctx, m, x, y, z, total_charge=1e-10, resize_mesh=False, at_cathode=cathode,
                                 precision=osc.PREC_FP64)
    assert np.abs(E - E0).max() <= 1e-10 * max(np.abs(e_ref).max(), 1e-300)
