"""Transform lengths without a compile-time engine, and the z pass at the short lengths 32 and 64,
through the fused step and the grid solves against the FP64 oracle.

The grids put every radix of the runtime plans (2 to 16) and one to four stages on some axis,
lines shorter and longer than a warp, and lengths whose lines no longer fit the widest tile.
Tolerances as in the free-space tests: FP64 1e-10, FP32 1e-5.
"""
import numpy as np
import pytest

import openspacecharge_b200 as osc
from openspacecharge_b200.bunch import gendist
from conftest import field_err

pytestmark = pytest.mark.gpu
TOL = {osc.PREC_FP64: 1e-10, osc.PREC_FP32: 1e-5}
GRIDS = [(5, 6, 9), (15, 18, 20), (25, 27, 30), (36, 40, 45), (50, 54, 10), (75, 12, 24), (8, 81, 90), (12, 100, 8),
         (10, 8, 135), (125, 9, 6), (6, 240, 5), (8, 6, 300), (5, 5, 729), (6, 9, 1000), (1000, 5, 6), (6, 900, 5),
         (16, 20, 16), (12, 16, 32), (32, 32, 16)]


@pytest.mark.parametrize("prec", [osc.PREC_FP64, osc.PREC_FP32])
@pytest.mark.parametrize("n", GRIDS)
def test_step_matches_oracle(ctx, oracle, n, prec):
    x, y, z = gendist(3000, sigma=(1e-3, 1e-3, 1e-3), seed=5)
    q = np.random.default_rng(1).uniform(0.5e-13, 1.5e-13, len(x))
    om = oracle.make_mesh((1, 1, 1), n, (1, 1, 1), gamma=3.0)
    rho, _ = oracle.deposit_particles(x, y, z, om, qa=q, resize_mesh=True)
    e_ref, b_ref = oracle.space_charge_3d(om, rho, calc_bfield=True)
    E0, B0, _ = oracle.interpolate_field(om, e_ref, x, y, z, bfield=b_ref)
    for want_b in (False, True):
        m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, gamma=3.0)
        E, B = osc.space_charge_step(ctx, m, x, y, z, qa=q, resize_mesh=True, precision=prec, want_b=want_b)
        assert field_err(E, E0)[0] <= TOL[prec]
        if want_b:
            assert np.abs(B[:, :2] - B0[:, :2]).max() / np.abs(B0).max() <= TOL[prec]


@pytest.mark.parametrize("prec", [osc.PREC_FP64, osc.PREC_FP32])
@pytest.mark.parametrize("n", [(6, 9, 10), (10, 15, 40), (12, 8, 16), (16, 6, 32), (9, 10, 125)])
def test_cathode_and_phi_match_oracle(ctx, oracle, n, prec):
    rng = np.random.default_rng(2)
    rho = np.asfortranarray(rng.uniform(0.0, 1e-12, n))
    mn, dl = np.array([-1e-3, -1e-3, 2e-4]), np.array([1e-4, 1.2e-4, 0.9e-4])
    mx = mn + (np.array(n) - 1) * dl
    om = oracle.make_mesh((1, 1, 1), n, (1, 1, 1), mn, mx, dl, 2.0)
    e_ref, b_ref = oracle.space_charge_3d(om, rho, at_cathode=True, calc_bfield=True)
    m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=mn, max=mx, delta=dl, gamma=2.0)
    m.rho = rho
    osc.space_charge_3d(ctx, m, at_cathode=True, calc_bfield=True, precision=prec)
    assert field_err(m.efield, e_ref)[0] <= TOL[prec]
    assert np.abs(m.bfield - b_ref).max() / np.abs(b_ref).max() <= TOL[prec]
    _, p_ref = oracle.freespace_solver2(rho, 2.0, dl, want_phi=True)
    _, p = osc.osc_freespace_solver2(ctx, rho, 2.0, dl, efield=False, phi=True, precision=prec)
    assert np.abs(p - p_ref).max() / np.abs(p_ref).max() <= TOL[prec]
