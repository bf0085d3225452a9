"""B at the particles from the fused steps, which form it from the gathered field, against the FP64
oracle: free space and cathode, every particle order, odd particle counts, and the pipe.
Tolerances as for E: FP64 1e-10, FP32 1e-5 of the largest component."""
import numpy as np
import pytest

import openspacecharge_b200 as osc
from openspacecharge_b200.bunch import gendist
from conftest import field_err

pytestmark = pytest.mark.gpu
TOL = {osc.PREC_FP64: 1e-10, osc.PREC_FP32: 1e-5}


@pytest.mark.parametrize("npart", [1, 31, 4099])
@pytest.mark.parametrize("order", [osc.ORDER_ANY, osc.ORDER_CELL_SORTED, osc.ORDER_SORT])
@pytest.mark.parametrize("cathode", [False, True])
@pytest.mark.parametrize("n", [(12, 15, 32), (32, 16, 20)])
@pytest.mark.parametrize("prec", [osc.PREC_FP64, osc.PREC_FP32])
def test_step_b_matches_oracle(oracle, n, cathode, order, npart, prec):
    x, y, z = gendist(5000, sigma=(1e-3, 1e-3, 1e-3), seed=3, centroid=(0, 0, 5e-3))
    mn = np.array([v.min() for v in (x, y, z)])
    mx = np.array([v.max() for v in (x, y, z)])
    dl = (mx - mn) / (np.array(n) - 1)
    x, y, z = (v[:npart].copy() for v in (x, y, z))
    om = oracle.make_mesh((1, 1, 1), n, (1, 1, 1), mn, mx, dl, 4.0)
    rho, _ = oracle.deposit_particles(x, y, z, om, total_charge=1e-10, resize_mesh=False)
    e_ref, b_ref = oracle.space_charge_3d(om, rho, at_cathode=cathode, calc_bfield=True)
    E0, B0, _ = oracle.interpolate_field(om, e_ref, x, y, z, bfield=b_ref)
    with osc.Context(0) as c:
        c.set_option(osc.OPT_PARTICLE_ORDER, order)
        m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=mn.copy(), max=mx.copy(), delta=dl.copy(), gamma=4.0)
        E, B = osc.space_charge_step(c, m, x, y, z, total_charge=1e-10, resize_mesh=False, at_cathode=cathode,
                                     precision=prec, want_b=True)
    # one particle: its own field cancels at its place, so the scale is the grid's field
    scale_e, scale_b = np.abs(e_ref).max(), np.abs(b_ref).max()
    assert np.abs(E - E0).max() / scale_e <= TOL[prec]
    assert np.abs(B - B0).max() / scale_b <= TOL[prec]
    assert np.all(B[:, 2] == 0)
