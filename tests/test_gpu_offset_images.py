"""space_charge_3d with a displaced kernel and cathode images together (the offset adds to the
image's own displacement, code/open_spacecharge_mod.f90:472): neither set of spectra is even
or odd along z then, at the lengths that have an image z pass and at others, along z alone and along
every axis, against the FP64 oracle (tolerances as in the other free-space comparisons)."""
import numpy as np
import pytest

import openspacecharge_b200 as osc
from conftest import field_err
from test_gpu_freespace import PRECS, TOL, make_rho

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [(0.0, 0.0, 3e-4), (3e-4, -2e-4, 1e-3)])
@pytest.mark.parametrize("nz", [16, 20, 32, 48, 64, 96, 128])
@pytest.mark.parametrize("prec", PRECS)
def test_offset_with_images_matches_oracle(ctx, oracle, nz, off, prec):
    n = (12, 10, nz)
    rho, delta, umin, umax = make_rho(oracle, n, sigma=(1e-3, 1e-3, 2e-3), centroid=(0, 0, 6e-3), isetzmin=1)
    gamma = 2.5
    om = oracle.make_mesh((1, 1, 1), n, (1, 1, 1), umin, umax, delta, gamma)
    e_ref, b_ref = oracle.space_charge_3d(om, rho, offset=off, at_cathode=True, calc_bfield=True)
    m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=umin.copy(), max=umax.copy(), delta=delta.copy(), gamma=gamma)
    m.rho = rho
    osc.space_charge_3d(ctx, m, offset=off, at_cathode=True, calc_bfield=True, precision=prec)
    mx, rm = field_err(m.efield, e_ref)
    assert mx <= TOL[prec], (mx, rm)
    for c in range(2):
        bm = np.abs(m.bfield[..., c] - b_ref[..., c]).max() / np.abs(b_ref[..., c]).max()
        assert bm <= TOL[prec], (c, bm)


# both sides of the column counts up to which the doubled lengths 32 and 64 run a warp per column
# (7168 in FP32, 3584 in FP64)
@pytest.mark.parametrize("off", [(0.0, 0.0, 3e-4), (3e-4, -2e-4, 1e-3)])
@pytest.mark.parametrize("n", [(20, 81, 16), (24, 75, 16), (32, 108, 16), (30, 120, 32), (54, 64, 32), (64, 60, 32)])
@pytest.mark.parametrize("prec", [osc.PREC_FP64, osc.PREC_FP32])
def test_offset_with_images_matches_plain_path(ctx, oracle, n, off, prec):
    rho, delta, umin, umax = make_rho(oracle, n, sigma=(1e-3, 2e-3, 1e-3), centroid=(0, 0, 4e-3), isetzmin=1)
    got = []
    for p in (osc.PREC_FP64_PLAIN, prec):
        m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=umin.copy(), max=umax.copy(), delta=delta.copy(), gamma=2.5)
        m.rho = rho
        osc.space_charge_3d(ctx, m, offset=off, at_cathode=True, precision=p)
        got.append(m.efield)
    mx, rm = field_err(got[1], got[0])
    assert mx <= TOL[prec], (mx, rm)
