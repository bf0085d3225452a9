"""The cell integrals of the Green build (corner differences near the origin, the series of the
box average farther out) through the solves that use them.

Grids sit at the edges of the tiles and of the near region: grids that are near throughout, grids
with a few near tiles, cells much longer along one axis than the others.  The reference takes
the IGF primitives (osc_get_cgrn_freespace, code/open_spacecharge_mod.f90:648-747) in extended
precision: in FP64 their corner differences lose (r/h)^3 of the round-off, up to 1e-7 of a
component at these cells (the FP64 oracle's error there, not the solver's).  Tolerances: E as in
the other FP64 tests (1e-10), phi 1e-9, FP32 1e-5, of each component's largest value.
"""
import numpy as np
import pytest

import openspacecharge_b200 as osc
from conftest import field_err

pytestmark = pytest.mark.gpu
LD = np.longdouble
FPEI = float(np.float32(299792458.0) * np.float32(299792458.0)) * 1.00000000055e-7


def xprim(x, y, z):
    r = np.sqrt(x * x + y * y + z * z)
    return x * np.arctan((y * z) / (r * x)) - z * np.log(r + y) + y * np.log((r - z) / (r + z)) / 2


def pprim(x, y, z):
    r = np.sqrt(x * x + y * y + z * z)
    t = -(z * z * np.arctan(x * y / (z * r)) + y * y * np.arctan(x * z / (y * r)) + x * x * np.arctan(y * z / (x * r))) / 2
    return t + y * z * np.log(x + r) + x * z * np.log(y + r) + x * y * np.log(z + r)


def reference(rho, gamma, delta):
    """E (n, 3) and phi of the free-space solve."""
    n = rho.shape
    h = [LD(delta[0]), LD(delta[1]), LD(delta[2]) * LD(gamma)]
    u, v, w = [(np.arange(-n[d], n[d] + 1).astype(LD) - LD(0.5)) * h[d] for d in range(3)]
    u, v, w = u[:, None, None], v[None, :, None], w[None, None, :]
    full = tuple(2 * m for m in n)
    hat = np.fft.rfftn(rho, full, axes=(0, 1, 2))
    out = []
    for comp, f in enumerate((pprim(u, v, w), xprim(u, v, w), xprim(v, w, u), xprim(w, u, v))):
        g = f * (LD(gamma if comp in (1, 2) else 1.0) / (h[0] * h[1] * h[2]))
        for axis in range(3):
            g = np.diff(g, axis=axis)
        g = np.roll(g.astype(np.float64), [-m for m in n], (0, 1, 2))
        out.append(FPEI * np.fft.irfftn(hat * np.fft.rfftn(g), full, axes=(0, 1, 2))[:n[0], :n[1], :n[2]])
    return np.stack(out[1:], -1), out[0]


@pytest.mark.parametrize("gamma,delta", [(1.0, (1e-4, 1e-4, 1e-4)), (9.785, (1e-4, 1.3e-4, 2e-4)),
                                         (200.0, (1e-4, 1e-4, 1e-4)), (1.0, (2e-3, 1e-4, 1e-4)),
                                         (1.0, (1e-4, 1e-4, 1e-5))])
@pytest.mark.parametrize("n", [(2, 3, 4), (32, 8, 4), (36, 9, 5), (64, 18, 6), (30, 25, 40), (5, 4, 64)])
def test_solver2_matches_oracle(ctx, oracle, n, gamma, delta):
    rho = np.asfortranarray(np.random.default_rng(3).uniform(0.0, 1e-12, n))
    e_ref, p_ref = reference(rho, gamma, np.array(delta))
    for prec, tol_e, tol_p in ((osc.PREC_FP64, 1e-10, 1e-9), (osc.PREC_FP32, 1e-5, 1e-5)):
        e, p = osc.osc_freespace_solver2(ctx, rho, gamma, delta, efield=True, phi=True, precision=prec)
        mx, _ = field_err(e, e_ref)
        pm = np.abs(p - p_ref).max() / np.abs(p_ref).max()
        assert mx <= tol_e and pm <= tol_p, (prec, mx, pm)
