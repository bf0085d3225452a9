"""The scalar deposits (FP64 atomics and fixed point), where two lanes share a particle: counts that
leave part of a warp or of a block empty, particles outside and non-finite in between, charges,
against the FP64 oracle.  Tolerances: FP64 sums in any order, 1e-13 of the absolute sum a
node takes; fixed point, half a unit more per particle (the unit is 2^-62 of a power of two below
twice npart times the largest charge)."""
import numpy as np
import pytest

import openspacecharge_b200 as osc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_q", [False, True])
@pytest.mark.parametrize("mode", [osc.DEPOSIT_ATOMIC, osc.DEPOSIT_DETERMINISTIC])
@pytest.mark.parametrize("npart", [1, 15, 16, 17, 31, 32, 33, 255, 257, 148 * 64 * 256 + 5])
def test_deposit_matches_oracle(oracle, npart, mode, use_q):
    rng = np.random.default_rng(npart)
    n = (7, 9, 11)
    umin, delta = np.array([-1e-3, -2e-3, 0.5e-3]), np.array([3e-4, 4e-4, 5e-5])
    umax = umin + (np.array(n) - 1) * delta
    x, y, z = (rng.uniform(umin[d] - 0.3 * delta[d], umax[d] + 0.3 * delta[d], npart) for d in range(3))
    if npart > 20:
        x[3], z[18] = np.nan, np.inf
    q = rng.uniform(0.5e-15, 2e-15, npart) if use_q else None
    kw = dict(qa=q, total_charge=None if use_q else 1e-9, resize_mesh=False)
    om = oracle.make_mesh((1, 1, 1), n, (1, 1, 1), umin, umax, delta, 1.0)
    ok = np.isfinite(x) & np.isfinite(y) & np.isfinite(z)
    kwo = dict(kw, qa=q[ok] if use_q else None, total_charge=None if use_q else 1e-9 * ok.sum() / npart)
    ref, nref = oracle.deposit_particles(x[ok], y[ok], z[ok], om, **kwo)
    with osc.Context(0) as c:
        c.set_option(osc.OPT_DEPOSIT_MODE, mode)
        m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=umin.copy(), max=umax.copy(), delta=delta.copy())
        nout = osc.deposit_particles(c, x, y, z, m, **kw)
    assert nout == nref + (~ok).sum()
    tol = 1e-13 * np.abs(ref).max()
    if mode == osc.DEPOSIT_DETERMINISTIC:
        tol += npart * 0.5 * 2.0**-62 * (2 * npart * (q.max() if use_q else 1e-9 / npart))
    assert np.abs(m.rho - ref).max() <= tol
