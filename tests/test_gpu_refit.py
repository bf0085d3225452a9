"""The bounding box of a refit and the sum of the charges, each one launch whose last block
finishes the reduction: block edges, one block, every block resident and grids that loop, the
extremes at the first and the last particle, against the FP64 oracle and the exact sum; repeated,
since the block ticket must be back at zero after each launch."""
import math

import numpy as np
import pytest

import openspacecharge_b200 as osc
from openspacecharge_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npart", [2, 31, 256, 257, 148 * 8 * 256, 148 * 8 * 256 + 1])
def test_refit_and_charge_match_oracle(ctx, oracle, npart):
    rng = np.random.default_rng(npart)
    n = (9, 12, 16)
    for rep in range(2):
        x, y, z = rng.uniform(-1e-3, 1e-3, (3, npart)) * (1 + rep)
        for v, s in ((x, 1), (y, -1), (z, 1)):
            v[0], v[-1] = -s * 4e-3, s * 5e-3
        q = rng.uniform(-1e-12, 3e-12, npart)
        m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n)
        nout = osc.deposit_particles(ctx, x, y, z, m, qa=q, resize_mesh=True)
        om = oracle.make_mesh((1, 1, 1), n, (1, 1, 1), np.zeros(3), np.ones(3), np.ones(3), 1.0)
        ref, nref = oracle.deposit_particles(x, y, z, om, qa=q, resize_mesh=True)
        assert nout == nref
        for got, want in ((m.min, om.min), (m.max, om.max), (m.delta, om.delta)):
            assert np.abs(np.asarray(got) - np.asarray(want)).max() <= 1e-15 * 5e-3
        assert np.abs(m.rho - ref).max() <= 1e-12 * np.abs(ref).max()
        # a tree sum of n terms: at most (serial chunk + tree depth) roundings of the absolute sum
        chunk = -(-npart // (1024 * 256)) + 20
        assert abs(m.charge - math.fsum(q)) <= chunk * 2.0**-53 * np.abs(q).sum()


@pytest.mark.parametrize("where", [0, 300, -1])
def test_refit_refuses_non_finite_then_recovers(ctx, where):
    x, y, z = np.random.default_rng(7).uniform(-1, 1, (3, 70001))
    y[where] = np.inf
    m = osc.Mesh3D(nlo=(1, 1, 1), nhi=(8, 8, 8))
    with pytest.raises(osc.OscError) as ei:
        osc.deposit_particles(ctx, x, y, z, m, total_charge=1e-9, resize_mesh=True)
    assert ei.value.code == native.OSC_E_NAN
    y[where] = 0.5
    osc.deposit_particles(ctx, x, y, z, m, total_charge=1e-9, resize_mesh=True)
    assert np.isfinite(m.rho).all() and y.min() - 1e-6 <= m.min[1] < y.min()
