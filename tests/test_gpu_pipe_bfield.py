"""B of the FP32 pipe step: gathered from FP64 differences of the potential, not from E as it is
rounded to FP32 for its own gather.  B = beta/c (-E_y, E_x, 0) (as in code/open_spacecharge_mod.f90:456-461),
so B and E of one call differ by E's FP32 rounding and no more: within 2^-23 of the component's
largest value, and, at most of the particles, by more than FP64 round-off."""
import numpy as np
import pytest

import openspacecharge_b200 as osc
from openspacecharge_b200.bunch import gendist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 16, 16), (20, 18, 25), (32, 24, 64)])
def test_b_keeps_more_bits_than_the_fp32_field(ctx, n):
    torch = pytest.importorskip("torch")
    a, b, gam = 20e-3, 10e-3, 3.0
    x, y, z = gendist(4001, sigma=(2e-3, 1e-3, 1e-3), seed=9, pipe=(a, b), centroid=(3e-3, -1e-3, 0))
    lo, hi = np.array([x.min(), y.min(), z.min()]), np.array([x.max(), y.max(), z.max()])
    d = 1.01 * (hi - lo) / (np.array(n) - 2)
    umin = lo - 0.3 * d
    m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=umin, max=umin + (np.array(n) - 1) * d, delta=d, gamma=gam)
    osc.osc_rectpipe_green(ctx, m, a, b, precision=osc.PREC_FP32)
    t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, y, z)]
    E = torch.empty((len(x), 3), dtype=torch.float64, device="cuda")
    B = torch.empty_like(E)
    osc.space_charge_step_rectpipe_dev(ctx, m, *t, E, a, b, total_charge=1e-9, precision=osc.PREC_FP32, B=B)
    ctx.synchronize()
    E, B = E.cpu().numpy(), B.cpu().numpy()
    coef = np.sqrt(1 - 1 / gam**2) / 299792458.0
    assert np.all(B[:, 2] == 0)
    for got, want in ((B[:, 1] / coef, E[:, 0]), (-B[:, 0] / coef, E[:, 1])):
        err = np.abs(got - want) / np.abs(want).max()
        assert err.max() <= 2.0**-23
        assert np.median(np.abs(got - want) / np.abs(want)) >= 1e-10
