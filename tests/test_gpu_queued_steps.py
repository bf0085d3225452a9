"""Steps queued back to back, whose kernels may start before the one ahead of them has finished:
each result equals, bit by bit, that of the same step with the device idle before and after it (the
fixed-point deposit, whose sums do not depend on their order).  Grids on both sides of the launch
sizes up to which kernels start early, several meshes through one context (their work
arrays are the same memory)."""
import numpy as np
import pytest

import openspacecharge_b200 as osc
from openspacecharge_b200.bunch import gendist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [osc.PREC_FP32, osc.PREC_FP64])
@pytest.mark.parametrize("sizes", [[(8, 8, 16), (16, 16, 32)], [(45, 36, 50), (64, 64, 64), (16, 16, 16)],
                                   [(96, 96, 40), (128, 96, 64)]])
def test_queued_steps_match_idle_ones(sizes, prec):
    torch = pytest.importorskip("torch")
    ctx = osc.Context(0)
    ctx.set_option(osc.OPT_DEPOSIT_MODE, osc.DEPOSIT_DETERMINISTIC)
    cases = []
    for s, n in enumerate(sizes):
        for npart in (3000, 200_000):
            x, y, z = gendist(npart, seed=10 * s + npart)
            t = [torch.from_numpy(v).cuda() for v in (x, y, z)]
            cases.append((n, t, s % 2 == 1))

    def step(n, t, cathode, out):
        m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, gamma=3.0)
        osc.space_charge_step_dev(ctx, m, *t, out, total_charge=1e-9, resize_mesh=True, at_cathode=cathode,
                                  precision=prec)
        m2 = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=m.min.copy(), max=m.max.copy(), delta=m.delta.copy(), gamma=3.0)
        out2 = torch.empty_like(out)
        osc.space_charge_step_dev(ctx, m2, *t, out2, total_charge=2e-9, resize_mesh=False, at_cathode=cathode,
                                  precision=prec)
        return out2

    want = []
    for n, t, cat in cases:
        torch.cuda.synchronize()
        e1 = torch.empty(len(t[0]), 3, dtype=torch.float64, device="cuda")
        e2 = step(n, t, cat, e1)
        torch.cuda.synchronize()
        want.append((e1.cpu().numpy(), e2.cpu().numpy()))
    got = [torch.empty(len(c[1][0]), 3, dtype=torch.float64, device="cuda") for _ in range(3) for c in cases]
    got2 = [step(*cases[i % len(cases)], got[i]) for i in range(3 * len(cases))]
    torch.cuda.synchronize()
    for i in range(3 * len(cases)):
        for g, w in ((got[i], want[i % len(cases)][0]), (got2[i], want[i % len(cases)][1])):
            assert np.array_equal(g.cpu().numpy(), w)
    ctx.close()
