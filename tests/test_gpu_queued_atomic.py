"""The default FP32 steps (quad-grid deposit by atomics, gathers in every particle order, B, charges
of the particles, the pipe) queued back to back on fixed meshes of several grids through one
context: their kernels start before the ones ahead have finished and their work arrays are the same
memory.  No two particles add to the same word (one to a cell, every other plane of cells), so the
results do not depend on the order of the atomics and equal, bit by bit, those of the same step with
the device idle before and after it."""
import numpy as np
import pytest

import openspacecharge_b200 as osc

pytestmark = pytest.mark.gpu
PIPE = (20e-3, 16e-3)


def make_case(torch, n, seed, npart):
    rng = np.random.default_rng(seed)
    d = np.array([1e-4, 1.2e-4, 1.5e-4])
    cells = np.array([n[0] - 1, n[1] - 1, (n[2] - 1) // 2])
    pick = np.sort(rng.choice(int(cells.prod()), size=min(npart, int(cells.prod())), replace=False))
    i, r = pick % cells[0], pick // cells[0]
    cell = np.stack([i, r % cells[1], 2 * (r // cells[1])])
    umin = -0.5 * d * np.array(n)
    p = umin[:, None] + (cell + rng.uniform(0.1, 0.9, cell.shape)) * d[:, None]
    m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=umin, max=umin + d * (np.array(n) - 1), delta=d, gamma=3.0)
    q = rng.uniform(0.5, 1.5, len(pick)) * 1e-13
    return m, [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (*p, q)]


@pytest.mark.parametrize("order", [osc.ORDER_ANY, osc.ORDER_CELL_SORTED, osc.ORDER_SORT])
@pytest.mark.parametrize("npart", [400, 150_000])
def test_queued_default_steps_match_idle_ones(order, npart):
    torch = pytest.importorskip("torch")
    grids = [(8, 8, 16), (45, 36, 50), (64, 64, 64), (16, 16, 32), (96, 96, 64)]
    cases = [make_case(torch, n, s, npart) for s, n in enumerate(grids)]
    with osc.Context(0) as ctx:
        ctx.set_option(osc.OPT_PARTICLE_ORDER, order)
        osc.osc_rectpipe_green(ctx, cases[3][0], *PIPE, precision=osc.PREC_FP32)
        kinds = [(c, use_q) for c in range(len(cases)) for use_q in (False, True)] + [("pipe", False), ("pipe", True)]

        def step(kind, use_q):
            m, (x, y, z, q) = cases[3 if kind == "pipe" else kind]
            out = [torch.empty((len(x), 3), dtype=torch.float64, device="cuda") for _ in range(2)]
            charge = dict(qa=q) if use_q else dict(total_charge=1e-9)
            if kind == "pipe":
                osc.space_charge_step_rectpipe_dev(ctx, m, x, y, z, out[0], *PIPE, B=out[1], **charge)
            else:
                osc.space_charge_step_dev(ctx, m, x, y, z, out[0], B=out[1], **charge)
            return out

        want = []
        for k in kinds:
            torch.cuda.synchronize()
            want.append(step(*k))
            torch.cuda.synchronize()
        got = [step(*kinds[i % len(kinds)]) for i in range(4 * len(kinds))]
        torch.cuda.synchronize()
        for i, g in enumerate(got):
            for a, b in zip(g, want[i % len(kinds)]):
                assert torch.isfinite(a).all() and torch.equal(a, b), kinds[i % len(kinds)]
