"""A device wait that gave up in a step that does not wait for the host is reported by the next
step that waits for its charges (as by any other call that waits), and the step after that runs.
The wait is made to run out without a fault (OSC_OPT_TEST_WAIT_TIMEOUT, as in
test_gpu_wait_timeout)."""
import pytest

import openspacecharge_b200 as osc
from openspacecharge_b200 import native
from openspacecharge_b200.bunch import gendist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [osc.DEPOSIT_ATOMIC, osc.DEPOSIT_DETERMINISTIC])
def test_step_with_charges_reports_the_earlier_step(mode):
    torch = pytest.importorskip("torch")
    n = (12, 10, 64)
    x, y, z = (torch.from_numpy(v).cuda() for v in gendist(5000, seed=5))
    q = torch.full_like(x, 2e-13)
    E = torch.empty((len(x), 3), dtype=torch.float64, device="cuda")
    with osc.Context(0) as ctx:
        ctx.set_option(osc.OPT_DEPOSIT_MODE, mode)
        m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, gamma=2.5)
        osc.space_charge_step_dev(ctx, m, x, y, z, E, total_charge=1e-9, resize_mesh=True)
        ctx.set_option(native.OPT_TEST_WAIT_TIMEOUT, 1)
        osc.space_charge_step_dev(ctx, m, x, y, z, E, total_charge=1e-9)
        ctx.set_option(native.OPT_TEST_WAIT_TIMEOUT, 0)
        with pytest.raises(osc.OscError) as ei:
            osc.space_charge_step_dev(ctx, m, x, y, z, E, qa=q)
        assert ei.value.code == native.OSC_E_TIMEOUT
        osc.space_charge_step_dev(ctx, m, x, y, z, E, qa=q)
        ctx.synchronize()
        assert m.charge == pytest.approx(1e-9, rel=1e-12) and torch.isfinite(E).all()
