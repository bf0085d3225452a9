"""Which z-pass kernel each value of the tuning key zconv_engine runs (0 one warp per column, 1 one
exchange per transform at the FP32 length 512 and as 0 elsewhere, 2 and unset the rows ky and
Ny - ky paired), told by the code that its bounded wait reports when it runs out (as in
test_gpu_wait_timeout); the context is usable afterwards and the fields match the oracle."""
import pytest

import openspacecharge_b200 as osc
from openspacecharge_b200 import native
from conftest import field_err
from test_gpu_freespace import TOL
from test_gpu_wait_timeout import _rho

pytestmark = pytest.mark.gpu
RADIX, PAIRED, EXCHANGE = 1, 2, 3


@pytest.mark.parametrize("engine", [None, 0, 1, 2])
@pytest.mark.parametrize("prec,n", [(osc.PREC_FP32, (9, 8, 16)), (osc.PREC_FP32, (16, 16, 64)), (osc.PREC_FP64, (16, 16, 64)),
                                    (osc.PREC_FP32, (8, 9, 96)), (osc.PREC_FP64, (8, 9, 192)),
                                    (osc.PREC_FP32, (12, 12, 256)), (osc.PREC_FP64, (12, 12, 256))])
def test_engine_values(oracle, prec, n, engine):
    rho, delta = _rho(oracle, n)
    key = f"zconv_engine:{'f32' if prec == osc.PREC_FP32 else 'f64'}:L{2 * n[2]}"
    want = {None: PAIRED, 2: PAIRED, 0: RADIX}.get(engine, EXCHANGE if key.endswith("f32:L512") else RADIX)
    e_ref, _ = oracle.freespace_solver2(rho, 2.5, delta)
    with osc.Context(0) as ctx:
        if engine is not None:
            ctx.set_tuning(key, engine)
        assert ctx.get_tuning(key) == (2 if engine is None else engine)
        ctx.set_option(native.OPT_TEST_WAIT_TIMEOUT, 1)
        with pytest.raises(osc.OscError) as ei:
            osc.osc_freespace_solver2(ctx, rho, 2.5, delta, precision=prec)
        assert ei.value.code == native.OSC_E_TIMEOUT and f"fault code {want})" in str(ei.value)
        ctx.set_option(native.OPT_TEST_WAIT_TIMEOUT, 0)
        e, _ = osc.osc_freespace_solver2(ctx, rho, 2.5, delta, precision=prec)
        mx, rm = field_err(e, e_ref)
        assert mx <= TOL[prec], (mx, rm)
