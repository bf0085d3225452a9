"""The z pass with rows ky and Ny - ky paired, the default at every length of the warp engine,
against the solve in extended precision (the FP64 oracle's corner differences lose up to 5e-10
here) and against the unpaired engine (tuning value 1; at the doubled length 512 in FP32 that is the
one-exchange engine): odd and even row and column counts, the smallest and largest lengths.
Tolerances as in the other engine comparisons: FP64 1e-10 to the reference and 1e-13 to each
other, FP32 1e-5 and 2e-6, of the largest component."""
import numpy as np
import pytest

import openspacecharge_b200 as osc
from conftest import field_err
from test_gpu_green_cells import reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxy", [(2, 3), (9, 8), (16, 15)])
@pytest.mark.parametrize("nz", [16, 32, 48, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("prec", [osc.PREC_FP64, osc.PREC_FP32])
def test_default_pairs_match_reference_and_unpaired(ctx, nz, nxy, prec):
    n = nxy + (nz,)
    rho = np.asfortranarray(np.random.default_rng(nz).uniform(0.0, 1e-12, n))
    delta, gamma = np.array([1e-4, 1.3e-4, 2e-4]), 2.5
    e_ref, _ = reference(rho, gamma, delta)
    tag, tol, tol2 = ("f32", 1e-5, 2e-6) if prec == osc.PREC_FP32 else ("f64", 1e-10, 1e-13)
    e0, _ = osc.osc_freespace_solver2(ctx, rho, gamma, delta, precision=prec)
    ctx.set_tuning(f"zconv_engine:{tag}:L{2 * nz}", 1)
    try:
        e1, _ = osc.osc_freespace_solver2(ctx, rho, gamma, delta, precision=prec)
    finally:
        ctx.set_tuning(f"zconv_engine:{tag}:L{2 * nz}", 0)
    assert field_err(e0, e_ref)[0] <= tol
    assert field_err(e0, e1)[0] <= tol2
