"""A step whose refit is refused leaves the whole mesh as it was, the charge included, and the
refusal names non-finite coordinates of any kind on any axis (the extremes are compared as FP64
values, where NaN orders with nothing)."""
import ctypes

import numpy as np
import pytest

import openspacecharge_b200 as osc
from openspacecharge_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_q", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_refused_step_leaves_the_mesh(ctx, axis, value, use_q):
    torch = pytest.importorskip("torch")
    p = np.random.default_rng(7).uniform(-1, 1, (3, 70001))
    p[axis, 300] = value
    x, y, z = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in p)
    q = torch.full_like(x, 1e-13)
    E = torch.empty((len(x), 3), dtype=torch.float64, device="cuda")
    c = osc.Mesh3D(nlo=(1, 1, 1), nhi=(8, 8, 8), min=np.full(3, -2.0), max=np.full(3, 2.0), delta=np.full(3, 4 / 7),
                   gamma=2.0, charge=3.0).to_c()
    before = bytes(c)
    total = ctypes.byref(ctypes.c_double(5e-9))
    with pytest.raises(osc.OscError) as ei:
        ctx.call("osc_space_charge_step_dev", ctypes.byref(c), x.numel(), x.data_ptr(), y.data_ptr(), z.data_ptr(),
                 q.data_ptr() if use_q else None, None if use_q else total, 1, 0, osc.PREC_FP32, E.data_ptr(), None)
    assert ei.value.code == native.OSC_E_NAN and bytes(c) == before


# one wave of blocks, each thread four particles a trip: the sizes where a second particle, a second
# trip and a partial one begin, the extremes at the first and the last particle
@pytest.mark.parametrize("npart", [148 * 5 * 256, 148 * 5 * 256 + 1, 4 * 148 * 5 * 256, 4 * 148 * 5 * 256 + 1])
def test_box_at_the_edges_of_a_trip(ctx, npart):
    torch = pytest.importorskip("torch")
    p = np.random.default_rng(npart).uniform(-1e-3, 1e-3, (3, npart))
    for v, s in zip(p, (1, -1, 1)):
        v[0], v[-1] = -s * 4e-3, s * 5e-3
    x, y, z = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in p)
    E = torch.empty((npart, 3), dtype=torch.float64, device="cuda")
    m = osc.Mesh3D(nlo=(1, 1, 1), nhi=(9, 12, 16), gamma=1.0)
    osc.space_charge_step_dev(ctx, m, x, y, z, E, total_charge=1e-9, resize_mesh=True)
    lo, hi = p.min(1), p.max(1)
    d = (hi - lo) / (np.array([9, 12, 16]) - 1)
    # refit pads by 1e-6 of a cell on both sides (code/open_spacecharge_mod.f90:176-189)
    assert np.all(np.abs(m.min - (lo - 1e-6 * d)) <= 1e-8 * d) and np.all(np.abs(m.max - (hi + 1e-6 * d)) <= 1e-8 * d)
