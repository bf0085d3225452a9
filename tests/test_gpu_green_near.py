"""FP64 cell integrals around the distance where the Green build changes from corner differences of
the primitives to the series: the field of one charged node of cubic cells at the nodes 8 and 9
cells along the axes (where tiles of cells begin), against the primitives in extended precision.
The bound is what corner differences lose in FP64 at that distance: the largest error of the same
differences evaluated by numpy in FP64 at the nodes 7.8 to 9.5 cells away, plus the transforms'
round-off, 1e-15 of the largest field of the grid."""
import numpy as np
import pytest

import openspacecharge_b200 as osc
from test_gpu_green_cells import FPEI, LD

pytestmark = pytest.mark.gpu


def xprim(x, y, z):
    # log((r - z)/(r + z))/2 without the cancellation of r - |z|, as the kernel has it
    r = np.sqrt(x * x + y * y + z * z)
    q = r + np.abs(z)
    return x * np.arctan((y * z) / (r * x)) - z * np.log(r + y) - y * np.sign(z) * np.log(q * q / (x * x + y * y)) / 2


def corner_field(n, h, T):
    u, v, w = [(np.arange(0, m + 1).astype(T) - T(0.5)) * T(h) for m in n]
    u, v, w = u[:, None, None], v[None, :, None], w[None, None, :]
    out = []
    for f in (xprim(u, v, w), xprim(v, w, u), xprim(w, u, v)):
        g = f / (T(h) * T(h) * T(h))
        for axis in range(3):
            g = np.diff(g, axis=axis)
        out.append(T(FPEI) * g)
    return np.stack(out, -1)


@pytest.mark.parametrize("h", [3e-3, 1.0])
@pytest.mark.parametrize("n", [(12, 12, 12), (16, 10, 12), (10, 16, 16)])
def test_no_worse_than_corner_differences(ctx, n, h):
    ref = corner_field(n, h, LD)
    mag = np.sqrt((ref.astype(np.float64) ** 2).sum(-1))
    r = np.sqrt(sum(np.arange(m).reshape([-1 if a == d else 1 for a in range(3)]) ** 2.0 for d, m in enumerate(n)))
    shell = (r >= 7.8) & (r <= 9.5)
    plain = np.abs(corner_field(n, h, np.float64).astype(LD) - ref).max(-1).astype(np.float64)
    rel = (plain[shell] / mag[shell]).max()
    rho = np.zeros(n, order="F")
    rho[0, 0, 0] = 1.0
    e, _ = osc.osc_freespace_solver2(ctx, rho, 1.0, (h, h, h), precision=osc.PREC_FP64)
    err = np.abs(e.astype(LD) - ref).max(-1).astype(np.float64)
    for node in [(a, 0, 0) for a in (8, 9)] + [(0, a, 0) for a in (8, 9)] + [(0, 0, a) for a in (8, 9)]:
        assert err[node] <= rel * mag[node] + 1e-15 * mag.max(), (node, err[node] / mag[node], rel)
