"""osc_slab_interp_dev queued right behind the kernels that write its coordinates (the gather is the
only kernel of that call, so nothing of the library lies between): the fields equal those gathered
with the device idle, bit by bit, for one block, several and more than start early."""
import ctypes

import numpy as np
import pytest

import openspacecharge_b200 as osc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npart", [1, 255, 256, 100_001, 700_000])
def test_gather_reads_coordinates_just_written(npart):
    torch = pytest.importorskip("torch")
    n = (9, 8, 16)
    d = np.full(3, 1e-3)
    m = osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=np.zeros(3), max=d * (np.array(n) - 1), delta=d, gamma=2.0).to_c()
    g = torch.Generator(device="cuda").manual_seed(npart)
    top = torch.tensor(d * (np.array(n) - 1.001), device="cuda")
    sets = [torch.rand((3, npart), generator=g, dtype=torch.float64, device="cuda") * top[:, None] for _ in range(3)]
    e8 = torch.rand((n[0] * n[1] * n[2], 8), generator=g, dtype=torch.float32, device="cuda")
    p = torch.zeros((3, npart), dtype=torch.float64, device="cuda")
    out = [torch.zeros((npart, 3), dtype=torch.float64, device="cuda") for _ in range(12)]
    with osc.Context(0) as ctx:
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)

        def gather(E):
            ctx.call("osc_slab_interp_dev", ctypes.byref(m), 0, n[2], npart, p[0].data_ptr(), p[1].data_ptr(),
                     p[2].data_ptr(), e8.data_ptr(), E.data_ptr())

        want = []
        for s in sets:
            p.copy_(s)
            torch.cuda.synchronize()
            E = torch.zeros((npart, 3), dtype=torch.float64, device="cuda")
            gather(E)
            torch.cuda.synchronize()
            want.append(E)
        for i, E in enumerate(out):
            p.copy_(sets[i % 3])
            gather(E)
        torch.cuda.synchronize()
        for i, E in enumerate(out):
            assert torch.equal(E, want[i % 3])
