"""The work that users of this framework have it do, as timed cases.

Every case is a call on device-resident particles (float64 CUDA tensors) through the package's
public functions: the fused space-charge step (`space_charge_step_dev`) in its precisions,
mesh and particle-order options, the batched step, the rectangular-pipe step and the
differentiable step.  `exact` restates each of them in plain 64-bit torch.
"""
import math

import numpy as np
import torch

import openspacecharge_b200 as osc
from openspacecharge_b200.autograd import space_charge_field

MC2 = 0.510998910e6
GAMMA = 5e6 / MC2
QTOT = 1e-9
C_F32 = float(np.float32(299792458.0))
FPEI = float(np.float32(299792458.0) * np.float32(299792458.0)) * 1.00000000055e-7
FPEI_PIPE = float(np.float32(299792458.0) * np.float32(299792458.0) * np.float32(1.0e-7))


def listed():
    step = {"kind": "step", "prec": "fp32", "refit": False, "cathode": False, "bfield": False, "charges": "total",
            "order": "any", "shape": "gauss"}
    return [
        # the smallest step: a few thousand macro-particles on a coarse fixed mesh, as in a
        # design loop that calls it per element; launches and host work are what it costs
        dict(step, name="step-16", nx=16, ny=16, nz=16, np=2000),
        # a small step with the reference's default resize_mesh: the mesh follows the bunch,
        # so the Green function is rebuilt on every call
        dict(step, name="step-32-refit", nx=32, ny=32, nz=48, np=100_000, refit=True),
        # the grid and particle count of the reference's example notebook, mesh kept
        dict(step, name="step-64", nx=64, ny=64, nz=128, np=1_000_000),
        # a ragged grid (doubled lengths 90, 72, 100), a charge on every particle, mesh refit
        dict(step, name="step-odd-refit", nx=45, ny=36, nz=50, np=333_333, refit=True, charges="each"),
        # the headline step of the benchmark
        dict(step, name="step-128x256", nx=128, ny=128, nz=256, np=10_000_000),
        # the same with the mesh refit, and so the Green function rebuilt, on every call
        dict(step, name="step-128x256-refit", nx=128, ny=128, nz=256, np=10_000_000, refit=True),
        # tracking with particles kept in cell order
        dict(step, name="step-128x256-cell", nx=128, ny=128, nz=256, np=10_000_000, order="cell"),
        # emission from a cathode: image charges, B wanted, mesh following the bunch; grid and
        # distribution of the notebook's cathode run
        dict(step, name="cathode-64-refit", nx=64, ny=64, nz=64, np=2_000_000, refit=True, cathode=True,
             bfield=True, shape="ball"),
        # double precision with E and B, as a user checks the single-precision step or runs a
        # study that needs it
        dict(step, name="step-128-fp64", nx=128, ny=128, nz=128, np=4_000_000, prec="fp64", bfield=True),
        # many bunches per call, mesh refit, mixed grids (the benchmark's batch)
        {"name": "batch-256", "kind": "batch", "bunches": 256, "np_min": 10_000, "np_max": 1_000_000,
         "edges": "32,48,64,96", "plan": 1},
        # a differentiable step in an optimisation: forward and backward
        {"name": "adjoint-128", "kind": "adjoint", "nx": 128, "ny": 128, "nz": 128, "np": 4_000_000,
         "prec": "fp32"},
        # a bunch off axis in a rectangular pipe
        {"name": "pipe-64", "kind": "pipe", "nx": 64, "ny": 64, "nz": 128, "np": 4_000_000, "prec": "fp32"},
    ]


# node counts whose doubled lengths are 2^a 3^b 5^c, the lengths the transforms take
SMOOTH = [n for n in range(12, 257) if not any((2 * n) % p == 0 for p in range(7, 2 * n + 1)
                                               if all(p % q for q in range(2, int(p ** 0.5) + 1)))]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, most_xy, most_z, most_nodes):
    while True:
        pick = [min(SMOOTH, key=lambda n, v=math.exp(rng.uniform(math.log(12), math.log(m))): abs(n - v))
                for m in (most_xy, most_xy, most_z)]
        if pick[0] * pick[1] * pick[2] <= most_nodes:
            return {"nx": pick[0], "ny": pick[1], "nz": pick[2]}


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["batch", "adjoint", "pipe"])
    if kind == "batch":
        return {"kind": "batch", "bunches": _log_int(rng, 2, 200), "np_min": 10_000,
                "np_max": _log_int(rng, 100_000, 1_000_000), "edges": "32,48,64,96", "plan": rng.randrange(1, 10 ** 6)}
    if kind in ("adjoint", "pipe"):
        return dict({"kind": kind, "np": _log_int(rng, 20_000, 4_000_000), "prec": "fp32"},
                    **_grid(rng, 128, 128, 1 << 21))
    cathode = rng.random() < 0.25
    prec = "fp64" if rng.random() < 0.2 else "fp32"
    small = cathode or prec == "fp64"
    g = _grid(rng, 96 if small else 128, 128 if small else 256, 600_000 if small else 1 << 22)
    return dict({"kind": "step", "prec": prec, "refit": rng.random() < 0.5, "cathode": cathode,
                 "bfield": rng.random() < 0.3, "charges": rng.choice(["total", "total", "each"]),
                 "order": "cell" if prec == "fp32" and rng.random() < 0.2 else "any",
                 "shape": "ball" if cathode else "gauss", "np": _log_int(rng, 2000, 10_000_000)}, **g)


# ---- inputs -----------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _bunch(n, sigma, g, shape="gauss", centroid=(0.0, 0.0, 0.0)):
    """n particles (3, n): Gaussian cut at 4 sigma or uniform in the unit ball, scaled and centred."""
    if shape == "gauss":
        r = torch.randn((3, n + n // 100 + 1000), dtype=torch.float64, device="cuda", generator=g)
        r = r[:, (r * r).sum(0) <= 16.0][:, :n]
    else:
        r = torch.rand((3, 2 * n + n // 5 + 1000), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        r = r[:, (r * r).sum(0) <= 1.0][:, :n]
    r = r * torch.tensor(sigma, dtype=torch.float64, device="cuda")[:, None]
    return r - r.mean(1, keepdim=True) + torch.tensor(centroid, dtype=torch.float64, device="cuda")[:, None]


def _fixed_mesh(n, lo, hi):
    """Mesh of get_mesh_quantities: one spare cell around the bunch."""
    eps = 1e-13
    hi = [v * (1.0 + math.copysign(1.0, v) * eps) for v in hi]
    lo = [v * (1.0 - math.copysign(1.0, v) * eps) for v in lo]
    delta = np.array([(hi[d] - lo[d]) / (n[d] - 3) for d in range(3)])
    umin = np.array(lo) - delta
    return umin, umin + (np.array(n) - 1) * delta, delta


def _plan(case):
    """Grids, particle counts, sizes and charges of a batch."""
    rng = np.random.default_rng(case["plan"])
    edges = [int(v) for v in case["edges"].split(",")]
    grids, counts, sigmas, charges = [], [], [], []
    for _ in range(case["bunches"]):
        grids.append(tuple(int(rng.choice(edges)) for _ in range(3)))
        counts.append(int(np.exp(rng.uniform(np.log(case["np_min"]), np.log(case["np_max"])))))
        sigmas.append(tuple(float(v) for v in rng.uniform(0.2e-3, 2e-3, 3)))
        charges.append(float(rng.uniform(0.1e-9, 2e-9)))
    return grids, counts, sigmas, charges


PIPE_AB = (20e-3, 10e-3)
PIPE_SIGMA = (2e-3, 1e-3, 1e-3)


def _inputs(case, seed):
    """Particles, charges and mesh of a case, from the seed alone."""
    g = _gen(seed)
    if case["kind"] == "batch":
        grids, counts, sigmas, charges = _plan(case)
        r = torch.cat([_bunch(n, s, g) for n, s in zip(counts, sigmas)], 1)
        return {"grids": grids, "counts": counts, "total": charges, "r": [v.contiguous() for v in r]}
    n = (case["nx"], case["ny"], case["nz"])
    npart = case["np"]
    out = {"n": n, "gamma": GAMMA, "total": QTOT, "q": None}
    if case["kind"] == "pipe":
        a, b = PIPE_AB
        r = torch.randn((3, npart + npart // 10 + 2000), dtype=torch.float64, device="cuda", generator=g)
        s = PIPE_SIGMA
        keep = ((r * r).sum(0) <= 16.0) & ((r[0] * s[0] / (0.5 * a)) ** 2 + (r[1] * s[1] / (0.5 * b)) ** 2 <= 0.81)
        r = r[:, keep][:, :npart] * torch.tensor(s, dtype=torch.float64, device="cuda")[:, None]
        r = r - r.mean(1, keepdim=True) + torch.tensor([3e-3, -1e-3, 0.0], dtype=torch.float64, device="cuda")[:, None]
        umin = np.array([-0.5 * a, -0.5 * b, -6 * s[2]])
        delta = np.array([a / (n[0] - 1), b / (n[1] - 1), 12 * s[2] / (n[2] - 1)])
        out.update(r=[v.contiguous() for v in r], min=umin, max=umin + (np.array(n) - 1) * delta, delta=delta)
        return out
    if case["kind"] == "adjoint":
        r = _bunch(npart, (1e-3, 1e-3, 1e-3), g)
        out["gE"] = torch.randn((npart, 3), dtype=torch.float64, device="cuda", generator=g)
        q = QTOT / npart * (0.5 + torch.rand(npart, dtype=torch.float64, device="cuda", generator=g))
    else:
        if case["cathode"]:
            r = _bunch(npart, (1e-3, 1e-3, 1e-3), g, case["shape"], (0.0, 0.0, 1.1e-3))
            out["gamma"] = 1e6 / MC2
        else:
            r = _bunch(npart, (0.5e-3, 0.5e-3, 2e-3), g, case["shape"])
        q = None
        if case["charges"] == "each":
            q = QTOT / npart * (0.5 + torch.rand(npart, dtype=torch.float64, device="cuda", generator=g))
    umin, umax, delta = _fixed_mesh(n, r.amin(1).tolist(), r.amax(1).tolist())
    if case.get("order") == "cell":
        # the order that sort_particles_dev gives, ties in the order of the input
        (i, j, k), _ = _cells(r, n, *(_refit(r, n)[::2] if case["refit"] else (umin, delta)))
        at = torch.sort(i + n[0] * (j + n[1] * k), stable=True).indices
        r, q = r[:, at], None if q is None else q[at]
    out.update(r=[v.contiguous() for v in r], q=q, min=umin, max=umax, delta=delta)
    return out


def _mesh(n, gamma, inp=None):
    if inp is None:
        return osc.Mesh3D(nlo=(1, 1, 1), nhi=n, gamma=gamma)
    return osc.Mesh3D(nlo=(1, 1, 1), nhi=n, min=inp["min"], max=inp["max"], delta=inp["delta"], gamma=gamma)


PREC = {"fp32": osc.PREC_FP32, "fp64": osc.PREC_FP64}


def prepare(case, seed):
    inp = _inputs(case, seed)
    ctx = osc.Context(torch.cuda.current_device())
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    s = {"case": case, "ctx": ctx, "inp": inp}
    npart = inp["r"][0].numel()
    if case["kind"] != "adjoint":
        s["E"] = torch.empty((npart, 3), dtype=torch.float64, device="cuda")
    if case["kind"] == "batch":
        s["meshes"] = [_mesh(n, GAMMA) for n in inp["grids"]]
        return s
    s["mesh"] = _mesh(inp["n"], inp["gamma"], inp)
    if case["kind"] == "pipe":
        osc.osc_rectpipe_green(ctx, s["mesh"], *PIPE_AB, precision=PREC[case["prec"]])
    elif case["kind"] == "adjoint":
        s["leaves"] = [t.requires_grad_() for t in (*inp["r"], inp["q"])]
    else:
        if case["refit"]:
            # between the calls of a program that refits, the particles move and no two
            # meshes are equal: a kept Green function would never be met again
            ctx.set_option(osc.OPT_GREEN_CACHE_MB, 0)
        if case["order"] == "cell":
            ctx.set_option(osc.OPT_PARTICLE_ORDER, osc.ORDER_CELL_SORTED)
        s["B"] = torch.empty_like(s["E"]) if case["bfield"] else None
    return s


def run(s):
    case, ctx, inp = s["case"], s["ctx"], s["inp"]
    kind = case["kind"]
    if kind == "batch":
        outside = osc.batch_space_charge_step_dev(ctx, s["meshes"], *inp["r"], inp["counts"], s["E"],
                                                  total_charges=inp["total"], resize_mesh=True)
        return {"E": s["E"], "outside": np.array(outside), "delta": np.stack([m.delta for m in s["meshes"]])}
    if kind == "pipe":
        osc.space_charge_step_rectpipe_dev(ctx, s["mesh"], *inp["r"], s["E"], *PIPE_AB, total_charge=inp["total"],
                                           precision=PREC[case["prec"]])
        return {"E": s["E"]}
    if kind == "adjoint":
        E = space_charge_field(*s["leaves"], s["mesh"], ctx, precision=PREC[case["prec"]])
        gx, gy, gz, gq = torch.autograd.grad(E, s["leaves"], inp["gE"])
        return {"E": E.detach(), "gx": gx, "gy": gy, "gz": gz, "gq": gq}
    mesh = s["mesh"]
    osc.space_charge_step_dev(ctx, mesh, *inp["r"], s["E"], qa=inp["q"],
                              total_charge=None if inp["q"] is not None else inp["total"],
                              resize_mesh=case["refit"], at_cathode=case["cathode"], precision=PREC[case["prec"]],
                              B=s["B"])
    out = {"E": s["E"], "min": mesh.min, "delta": mesh.delta}
    if s["B"] is not None:
        out["B"] = s["B"]
    return out


# ---- compulsory work ----------------------------------------------------------------------
def _solve_work(n, comps, rebuild, image, width):
    """Flops of the doubled-grid convolution (one real forward and `comps` real inverse
    transforms, and the Green function's where it is rebuilt) and the stored spectra's bytes."""
    m = 8 * n[0] * n[1] * n[2]
    oct_ = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    fft = 2.5 * m * math.log2(m)
    flops = (1 + comps) * fft + 6 * comps * m / 2
    spectra = width * comps * oct_ * (3 if image else 1)
    if rebuild:
        flops += comps * (60 * oct_ + fft / 8) * (3 if image else 1)
        spectra = 0
    return flops, spectra


def work(case):
    if case["kind"] == "batch":
        grids, counts, _, _ = _plan(case)
        flops = sum(_solve_work(n, 3, True, False, 4)[0] for n in grids) + 150 * sum(counts)
        return {"bytes": 48 * sum(counts), "flops": flops}
    n, npart = (case["nx"], case["ny"], case["nz"]), case["np"]
    width = 8 if case["prec"] == "fp64" else 4
    if case["kind"] == "pipe":
        flops, _ = _solve_work(n, 1, False, False, 4)
        return {"bytes": 48 * npart + 8 * (n[0] + 1) * 4 * n[1] * n[2], "flops": flops + 150 * npart}
    if case["kind"] == "adjoint":
        f, b = _solve_work(n, 3, False, False, 4)
        # x, y, z, q, dL/dE in; E and four gradients out; the adjoint convolution transforms
        # three grids and returns one
        return {"bytes": (32 + 24 + 24 + 32) * npart + b, "flops": 2 * f + 450 * npart}
    comps = 3
    flops, spectra = _solve_work(n, comps, case["refit"], case["cathode"], width)
    per = 48 + (8 if case["charges"] == "each" else 0) + (24 if case["bfield"] else 0)
    return {"bytes": per * npart + spectra, "flops": flops + (150 + 60 * case["bfield"]) * npart}


# ---- the same in plain 64-bit torch ---------------------------------------------------------
def _cells(r, n, lo, delta):
    """Lowest corner and low-node weight of each particle's cell, per axis."""
    idx, w = [], []
    for d in range(3):
        f = torch.floor((r[d].detach() - lo[d]) * (1.0 / delta[d]) + 1.0).clamp(1, n[d] - 1)
        idx.append(f.long() - 1)
        w.append(((lo[d] - r[d]) + f * delta[d]) * (1.0 / delta[d]))
    return idx, w


def _corners(cells, n):
    """The eight (node, weight) pairs of every particle."""
    (i, j, k), (a, b, c) = cells
    base = i + n[0] * (j + n[1] * k)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                wt = (a if not dx else 1 - a) * (b if not dy else 1 - b) * (c if not dz else 1 - c)
                yield base + dx + n[0] * (dy + n[1] * dz), wt


def _deposit(cells, n, q):
    rho = torch.zeros(n[0] * n[1] * n[2], dtype=torch.float64, device="cuda")
    for node, wt in _corners(cells, n):
        rho = rho.index_add(0, node, wt * q)
    return rho.view(n[2], n[1], n[0])


def _gather(cells, n, F):
    out = []
    for c in range(3):
        flat, v = F[c].reshape(-1), 0
        for node, wt in _corners(cells, n):
            v = v + flat[node] * wt
        out.append(v)
    return torch.stack(out, 1)


def _primitive(x, y, z):
    r = torch.sqrt(x * x + y * y + z * z)
    return x * torch.atan((y * z) / (r * x)) - z * torch.log(r + y) + y * torch.log((r - z) / (r + z)) / 2


def _green(n, delta, gamma, zoff, comp):
    """Integrated Green function of E component `comp` at the displacements -n .. n-1 of each
    axis, rolled so that displacement 0 comes first; transformed."""
    h = (delta[0], delta[1], delta[2] * gamma)
    off = (0.0, 0.0, zoff * gamma)
    u, v, w = [(torch.arange(-n[d], n[d] + 1, dtype=torch.float64, device="cuda") - 0.5) * h[d] + off[d]
               for d in range(3)]
    u, v, w = u[None, None, :], v[None, :, None], w[:, None, None]
    F = _primitive(*((u, v, w), (v, w, u), (w, u, v))[comp])
    F = F * ((gamma if comp < 2 else 1.0) / (h[0] * h[1] * h[2]))
    for axis in range(3):
        F = torch.diff(F, dim=axis)
    return torch.fft.rfftn(torch.roll(F, (-n[2], -n[1], -n[0]), (0, 1, 2)))


def _solve(rho, n, delta, gamma, image=None):
    """E on the grid; with `image` (the z offset of the image charges) E of the charges and of
    their images apart."""
    full = (2 * n[2], 2 * n[1], 2 * n[0])
    hat = torch.fft.rfftn(rho, full)
    direct = [FPEI * torch.fft.irfftn(hat * _green(n, delta, gamma, 0.0, c), full)[:n[2], :n[1], :n[0]]
              for c in range(3)]
    if image is None:
        return direct, None
    hat = torch.fft.rfftn(-torch.flip(rho, (0,)), full)
    return direct, [FPEI * torch.fft.irfftn(hat * _green(n, delta, gamma, image, c), full)[:n[2], :n[1], :n[0]]
                    for c in range(3)]


def _refit(r, n):
    lo, hi = np.array([float(v.min()) for v in r]), np.array([float(v.max()) for v in r])
    d = (hi - lo) / (np.array(n) - 1)
    lo, hi = lo - 1.0e-6 * d, hi + 1.0e-6 * d
    return lo, hi, (hi - lo) / (np.array(n) - 1)


def _pipe_term(n, lo, delta, gamma, sx, sy):
    """One of the pipe's four kernels, sum over 5 x 5 modes, at displacements from low to high."""
    a, b = PIPE_AB
    hz = delta[2]
    disp = [torch.arange(2 * n[d], dtype=torch.float64, device="cuda") for d in range(3)]
    disp = [torch.where(t < n[d], t, t - 2 * n[d]) for d, t in enumerate(disp)]
    u = disp[0] * delta[0] if sx > 0 else 2 * lo[0] + torch.arange(2 * n[0], dtype=torch.float64, device="cuda") * delta[0]
    v = disp[1] * delta[1] if sy > 0 else 2 * lo[1] + torch.arange(2 * n[1], dtype=torch.float64, device="cuda") * delta[1]
    w = disp[2] * hz
    G = 0
    for m in range(1, 6):
        for k in range(1, 6):
            kap = math.sqrt((m * math.pi / a) ** 2 + (k * math.pi / b) ** 2)
            zf = (torch.exp(-kap * (gamma * w - hz).abs()) - 2 * torch.exp(-kap * (gamma * w).abs()) +
                  torch.exp(-kap * (gamma * w + hz).abs())) / (hz * hz * kap * kap)
            zf = torch.where(w == 0, zf + 2.0 / (hz * kap), zf)
            G = G + (sx ** m * sy ** k / kap) * zf[:, None, None] * torch.cos(k * v * math.pi / b)[None, :, None] * \
                torch.cos(m * u * math.pi / a)[None, None, :]
    return G * (2 * math.pi / (a * b))


def _pipe_field(rho, n, lo, delta, gamma):
    full = (2 * n[2], 2 * n[1], 2 * n[0])
    phi = 0
    for sx, sy in ((1, 1), (1, -1), (-1, 1), (-1, -1)):
        # the terms with a minus sign correlate along that axis: a convolution with the
        # charge mirrored, whose result starts at the far end of the full correlation
        G = _pipe_term(n, lo, delta, gamma, sx, sy)
        src = torch.zeros(full, dtype=torch.float64, device="cuda")
        src[:n[2], :n[1], :n[0]] = rho
        for sign, axis in ((sx, 2), (sy, 1)):
            if sign < 0:  # index -i of the periodic array
                src = torch.roll(torch.flip(src, (axis,)), 1, axis)
        term = torch.fft.irfftn(torch.fft.rfftn(src) * torch.fft.rfftn(G), full)
        phi = phi + sx * sy * term[:n[2], :n[1], :n[0]]
    phi = FPEI_PIPE * phi
    E = []
    for axis, h, f in ((2, delta[0], gamma), (1, delta[1], gamma), (0, delta[2], 1.0 / gamma)):
        m = phi.shape[axis]
        i = torch.arange(m, device="cuda")
        lo_i, hi_i = (i - 1).clamp(min=0), (i + 1).clamp(max=m - 1)
        shape = [1, 1, 1]
        shape[axis] = m
        span = ((hi_i - lo_i) * h).view(shape)
        E.append(-(phi.index_select(axis, hi_i) - phi.index_select(axis, lo_i)) / span * f)
    return E


def exact(case, seed):
    inp = _inputs(case, seed)
    if case["kind"] == "batch":
        E, deltas, at = [], [], 0
        for n, npart, q in zip(inp["grids"], inp["counts"], inp["total"]):
            r = [v[at:at + npart] for v in inp["r"]]
            at += npart
            lo, _, delta = _refit(r, n)
            cells = _cells(r, n, lo, delta)
            E.append(_gather(cells, n, _solve(_deposit(cells, n, q / npart), n, delta, GAMMA)[0]))
            deltas.append(delta)
        return {"E": torch.cat(E), "outside": None, "delta": np.stack(deltas)}
    n, npart = inp["n"], case["np"]
    if case["kind"] == "pipe":
        cells = _cells(inp["r"], n, inp["min"], inp["delta"])
        rho = _deposit(cells, n, inp["total"] / npart)
        return {"E": _gather(cells, n, _pipe_field(rho, n, inp["min"], inp["delta"], inp["gamma"]))}
    if case["kind"] == "adjoint":
        leaves = [t.requires_grad_() for t in (*inp["r"], inp["q"])]
        cells = _cells(leaves[:3], n, inp["min"], inp["delta"])
        rho = _deposit(cells, n, leaves[3])
        E = _gather(cells, n, _solve(rho, n, inp["delta"], inp["gamma"])[0])
        gx, gy, gz, gq = torch.autograd.grad(E, leaves, inp["gE"])
        return {"E": E.detach(), "gx": gx, "gy": gy, "gz": gz, "gq": gq}
    lo, hi, delta = (inp["min"], inp["max"], inp["delta"]) if not case["refit"] else _refit(inp["r"], n)
    cells = _cells(inp["r"], n, lo, delta)
    q = inp["q"] if inp["q"] is not None else inp["total"] / npart
    rho = _deposit(cells, n, q)
    direct, image = _solve(rho, n, delta, inp["gamma"], 2 * lo[2] + (hi[2] - lo[2]) if case["cathode"] else None)
    E = direct if image is None else [a + b for a, b in zip(direct, image)]
    out = {"E": _gather(cells, n, E), "min": lo, "delta": delta}
    if case["bfield"]:
        # image charges move the other way
        src = direct if image is None else [a - b for a, b in zip(direct, image)]
        beta = math.sqrt(1 - 1 / inp["gamma"] ** 2)
        out["B"] = _gather(cells, n, [-(beta / C_F32) * src[1], (beta / C_F32) * src[0], torch.zeros_like(src[2])])
    return out
