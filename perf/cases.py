"""The work that a program on this framework has it do, as cases that can be timed and checked.

A hex case is one structured mesh of the unit cube with shared nodes and jittered vertices, resident on
the GPU, and the calls that a solver makes on it: the convection and diffusion residuals of one step,
both in one call, an RK4 step, the entropy viscosity, the learned viscosity, the FP16 tensor-core mode
and the FP64 build.  A tet case is the linear-tetrahedron pair of residuals.

Fields are what a marginally resolved compressible flow looks like: a few Fourier modes of order 0.1 and
a fluctuation of a few per cent at the grid scale in density, velocity and pressure; the momentum is the
product rho u in the fields' own precision, as a solver stores it.  (On perfectly smooth fields the
diffusion's energy residual is a difference of nearly equal numbers, and its last digits say nothing.)
"""
import math
import types

import numpy as np
import torch

from minisod2d_gb300 import capi, fem, kernels, learn, timestep

GAMMA, RGAS, CP, PR = 1.4, 287.0, 1004.5, 0.71
CE, CMAX = 0.1, 0.5
NOISE = 0.05
HEX_OPS = ("step", "onecall", "rk4", "mode_fp16", "visc", "learned", "f64")


def _hex(name, op, porder, nx, ny, nz, jitter=0.05):
    return {"name": name, "op": op, "porder": porder, "nx": nx, "ny": ny, "nz": nz, "jitter": jitter}


def listed():
    return [
        # The smallest mesh of the repository's workloads: a test or a coarse start-up run, where launches count.
        _hex("step_p4_16", "step", 4, 16, 16, 16, 0.0),
        # The throughput workload: the two residual calls of a step, porder 4 on 64^3 hexes.
        _hex("step_p4_64", "step", 4, 64, 64, 64),
        # The largest workload, porder 5 on 96^3 hexes: 191 million element points.
        _hex("step_p5_96", "step", 5, 96, 96, 96),
        # High order, porder 7 on 32^3 hexes.
        _hex("step_p7_32", "step", 7, 32, 32, 32),
        # Low order on a mesh of odd dimensions (element counts that fill no group of elements evenly).
        _hex("step_p2_61x45x83", "step", 2, 61, 45, 83),
        # Both residuals in one call, as the time loop uses them, on a ragged mesh.
        _hex("onecall_p4_47x31x53", "onecall", 4, 47, 31, 53),
        # One classical RK4 step: four evaluations of both residuals and the stage updates.
        _hex("rk4_p4_48", "rk4", 4, 48, 48, 48),
        # The two drop-in calls with the FP16 hi + lo tensor-core contractions switched on.
        _hex("mode_fp16_p7_24", "mode_fp16", 7, 24, 24, 24),
        # Entropy viscosity, then the diffusion that consumes it.
        _hex("visc_p5_40x48x36", "visc", 5, 40, 48, 36),
        # The learned viscosity with the network shipped for this workload, shock-like fields.
        _hex("learned_p4_48", "learned", 4, 48, 48, 48, 0.0),
        # The FP64 build, which a user runs to judge an FP32 result.
        _hex("f64_p4_20", "f64", 4, 20, 20, 20),
        # Linear tetrahedra: the driver's disconnected mesh over the nodes of the throughput workload.
        {"name": "tet_4243648", "op": "tet", "nelem": 4243648, "shared": False},
    ]


# Element points of the largest drawn case per kind (each no dearer than porder 5 on 96^3 hexes).
_MOST_POINTS = {"step": 1.2e8, "onecall": 1.2e8, "rk4": 2.5e7, "mode_fp16": 3e7, "visc": 6e7, "learned": 3e7,
                "f64": 4e6}


def draw(rng):
    kind = rng.choice(("step",) * 6 + ("onecall", "rk4", "visc", "tet", "mode_fp16", "learned", "f64"))
    if kind == "tet":
        return {"op": "tet", "nelem": int(math.exp(rng.uniform(math.log(2e4), math.log(5e6)))),
                "shared": rng.random() < 0.5}
    if kind == "learned":
        p = 4
    elif kind == "mode_fp16":
        p = rng.choice((4, 5, 6, 7))
    else:
        p = rng.choice((1, 2, 3, 4, 4, 4, 4, 5, 5, 6, 7, 7, 8))
    points = math.exp(rng.uniform(math.log(1e5), math.log(_MOST_POINTS[kind])))
    side = (points / (p + 1) ** 3) ** (1.0 / 3.0)
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    dims = [max(2, int(side * f)) for f in (a, b, 1.0 / (a * b))]
    if kind == "learned":
        dims = [max(8, int(side))] * 3
    return {"op": kind, "porder": p, "nx": dims[0], "ny": dims[1], "nz": dims[2],
            "jitter": 0.0 if kind == "learned" else rng.choice((0.0, 0.05, 0.1))}


# ---------------------------------------------------------------------------------------------------
# Meshes and fields
# ---------------------------------------------------------------------------------------------------
def _gll(P):
    inner = np.polynomial.legendre.Legendre.basis(P).deriv().roots() if P > 1 else np.zeros(0)
    return np.concatenate([[-1.0], np.sort(np.real(inner)), [1.0]])


def _natural(sod, P):
    """1-based SOD 1-D index (the two ends, then the interior) -> natural index."""
    s = np.asarray(sod) - 1
    return np.where(s == 0, 0, np.where(s == 1, P, s - 1))


def _structured(case, tables, gen, dev):
    """connec (a * nelem + e, 1-based), coord (d * npoin + p) of the jittered structured mesh."""
    P, dims = case["porder"], (case["nx"], case["ny"], case["nz"])
    nodes = [d * P + 1 for d in dims]
    ix = [torch.arange(d, device=dev, dtype=torch.int64) for d in dims]
    base = (ix[2].view(-1, 1, 1) * P * nodes[1] + ix[1].view(1, -1, 1) * P) * nodes[0] + ix[0].view(1, 1, -1) * P
    nat = [torch.from_numpy(_natural(tables[k], P)).to(dev) for k in ("AtoI", "AtoJ", "AtoK")]
    off = ((nat[2] * nodes[1] + nat[1]) * nodes[0] + nat[0] + 1).to(torch.int32)
    connec = (off.view(-1, 1) + base.reshape(1, -1).to(torch.int32)).reshape(-1)
    # Vertices: a uniform grid, its interior ones moved by up to +-jitter of the element size per component.
    vert = [torch.arange(d + 1, device=dev, dtype=torch.float64) / d for d in dims]
    shape = (dims[2] + 1, dims[1] + 1, dims[0] + 1)
    coord = []
    for d in range(3):
        v = vert[d].view([-1 if 2 - k == d else 1 for k in range(3)]).expand(shape).clone()
        move = (2.0 * torch.rand(shape, generator=gen, device=dev, dtype=torch.float64) - 1.0) * case["jitter"] / dims[d]
        inside = [slice(None)] * 3
        inside[2 - d] = slice(1, -1)
        v[tuple(inside)] += move[tuple(inside)]
        for ax in range(3):  # linear along each axis in turn: trilinear within the element
            m = dims[2 - ax]
            at = torch.arange(m * P + 1, device=dev)
            e = torch.clamp(at // P, max=m - 1)
            s = torch.from_numpy(0.5 * (_gll(P) + 1.0)).to(dev)[at - e * P]
            s = s.view([-1 if k == ax else 1 for k in range(3)])
            v = torch.index_select(v, ax, e) * (1.0 - s) + torch.index_select(v, ax, e + 1) * s
        coord.append(v.reshape(-1).float())
    return connec, torch.cat(coord), nodes


def _fields(nodes, gen, dev, dtype):
    """Density, velocity, pressure and what follows from them at nodes[2] x nodes[1] x nodes[0] points."""
    f32 = torch.float32
    npoin = nodes[0] * nodes[1] * nodes[2]
    x = [torch.linspace(0, 2 * math.pi, n, device=dev, dtype=f32).view([-1 if 2 - k == d else 1 for k in range(3)])
         for d, n in enumerate(nodes)]

    def modes(amp, count=4):
        out = torch.zeros(nodes[::-1], device=dev, dtype=f32)
        k = torch.randint(-3, 4, (count, 3), generator=gen, device=dev).cpu().tolist()
        r = torch.rand(count, 2, generator=gen, device=dev).cpu().tolist()
        for (kx, ky, kz), (a, ph) in zip(k, r):
            out += amp * (a + 0.5) * torch.sin(kx * x[0] + ky * x[1] + kz * x[2] + 2 * math.pi * ph)
        return out.reshape(-1)

    def noise():
        return NOISE * torch.randn(npoin, generator=gen, device=dev, dtype=f32)

    rho = ((1.0 + 0.05 * modes(1.0)) * (1.0 + noise())).clamp_(0.3).to(dtype)
    pr = ((1.0 + 0.03 * modes(1.0)) * (1.0 + noise())).clamp_(0.3).to(dtype)
    u = torch.cat([(modes(0.1) + noise()) for _ in range(3)]).to(dtype)
    return _derived(rho, u, pr)


def _derived(rho, u, pr):
    n = rho.numel()
    q = (u.view(3, n) * rho).reshape(-1)
    E = pr / (GAMMA - 1.0) / rho + 0.5 * u.view(3, n).square().sum(0)
    Tem = pr / (rho * RGAS)
    mu = 1.8e-5 * (Tem * RGAS) ** 0.7
    return {"rho": rho, "u": u, "q": q, "pr": pr, "E": E, "Tem": Tem, "mu_fluid": mu}


def _shock_fields(coord, gen):
    """The shock-like recipe of the learned viscosity: a density front, uniform pressure."""
    n = coord.numel() // 3
    seed = int(torch.randint(0, 2 ** 31 - 1, (1,), generator=gen, device=coord.device).item())
    f = fem.fields_recipe(capi.MSOD_FIELDS_SHOCK, 8, seed, n, coord.cpu().numpy())
    return {k: torch.from_numpy(v).to(coord.device) for k, v in f.items()}


def _hex_state(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    P, op = case["porder"], case["op"]
    real = torch.float64 if op == "f64" else torch.float32
    t = fem.element_tables(P, np.float64 if op == "f64" else np.float32)
    n = (P + 1) ** 3
    connec, coord, nodes = _structured(case, t, gen, dev)
    s = types.SimpleNamespace(op=op, cfg=types.SimpleNamespace(porder=P, nnode=n, Cp=CP, Pr=PR))
    s.nelem, s.npoin, s.connec = case["nx"] * case["ny"] * case["nz"], nodes[0] * nodes[1] * nodes[2], connec

    def up(k):
        return torch.from_numpy(t[k]).to(dev)

    s.dlxigp_ip, s.invAtoIJK, s.AtoI, s.AtoJ, s.AtoK = (up(k) for k in ("dlxigp_ip", "invAtoIJK", "AtoI", "AtoJ", "AtoK"))
    s.He = torch.empty(9 * s.nelem * n, dtype=real, device=dev)
    s.gpvol = torch.empty(s.nelem * n, dtype=real, device=dev)
    kernels.elem_jacobian(P, s.nelem, s.npoin, connec, coord.to(real), up("dNgp"), up("wgp"), s.gpvol, s.He)
    f = _shock_fields(coord, gen) if op == "learned" else _fields(nodes, gen, dev, real)
    for k, v in f.items():
        setattr(s, k, v)
    if op != "learned":
        s.mu_e = 2e-4 * torch.rand(s.nelem * n, generator=gen, device=dev, dtype=real)
        s.mu_sgs = 1e-4 * torch.rand(s.nelem * n, generator=gen, device=dev, dtype=real)
        s.C = tuple(torch.empty(k * s.npoin, dtype=real, device=dev) for k in (1, 3, 1))
        s.D = tuple(torch.empty(k * s.npoin, dtype=real, device=dev) for k in (1, 3, 1))
    if op == "visc":
        s.nu, s.numax = torch.empty(s.nelem, device=dev), torch.empty(s.nelem, device=dev)
    if op == "learned":
        s.mlp = learn.Mlp()
        s.mlp.load(learn.shipped_weights("learned_48"))
        s.nu, s.flag = torch.empty(s.nelem, device=dev), torch.empty(s.nelem, dtype=torch.int32, device=dev)
    if op == "rk4":
        s.Ml = timestep.lumped_mass(s)
        s.ws = timestep.workspace(s)
        s.rhoE = s.rho * s.E
        # A tenth of the acoustic step on the GLL grid.
        s.dt = 0.1 / (2.0 * P * P * max(case["nx"], case["ny"], case["nz"]))
    s.geo = (s.nelem, s.npoin, s.connec, None, None, s.He, s.gpvol, s.dlxigp_ip, None, s.invAtoIJK, s.AtoI, s.AtoJ,
             s.AtoK)
    return s


def _kuhn(m, dev):
    """Six tetrahedra per cube of an m^3 grid, around its main diagonal."""
    g = torch.arange(m, device=dev)
    v = m + 1
    corner = (g.view(-1, 1, 1) * v * v + g.view(1, -1, 1) * v + g.view(1, 1, -1)).reshape(-1, 1)
    step = (1, v, v * v)
    rows = []
    for a, b, c in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        o = [0, step[a], step[a] + step[b], step[a] + step[b] + step[c]]
        if (a, b, c) in ((0, 2, 1), (1, 0, 2), (2, 1, 0)):  # keep the volume positive
            o[1], o[2] = o[2], o[1]
        rows.append(corner + torch.tensor(o, device=dev))
    con = torch.cat(rows)
    x = torch.arange(v, device=dev, dtype=torch.float32) / m
    coord = torch.cat([x.view([-1 if 2 - k == d else 1 for k in range(3)]).expand(v, v, v).reshape(-1) for d in range(3)])
    return con, coord, v ** 3


def _tet_state(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    t = fem.tet_element_tables(np.float32)
    if case["shared"]:
        m = max(2, round((case["nelem"] / 6) ** (1.0 / 3.0)))
        con, coord, npoin = _kuhn(m, dev)
        coord = coord + (torch.rand(coord.numel(), generator=gen, device=dev) - 0.5) * (0.1 / m)
        nelem = con.shape[0]
        connec = (con.t().contiguous() + 1).to(torch.int32).reshape(-1)
    else:
        nelem = case["nelem"]
        npoin = 4 * nelem
        connec = torch.arange(1, npoin + 1, device=dev, dtype=torch.int32).view(nelem, 4).t().contiguous().reshape(-1)
        coord = torch.from_numpy(fem.TET_BASE).to(dev).view(3, 1, 4).expand(3, nelem, 4).reshape(-1).contiguous()
    s = types.SimpleNamespace(op="tet", nelem=nelem, npoin=npoin, connec=connec)
    s.Ngp, s.dNgp = torch.from_numpy(t["Ngp"]).to(dev), torch.from_numpy(t["dNgp"]).to(dev)
    s.He, s.gpvol = torch.empty(36 * nelem, device=dev), torch.empty(4 * nelem, device=dev)
    kernels.tet_jacobian(nelem, npoin, connec, coord, s.dNgp, torch.from_numpy(t["wgp"]).to(dev), s.gpvol, s.He)
    side = max(2, round(npoin ** (1.0 / 3.0)))
    f = _fields([side, side, -(-npoin // (side * side))], gen, dev, torch.float32)
    full = f["rho"].numel()
    for k, v in f.items():
        setattr(s, k, v.view(-1, full)[:, :npoin].reshape(-1).contiguous())
    s.mu_e = 2e-4 * torch.rand(4 * nelem, generator=gen, device=dev)
    s.mu_sgs = 1e-4 * torch.rand(4 * nelem, generator=gen, device=dev)
    s.C = tuple(torch.empty(k * npoin, device=dev) for k in (1, 3, 1))
    s.D = tuple(torch.empty(k * npoin, device=dev) for k in (1, 3, 1))
    s.geo = (nelem, npoin, connec, s.Ngp, s.dNgp, s.He, s.gpvol)
    return s


def prepare(case, seed):
    return _tet_state(case, seed) if case["op"] == "tet" else _hex_state(case, seed)


# ---------------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------------
def run(s):
    if s.op == "tet":
        kernels.fem_convec(*s.geo, s.u, s.q, s.rho, s.pr, s.E, *s.C)
        kernels.fem_diffu(*s.geo, CP, PR, s.rho, s.u, s.Tem, s.mu_fluid, s.mu_e, s.mu_sgs, *s.D)
        return {"convec": s.C, "diffu": s.D}
    if s.op == "onecall":
        kernels.full_convec_diffusion_ijk(*s.geo, CP, PR, s.u, s.q, s.rho, s.pr, s.E, s.Tem, s.mu_fluid, s.mu_e,
                                          s.mu_sgs, *s.C, *s.D)
        return {"convec": s.C, "diffu": s.D}
    if s.op == "rk4":
        timestep.rk4_step(s, s.Ml, s.dt, s.rho, s.q, s.rhoE, s.ws)
        return {"state": (s.rho, s.q, s.rhoE)}
    if s.op == "visc":
        learn.entropy_viscosity(s, s.mu_e, s.nu, s.numax)
        kernels.full_diffusion_ijk(*s.geo, CP, PR, s.rho, s.u, s.Tem, s.mu_fluid, s.mu_e, s.mu_sgs, *s.D)
        return {"nu": s.nu, "numax": s.numax, "mu_e": s.mu_e, "diffu": s.D}
    if s.op == "learned":
        learn.learned_viscosity(s.mlp, s, s.nu, s.flag)
        return {"nu": s.nu, "flag": s.flag}
    if s.op == "mode_fp16":
        kernels.set_mode("fp16")
    kernels.full_convec_ijk(*s.geo, s.u, s.q, s.rho, s.pr, s.E, *s.C)
    kernels.full_diffusion_ijk(*s.geo, CP, PR, s.rho, s.u, s.Tem, s.mu_fluid, s.mu_e, s.mu_sgs, *s.D)
    if s.op == "mode_fp16":
        kernels.set_mode("fp32")
    return {"convec": s.C, "diffu": s.D}


def work(case):
    if case["op"] == "tet":
        if case["shared"]:
            m = max(2, round((case["nelem"] / 6) ** (1.0 / 3.0)))
            ne, nodes = 6 * m ** 3, (m + 1) ** 3
        else:
            ne, nodes = case["nelem"], 4 * case["nelem"]
        return {"bytes": ne * 2 * (16 + 144 + 16) + ne * 32 + 4 * nodes * (9 + 6 + 10), "flops": 3000.0 * ne}
    P = case["porder"]
    ne = case["nx"] * case["ny"] * case["nz"]
    pts = float(ne) * (P + 1) ** 3
    nodes = float(case["nx"] * P + 1) * (case["ny"] * P + 1) * (case["nz"] * P + 1)
    # Per point connec, He and gpvol, the element arrays; per node the fields in and the residuals out.
    conv_b, diff_b = pts * 44 + nodes * 56, pts * 52 + nodes * 44
    # Per point and direction: 22 convection and 11 diffusion contractions of P + 1 products, and the pointwise part.
    conv_f, diff_f = pts * (3 * 2 * 22 * (P + 1) + 150), pts * (3 * 2 * 11 * (P + 1) + 250)
    op = case["op"]
    if op in ("step", "mode_fp16"):
        return {"bytes": conv_b + diff_b, "flops": conv_f + diff_f}
    if op == "f64":
        return {"bytes": 2 * (conv_b + diff_b) - 8 * pts, "flops": conv_f + diff_f}
    if op == "onecall":  # connec, He, gpvol, rho and u once
        return {"bytes": conv_b + diff_b - pts * 44 - nodes * 16, "flops": conv_f + diff_f}
    if op == "rk4":  # four evaluations; the state in and out per stage, the running sum and the start's state
        return {"bytes": 4 * (conv_b + diff_b - pts * 44 - nodes * 16) + nodes * 4 * 60, "flops": 4 * (conv_f + diff_f)}
    if op == "visc":
        return {"bytes": diff_b + pts * (44 + 4) + nodes * 28, "flops": diff_f + pts * (3 * 2 * 7 * (P + 1) + 60)}
    return {"bytes": pts * 8 + nodes * 28 + 8 * ne, "flops": pts * 60 + 3000.0 * ne}


# ---------------------------------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------------------------------
class _Lattice:
    """Element points in lattice order [e, K, J, I] with the metric, for elements e0 .. e1."""

    def __init__(self, s, e0, e1):
        P, n = s.cfg.porder, s.cfg.nnode
        Q = P + 1
        inv = s.invAtoIJK.long() - 1
        dl = s.dlxigp_ip.double().view(Q, 3, n)
        v = inv.view(Q, Q, Q)
        self.Dm = [dl[:, 0, v[0, 0, :]].t(), dl[:, 1, v[0, :, 0]].t(), dl[:, 2, v[:, 0, 0]].t()]  # [r, c]
        self.m, self.Q, self.inv, self.npoin = e1 - e0, Q, inv, s.npoin
        self.nodes = (s.connec.view(n, s.nelem)[:, e0:e1][inv].long() - 1).t().reshape(self.m, Q, Q, Q)
        self.H = s.He.view(s.nelem, n, 3, 3)[e0:e1][:, inv].double().reshape(self.m, Q, Q, Q, 3, 3)  # [..., dir, i]
        self.gp = s.gpvol.view(s.nelem, n)[e0:e1][:, inv].double().reshape(self.m, Q, Q, Q)

    def at(self, f):
        return f.double()[self.nodes]

    def elem(self, f, s, e0, e1):
        return f.view(s.cfg.nnode, s.nelem)[:, e0:e1][self.inv].double().t().reshape(self.m, self.Q, self.Q, self.Q)

    def iso(self, f, d, transposed=False):
        """Derivative of f along lattice direction d (or the transposed operator)."""
        ax = 3 - d
        D = self.Dm[d].t() if transposed else self.Dm[d]
        out = torch.zeros_like(f)
        shape = [-1 if k == ax else 1 for k in range(4)]
        for c in range(self.Q):
            out.addcmul_(D[:, c].reshape(shape), f.narrow(ax, c, 1))
        return out

    def grad(self, f):
        g = [self.iso(f, d) for d in range(3)]
        return [sum(self.H[..., d, i] * g[d] for d in range(3)) for i in range(3)]

    def div(self, v):
        return sum(self.H[..., d, i] * self.iso(v[i], d) for d in range(3) for i in range(3))

    def wdiv(self, X):
        """Weak divergence: transposed derivatives of gpvol He(:, d) . X."""
        return sum(self.iso(self.gp * sum(self.H[..., d, i] * X[i] for i in range(3)), d, True) for d in range(3))

    def add(self, out, val, c=0):
        out[c * self.npoin:(c + 1) * self.npoin].index_add_(0, self.nodes.reshape(-1), val.reshape(-1))


def _chunks(s):
    step = max(1, int(2e6) // s.cfg.nnode)
    return [(e, min(e + step, s.nelem)) for e in range(0, s.nelem, step)]


def _zeros(npoin, dev):
    return tuple(torch.zeros(k * npoin, dtype=torch.float64, device=dev) for k in (1, 3, 1))


def _convec64(s, f):
    out = _zeros(s.npoin, s.He.device)
    for e0, e1 in _chunks(s):
        L = _Lattice(s, e0, e1)
        u = [L.at(f["u"][c * s.npoin:(c + 1) * s.npoin]) for c in range(3)]
        q = [L.at(f["q"][c * s.npoin:(c + 1) * s.npoin]) for c in range(3)]
        r, p = L.at(f["rho"]), L.at(f["pr"])
        H = L.at(f["E"]) + 0.5 * sum(x * x for x in u)
        gr, gp_, gH, grH = L.grad(r), L.grad(p), L.grad(H), L.grad(r * H)
        gu, gq = [L.grad(x) for x in u], [L.grad(x) for x in q]
        du, dq = sum(gu[i][i] for i in range(3)), sum(gq[i][i] for i in range(3))
        ugr = sum(u[i] * gr[i] for i in range(3))
        L.add(out[0], L.gp * 0.5 * (dq + r * du + ugr))
        for i in range(3):
            m = (L.div([q[i] * u[j] for j in range(3)]) + u[i] * dq + q[i] * du
                 + r * L.div([u[i] * u[j] for j in range(3)])) * 0.25 + gp_[i]
            m = m + 0.25 * (u[i] * ugr + sum(q[j] * gu[i][j] + u[j] * gq[i][j] for j in range(3)))
            L.add(out[1], L.gp * m, i)
        e = 0.25 * (L.div([r * H * x for x in u]) + H * dq + r * H * du + r * L.div([H * x for x in u])
                    + sum(q[i] * gH[i] + u[i] * grH[i] for i in range(3)) + H * ugr)
        L.add(out[2], L.gp * e)
    return out


def _diffu64(s, f, mu_e=None):
    out = _zeros(s.npoin, s.He.device)
    for e0, e1 in _chunks(s):
        L = _Lattice(s, e0, e1)
        u = [L.at(f["u"][c * s.npoin:(c + 1) * s.npoin]) for c in range(3)]
        r, T, muf = L.at(f["rho"]), L.at(f["Tem"]), L.at(f["mu_fluid"])
        me, ms = L.elem(s.mu_e if mu_e is None else mu_e, s, e0, e1), L.elem(s.mu_sgs, s, e0, e1)
        gr, gT, gu = L.grad(r), L.grad(T), [L.grad(x) for x in u]
        mu_f = muf + r * ms
        du = sum(gu[i][i] for i in range(3))
        tau = [[(mu_f + me) * (gu[i][j] + gu[j][i]) - (mu_f * (2.0 / 3.0) * du if i == j else 0.0) for j in range(3)]
               for i in range(3)]
        tu = [sum(tau[i][j] * u[j] for j in range(3)) for i in range(3)]
        L.add(out[0], me / r * L.wdiv(gr))
        L.add(out[2], L.wdiv(tu) + (muf * CP / PR + me * CP / PR + CP * r * ms / 0.9) * L.wdiv(gT))
        for m in range(3):
            L.add(out[1], L.wdiv(tau[m]), m)
    return out


def _visc64(s):
    r, p = s.rho.double(), s.pr.double()
    eta = r / (GAMMA - 1.0) * (p.log() - GAMMA * r.log())
    n_eta = (eta - eta.mean()).abs().max()
    nu, numax = (torch.empty(s.nelem, dtype=torch.float64, device=r.device) for _ in range(2))
    n = s.cfg.nnode
    mu_e = torch.empty(n, s.nelem, dtype=torch.float64, device=r.device)
    for e0, e1 in _chunks(s):
        L = _Lattice(s, e0, e1)
        u = [L.at(s.u[c * s.npoin:(c + 1) * s.npoin]) for c in range(3)]
        et, rr, pp = L.at(eta), L.at(r), L.at(p)
        ge = L.grad(et)
        R = L.div([et * x for x in u]) - et * L.div(u) - sum(u[i] * ge[i] for i in range(3))
        h = L.gp.reshape(L.m, -1).sum(1) ** (1.0 / 3.0) / s.cfg.porder
        speed = sum(x * x for x in u).sqrt() + (GAMMA * pp / rr).sqrt()
        numax[e0:e1] = CMAX * h * speed.reshape(L.m, -1).amax(1)
        nu[e0:e1] = torch.minimum(numax[e0:e1], CE * h * h * R.abs().reshape(L.m, -1).amax(1) / n_eta)
        mu_e[:, e0:e1] = r[s.connec.view(n, s.nelem)[:, e0:e1].long() - 1] * nu[e0:e1]
    return nu, numax, mu_e.reshape(-1)


def _rk64(s):
    Ml = torch.zeros(s.npoin, dtype=torch.float64, device=s.He.device)
    node = s.connec.view(s.cfg.nnode, s.nelem).t().reshape(-1).long() - 1
    Ml.index_add_(0, node, s.gpvol.double())
    U0 = [s.rho.double(), s.q.double(), s.rhoE.double()]

    def rhs(r, q, re):
        u = (q.view(3, -1) / r).reshape(-1)
        pr = (GAMMA - 1.0) * (re - 0.5 * r * u.view(3, -1).square().sum(0))
        f = {"rho": r, "u": u, "q": q, "pr": pr, "E": re / r, "Tem": pr / (r * RGAS), "mu_fluid": s.mu_fluid}
        return [-((a + b).view(-1, s.npoin) / Ml).reshape(-1) for a, b in zip(_convec64(s, f), _diffu64(s, f))]

    k1 = rhs(*U0)
    k2 = rhs(*[a + 0.5 * s.dt * k for a, k in zip(U0, k1)])
    k3 = rhs(*[a + 0.5 * s.dt * k for a, k in zip(U0, k2)])
    k4 = rhs(*[a + s.dt * k for a, k in zip(U0, k3)])
    return tuple(a + s.dt / 6.0 * (w + 2.0 * x + 2.0 * y + z) for a, w, x, y, z in zip(U0, k1, k2, k3, k4))


def _tet64(s):
    c, d = _zeros(s.npoin, s.He.device), _zeros(s.npoin, s.He.device)
    Nf = s.Ngp.double().view(4, 4).t()  # Ngp(igaus, inode) -> [igaus, inode]
    dN = s.dNgp.double().view(4, 4, 3)  # [igaus, inode, idime]
    ein = torch.einsum
    for e0 in range(0, s.nelem, 1 << 18):
        e1 = min(e0 + (1 << 18), s.nelem)
        con = s.connec.view(4, s.nelem)[:, e0:e1].long().t() - 1
        H = s.He.double().view(s.nelem, 4, 3, 3)[e0:e1]  # [e, g, dir, i]
        gv = s.gpvol.double().view(s.nelem, 4)[e0:e1]
        gc = ein("egdi,gad->egai", H, dN)

        def sc(f):
            return f.double()[con]

        def vec(f):
            return torch.stack([f[k * s.npoin:(k + 1) * s.npoin].double()[con] for k in range(3)], -1)

        def add(out, val):
            for k in range(out.numel() // s.npoin):
                w = val if val.dim() == 2 else val[..., k]
                out[k * s.npoin:(k + 1) * s.npoin].index_add_(0, con.reshape(-1), w.reshape(-1))

        U, Qv, r, p = vec(s.u), vec(s.q), sc(s.rho), sc(s.pr)
        Ep = sc(s.E) + p
        gR, gE, gP = (ein("egai,ea->egi", gc, x) for x in (r, Ep, p))
        gU = ein("egaj,eai->egij", gc, U)
        divQ, divU = ein("egai,eai->eg", gc, Qv), ein("egii->eg", gU)
        divFe = ein("egai,ea,eai->eg", gc, Ep, U)
        divF = ein("egaj,eai,eaj->egi", gc, Qv, U)
        w = gv[:, :, None] * Nf[None] * 0.5
        add(c[0], (w * (divQ[:, :, None] + r[:, None, :] * divU[:, :, None] + ein("egi,eai->ega", gR, U))).sum(1))
        add(c[2], (w * (divFe[:, :, None] + Ep[:, None, :] * divU[:, :, None] + ein("egi,eai->ega", gE, U))).sum(1))
        mom = (divF[:, :, None, :] + Qv[:, None] * divU[:, :, None, None] + ein("egij,eaj->egai", gU, Qv)
               + ein("eai,eaj,egj->egai", U, U, gR) + gP[:, :, None, :])
        add(c[1], (w[..., None] * mom).sum(1))
        # The reference's diffusion reads Ngp(inode, igaus): the transpose of the convection's.
        T, mf = sc(s.Tem), sc(s.mu_fluid)
        me, ms = (x.double().view(4, s.nelem)[:, e0:e1].t() for x in (s.mu_e, s.mu_sgs))
        N2 = Nf
        aR = r @ N2.t()
        aNu = (me @ N2.t()) / aR
        aMu = ein("ga,ega->eg", N2, mf[:, None] + aR[:, :, None] * ms[:, None] + me[:, None])
        aK = ein("ga,ega->eg", N2, mf[:, None] * (CP / PR) + me[:, None] / 0.4 + aR[:, :, None] * ms[:, None] / 0.9)
        gT = ein("egai,ea->egi", gc, T)
        gV = ein("egai,eaj->egij", gc, U)
        tau = gV + gV.transpose(2, 3) - (2.0 / 3.0) * ein("egii->eg", gV)[:, :, None, None] * torch.eye(3, device=r.device)
        tU = ein("egij,egj->egi", tau, ein("ga,eaj->egj", N2, U))
        add(d[0], ein("eg,egai,egi->ea", gv * aNu, gc, gR))
        add(d[2], ein("eg,egai,egi->ea", gv, gc, aMu[:, :, None] * tU + aK[:, :, None] * gT))
        add(d[1], ein("eg,egaj,egij->eai", gv * aMu, gc, tau))
    return c, d


def exact(case, seed):
    if case["op"] == "learned":  # a network's output with a threshold: no value of its own in 64 bits
        return None
    s = prepare(case, seed)
    if s.op == "tet":
        c, d = _tet64(s)
        return {"convec": c, "diffu": d}
    if s.op == "rk4":
        return {"state": _rk64(s)}
    f = {k: getattr(s, k) for k in ("rho", "u", "q", "pr", "E", "Tem", "mu_fluid")}
    if s.op == "visc":
        nu, numax, mu_e = _visc64(s)
        return {"nu": nu, "numax": numax, "mu_e": mu_e, "diffu": _diffu64(s, f, mu_e)}
    return {"convec": _convec64(s, f), "diffu": _diffu64(s, f)}
