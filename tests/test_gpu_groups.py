"""The element-group kernels at their edges, against the oracle.

Element counts that leave the last group of a block partly empty; He and gpvol that start off a
16-byte boundary (the bulk copies' unaligned ends); derivative tables whose directions differ and
whose rows do not sum to zero; a momentum that is not rho u.  Tolerance: the FP32 criterion of
tests/test_gpu_parity.py (1e-5 of the FP32 oracle, or within the FP32 floor where that is larger)."""
import numpy as np
import pytest

from minisod2d_gb300 import fem, kernels
from oracle import oracle as O
from tests.test_gpu_parity import NTH, TOL32, _compare

pytestmark = pytest.mark.gpu


def _tables(P, odd):
    t = fem.element_tables(P, np.float32)
    if odd:
        n, Q = (P + 1) ** 3, P + 1
        d = t["dlxigp_ip"].reshape(Q, 3, n)
        for k in range(3):
            d[:, k] = d[:, k] * np.float32(1.0 + 0.2 * k) + np.float32(0.05 * (k + 1))
    return t


def _up(a, cuda, shift=0):
    import torch

    buf = torch.zeros(a.size + 4, dtype=torch.float32, device=cuda)
    buf[shift:shift + a.size] = torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    return buf[shift:shift + a.size]


@pytest.mark.parametrize("P,dims,shift,odd", [(1, (5, 7, 2), 0, False), (1, (3, 3, 1), 1, True), (2, (17, 1, 1), 3, True),
                                              (3, (3, 3, 1), 1, False), (3, (4, 2, 1), 0, True), (4, (3, 2, 1), 0, False),
                                              (4, (11, 1, 1), 2, True), (5, (5, 1, 1), 1, True), (6, (1, 1, 1), 3, False),
                                              (6, (3, 1, 1), 0, True), (7, (3, 1, 1), 1, True), (8, (3, 1, 1), 2, True)])
def test_group_edges(cuda, P, dims, shift, odd):
    import torch

    t = _tables(P, odd)
    mesh_t = fem.element_tables(P, np.float32)
    connec, coord, ne, npn = fem.structured_mesh(P, *dims, mesh_t, 0.1, P)
    He, gp = O.elem_jacobian(P, ne, npn, connec, coord, mesh_t["dNgp"], mesh_t["wgp"], np.float32)
    geom = dict(t, connec=connec, He=He, gpvol=gp)
    g64 = dict(t, connec=connec, He=He.astype(np.float64), gpvol=gp.astype(np.float64),
               dlxigp_ip=t["dlxigp_ip"].astype(np.float64))
    rng = np.random.default_rng(P)
    f = {k: (1.0 + 0.3 * rng.random(npn)).astype(np.float32) for k in ("rho", "pr", "E", "Tem", "mu_fluid")}
    f["u"], f["q"] = (rng.standard_normal(3 * npn).astype(np.float32) for _ in range(2))
    n = (P + 1) ** 3
    mu = [rng.random(ne * n).astype(np.float32) for _ in range(2)]
    dev = {k: torch.from_numpy(v).to(cuda) for k, v in f.items()}
    ti = {k: torch.from_numpy(t[k]).to(cuda) for k in ("dlxigp_ip", "invAtoIJK", "AtoI", "AtoJ", "AtoK")}
    geo = (ne, npn, torch.from_numpy(connec).to(cuda), None, None, _up(He, cuda, shift), _up(gp, cuda, shift),
           ti["dlxigp_ip"], None, ti["invAtoIJK"], ti["AtoI"], ti["AtoJ"], ti["AtoK"])
    out = [torch.empty(k * npn, device=cuda) for k in (1, 3, 1)]
    kernels.full_convec_ijk(*geo, dev["u"], dev["q"], dev["rho"], dev["pr"], dev["E"], *out)
    a = (P, ne, npn)
    ref = [O.full_convec_ijk(*a, g, f["u"], f["q"], f["rho"], f["pr"], f["E"], dt, nthreads=NTH)
           for g, dt in ((geom, np.float32), (g64, np.float64))]
    _compare(out, ref[0], TOL32, "convec group edges P=%d" % P, ref[1])
    kernels.full_diffusion_ijk(*geo, 1004.5, 0.71, dev["rho"], dev["u"], dev["Tem"], dev["mu_fluid"],
                               *[torch.from_numpy(m).to(cuda) for m in mu], *out)
    ref = [O.full_diffusion_ijk(*a, g, 1004.5, 0.71, f["rho"], f["u"], f["Tem"], f["mu_fluid"], *mu, dt, nthreads=NTH)
           for g, dt in ((geom, np.float32), (g64, np.float64))]
    _compare(out, ref[0], TOL32, "diffu group edges P=%d" % P, ref[1])


@pytest.mark.parametrize("P", range(1, 9))
def test_large_meshes_as_small_ones(cuda, P):
    """Large meshes take the diffusion's matrices from the constant bank (the line lies between half a
    million and twelve million element points): copies of a small mesh, whose own call reads them
    from shared memory, give the small mesh's residuals on every copy.  The operations are the same;
    1e-6 leaves room for the order of the nodes' sums."""
    import torch

    t = fem.element_tables(P, np.float32)
    connec, coord, ne, npn = fem.structured_mesh(P, 3, 2, 2, t, 0.1, P)
    He, gp = O.elem_jacobian(P, ne, npn, connec, coord, t["dNgp"], t["wgp"], np.float32)
    n = (P + 1) ** 3
    rng = np.random.default_rng(P)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    f = {k: up((1.0 + 0.3 * rng.random(npn)).astype(np.float32)) for k in ("rho", "Tem", "mu_fluid")}
    f["u"] = up(rng.standard_normal(3 * npn).astype(np.float32))
    mu = [up(rng.random(ne * n).astype(np.float32)) for _ in range(2)]
    con, He, gp = up(connec), up(He), up(gp)
    tab = [up(t[k]) for k in ("dlxigp_ip", "invAtoIJK", "AtoI", "AtoJ", "AtoK")]

    def run(copies):
        c = con.view(n, 1, ne) + (torch.arange(copies, device=cuda, dtype=torch.int32) * npn).view(1, -1, 1)
        rep = lambda x, lead: x.view(lead, 1, -1).expand(lead, copies, -1).reshape(-1).contiguous()
        m = npn * copies
        out = [torch.empty(k * m, device=cuda) for k in (1, 3, 1)]
        kernels.full_diffusion_ijk(ne * copies, m, c.reshape(-1).contiguous(), None, None, rep(He, 1), rep(gp, 1), tab[0],
                                   None, *tab[1:], 1004.5, 0.71, rep(f["rho"], 1), rep(f["u"], 3), rep(f["Tem"], 1),
                                   rep(f["mu_fluid"], 1), *[rep(x, n) for x in mu], *out)
        return [o.view(k, copies, npn) for o, k in zip(out, (1, 3, 1))]

    small = run(1)
    limit = 500000 if P in (5, 6) else (12000000 if P == 4 else 3000000)
    large = run(limit // (ne * n) + 2)
    for a, b in zip(large, small):
        err = torch.linalg.vector_norm((a - b).double()) / torch.linalg.vector_norm(b.double().expand_as(a))
        assert float(err) <= 1e-6, (P, float(err))


@pytest.mark.parametrize("P,nx", [(4, 12), (2, 5)])
def test_estimator_without_normalisation(cuda, P, nx):
    """normalise = 0 takes n_eta = 1, so nu = min(nu_max, nu_E n_eta) of the normalised call: nu_E scales by
    the same factor in every element that nu_max does not cap (two float roundings of the ratio)."""
    import torch

    from minisod2d_gb300 import capi, learn, workload

    dev = workload.DeviceCase(workload.HostCase(workload.custom(P, nx, 0.05)))
    nu = [torch.empty(dev.nelem, device=cuda) for _ in range(2)]
    cap = torch.empty(dev.nelem, device=cuda)
    for norm in (1, 0):  # ce small: no element is capped
        capi.call("msod_entropy_viscosity", *learn._geo(dev), *(learn._p(t) for t in (dev.rho, dev.u, dev.pr)), 1.4,
                  1e-6, 0.5, norm, None, learn._p(nu[norm]), learn._p(cap), capi.current_stream())
    live = (nu[0] < 0.9 * cap) & (nu[1] < 0.9 * cap) & (nu[1] > 0)
    assert int(live.sum()) > dev.nelem // 2
    ratio = (nu[0][live].double() / nu[1][live].double())
    assert float((ratio / ratio.median() - 1).abs().max()) < 5e-7
