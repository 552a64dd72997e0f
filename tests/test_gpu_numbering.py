"""The element-group kernels on meshes that are not numbered along x.

How a warp gathers (past the L1 or through it, lanes along the elements or along xi) depends on the order
and on the numbers that it meets; the results may not.  One mesh in four numberings: along x, nodes in
random order, elements in random order, every element with nodes of its own (the reference driver's
form, whose residuals add up to the shared mesh's node by node).  An element's contributions are the same
operations in each; 1e-6 leaves room for the order of the nodes' sums, which the fields' grid-scale
content keeps from cancelling."""
import numpy as np
import pytest

from minisod2d_gb300 import capi, fem, kernels, learn
from oracle import oracle as O
from tests.test_gpu_groups import _tables

pytestmark = pytest.mark.gpu
FIELDS = dict(rho=1, pr=1, E=1, Tem=1, mu_fluid=1, u=3, q=3)


class Mesh:
    def __init__(self, cuda, P, dims, odd):
        import torch

        t = _tables(P, odd)
        connec, coord, self.ne, self.npn = fem.structured_mesh(P, *dims, t, 0.1, P)
        tj = fem.element_tables(P, np.float32)
        He, gp = O.elem_jacobian(P, self.ne, self.npn, connec, coord, tj["dNgp"], tj["wgp"], np.float32)
        rng = np.random.default_rng(P)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
        self.P, self.n, self.cuda = P, (P + 1) ** 3, cuda
        self.tab = [up(t[k]) for k in ("dlxigp_ip", "invAtoIJK", "AtoI", "AtoJ", "AtoK")]
        self.connec, self.He, self.gp = up(connec).view(self.n, -1), up(He).view(self.ne, -1), up(gp).view(self.ne, -1)
        self.f = {k: up((1.0 + 0.3 * rng.random((c, self.npn))).astype(np.float32)) for k, c in FIELDS.items()}
        self.f["u"] = self.f["u"] - 1.15
        self.mu = [up(rng.random((self.n, self.ne)).astype(np.float32)) for _ in range(2)]
        self.nu = up(rng.random(self.ne).astype(np.float32))

    def results(self, connec=None, order=None, f=None, npn=None):
        """Residuals (component, node) of convection, diffusion and its per-element form, and the
        estimator's viscosity, for this connec (row a, element e), element order and node fields."""
        import torch

        ne = self.ne
        npn = npn or self.npn
        order = torch.arange(ne, device=self.cuda) if order is None else order
        connec = (self.connec if connec is None else connec)[:, order].contiguous().view(-1)
        f = {k: v.contiguous().view(-1) for k, v in (f or self.f).items()}
        He, gp = (x[order].contiguous().view(-1) for x in (self.He, self.gp))
        mu = [x[:, order].contiguous().view(-1) for x in self.mu]
        nu = self.nu[order].contiguous()
        geo = (ne, npn, connec, None, None, He, gp, self.tab[0], None, *self.tab[1:])
        new = lambda: [torch.full((k, npn), 7.0, device=self.cuda) for k in (1, 3, 1)]
        ptr = lambda *x: [learn._p(a) for a in x]
        out = [new() for _ in range(3)]
        flat = [[x.view(-1) for x in o] for o in out]
        kernels.full_convec_ijk(*geo, f["u"], f["q"], f["rho"], f["pr"], f["E"], *flat[0])
        kernels.full_diffusion_ijk(*geo, 1004.5, 0.71, f["rho"], f["u"], f["Tem"], f["mu_fluid"], *mu, *flat[1])
        c_geo = [self.P, ne, npn] + ptr(connec, He, gp, *self.tab)
        capi.call("msod_diffusion_ijk_nu", *c_geo, 1004.5, 0.71, *ptr(f["rho"], f["u"], f["Tem"], f["mu_fluid"], nu,
                                                                     mu[1], *out[2]), capi.current_stream())
        visc = []
        if self.P < 8:
            est, cap = torch.empty(ne, device=self.cuda), torch.empty(ne, device=self.cuda)
            mu_e = torch.empty(self.n * ne, device=self.cuda)
            capi.call("msod_entropy_viscosity", *c_geo, *ptr(f["rho"], f["u"], f["pr"]), 1.4, 0.1, 0.5, 1,
                      *ptr(mu_e, est, cap), capi.current_stream())
            back = torch.argsort(order)
            visc = [est[back], cap[back], mu_e.view(self.n, ne)[:, back]]
        return out, visc


def _same(a, b, what):
    import torch

    (ra, va), (rb, vb) = a, b
    for call, x, y in zip(("convection", "diffusion", "nu form"), ra, rb):
        for name, p, q in zip(("mass", "mom", "ener"), x, y):
            err = float((p.double() - q.double()).norm() / q.double().norm())
            assert err <= 1e-6, (what, call, name, err)
    for p, q in zip(va, vb):
        assert float((p.double() - q.double()).norm() / q.double().norm()) <= 1e-6, (what, "estimator")


CASES = [(1, (5, 7, 3), False), (1, (9, 5, 2), True), (2, (5, 3, 2), True), (2, (7, 1, 1), False), (3, (5, 3, 2), True),
         (4, (3, 2, 2), False), (5, (3, 2, 1), True), (6, (2, 2, 1), False), (7, (3, 1, 1), True), (8, (2, 2, 1), False)]


@pytest.mark.parametrize("P,dims,odd", CASES)
def test_numberings(cuda, P, dims, odd):
    import torch

    m = Mesh(cuda, P, dims, odd)
    ref = m.results()
    g = torch.Generator(device=cuda)
    g.manual_seed(P)
    # Elements in random order.
    _same(m.results(order=torch.randperm(m.ne, generator=g, device=cuda)), ref, "elements")
    # Nodes in random order: new number of node p is to[p].
    to = torch.randperm(m.npn, generator=g, device=cuda)
    f = {k: torch.empty_like(v) for k, v in m.f.items()}
    for k, v in m.f.items():
        f[k][:, to] = v
    r, v = m.results(connec=(to[m.connec.long() - 1] + 1).int(), f=f)
    _same(([[x[:, to] for x in o] for o in r], v), ref, "nodes")
    # Nodes of its own for every element.  (The estimator's statistics are over the nodes, so its
    # normalisation differs and only its cap is compared.)
    own = (torch.arange(m.ne * m.n, device=cuda, dtype=torch.int32).view(m.ne, m.n).t() + 1).contiguous()
    at = m.connec.t().reshape(-1).long() - 1
    r, v = m.results(connec=own, f={k: x[:, at] for k, x in m.f.items()}, npn=m.ne * m.n)
    back = lambda x: torch.zeros(x.shape[0], m.npn, dtype=torch.float64, device=cuda).index_add_(1, at, x.double())
    # mass flux and kappa are formed at the output point: the same in either form
    _same(([[back(x) for x in o] for o in r], v[1:2]), (ref[0], ref[1][1:2]), "own nodes")


@pytest.mark.parametrize("P", range(1, 9))
def test_missing_nodes(cuda, P):
    """Entries outside 1..npoin read as a node of zeros and are not assembled, whatever the numbering:
    the residuals of the mesh in which such a node exists."""
    import torch

    m = Mesh(cuda, P, (3, 2, 1), True)
    own = (torch.arange(m.ne * m.n, device=cuda, dtype=torch.int32).view(m.ne, m.n).t() + 1).contiguous()
    at = m.connec.t().reshape(-1).long() - 1
    fown = {k: x[:, at] for k, x in m.f.items()}
    for connec, f, npn in ((m.connec, m.f, m.npn), (own, fown, m.ne * m.n)):
        bad, more = connec.clone(), connec.clone()
        bad[5, 1], bad[2, 0], bad[0, 3] = 0, npn + 9, -4
        more[5, 1] = more[2, 0] = more[0, 3] = npn + 1
        g = {k: torch.cat([v, torch.zeros(v.shape[0], 1, device=cuda)], 1) for k, v in f.items()}
        a, _ = m.results(connec=bad, f=f, npn=npn)
        b, _ = m.results(connec=more, f=g, npn=npn + 1)
        _same((a, []), ([[x[:, :npn] for x in o] for o in b], []), "missing")
