"""The diffusion's derivative matrices in the constant bank, where they can be wrong or stale.

Large FP32 meshes take the matrices from a bank that each call fills on its stream.  Tables whose three
directions differ, and calls with other tables right behind one another (eager and replayed from a
graph), against copies of a small mesh whose own call reads the caller's tables in every block.  The
operations are the same on both paths; 1e-6 leaves room for the order of the nodes' sums."""
import numpy as np
import pytest

from minisod2d_gb300 import fem, kernels
from oracle import oracle as O
from tests.test_gpu_groups import _tables

pytestmark = pytest.mark.gpu
LIMIT = {P: 500000 if P in (5, 6) else (12000000 if P == 4 else 3000000) for P in range(1, 9)}


class Copies:
    """Enough copies of a small mesh for the bank, and the small mesh itself, with several tables."""

    def __init__(self, cuda, P):
        import torch

        t = fem.element_tables(P, np.float32)
        connec, coord, self.ne, self.npn = fem.structured_mesh(P, 3, 2, 2, t, 0.1, P)
        He, gp = O.elem_jacobian(P, self.ne, self.npn, connec, coord, t["dNgp"], t["wgp"], np.float32)
        self.n = (P + 1) ** 3
        rng = np.random.default_rng(P)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
        f = lambda k: up((1.0 + 0.3 * rng.random(k * self.npn)).astype(np.float32))
        base = dict(con=up(connec), He=up(He), gp=up(gp), rho=f(1), Tem=f(1), mu=f(1), u=f(3) - 1.15,
                    me=up(rng.random(self.ne * self.n).astype(np.float32)), ms=up(rng.random(self.ne * self.n).astype(np.float32)),
                    nu=up(rng.random(self.ne).astype(np.float32)), pr=f(1), E=f(1), q=f(3) - 1.15)
        self.tab = [[up(x[k]) for k in ("dlxigp_ip", "invAtoIJK", "AtoI", "AtoJ", "AtoK")]
                    for x in (_tables(P, False), _tables(P, True))]
        self.case = {}
        for copies in (1, LIMIT[P] // (self.ne * self.n) + 2):
            rep = lambda x, lead: x.view(lead, 1, -1).expand(lead, copies, -1).reshape(-1).contiguous()
            c = base["con"].view(self.n, 1, self.ne) + (torch.arange(copies, device=cuda, dtype=torch.int32)
                                                        * self.npn).view(1, -1, 1)
            lead = dict(He=1, gp=1, rho=1, Tem=1, mu=1, u=3, me=self.n, ms=self.n, nu=1, pr=1, E=1, q=3)
            d = {k: rep(base[k], v) for k, v in lead.items()}
            d.update(con=c.reshape(-1).contiguous(), copies=copies)
            self.case[copies > 1] = d
        self.P, self.cuda = P, cuda

    def outputs(self, large):
        import torch

        return [torch.full((k * self.npn * self.case[large]["copies"],), 7.0, device=self.cuda) for k in (1, 3, 1)]

    def call(self, large, odd, out, nu=False):
        from minisod2d_gb300 import capi
        from minisod2d_gb300.learn import _p

        d, t = self.case[large], self.tab[odd]
        ne, npn = self.ne * d["copies"], self.npn * d["copies"]
        if nu:
            capi.call("msod_diffusion_ijk_nu", self.P, ne, npn, _p(d["con"]), _p(d["He"]), _p(d["gp"]), *[_p(x) for x in t],
                      1004.5, 0.71, _p(d["rho"]), _p(d["u"]), _p(d["Tem"]), _p(d["mu"]), _p(d["nu"]), _p(d["ms"]),
                      *[_p(x) for x in out], capi.current_stream())
        else:
            kernels.full_diffusion_ijk(ne, npn, d["con"], None, None, d["He"], d["gp"], t[0], None, *t[1:], 1004.5, 0.71,
                                       d["rho"], d["u"], d["Tem"], d["mu"], d["me"], d["ms"], *out)

    def both(self, large, odd, out):
        """Convection and diffusion in one call."""
        d, t = self.case[large], self.tab[odd]
        kernels.full_convec_diffusion_ijk(self.ne * d["copies"], self.npn * d["copies"], d["con"], None, None, d["He"],
                                          d["gp"], t[0], None, *t[1:], 1004.5, 0.71, d["u"], d["q"], d["rho"], d["pr"],
                                          d["E"], d["Tem"], d["mu"], d["me"], d["ms"], *out)

    def check(self, large, small, what):
        import torch

        for k, a, b in zip((1, 3, 1), large, small):
            a, b = a.view(k, -1, self.npn), b.view(k, 1, self.npn)
            err = torch.linalg.vector_norm((a - b).double()) / torch.linalg.vector_norm(b.double().expand_as(a))
            assert float(err) <= 1e-6, (self.P, what, float(err))


@pytest.mark.parametrize("P", range(1, 9))
def test_calls_with_other_tables_back_to_back(cuda, P):
    import torch

    m = Copies(cuda, P)
    small = {}
    for nu in (False, True):
        for odd in (0, 1):
            small[nu, odd] = m.outputs(False)
            m.call(False, odd, small[nu, odd], nu)
        # The two tables' residuals differ by far more than the bound.
        assert float((small[nu, 0][1] - small[nu, 1][1]).norm() / small[nu, 0][1].norm()) > 1e-2
    order = [(False, 0), (False, 1), (False, 0), (True, 1), (True, 0), (False, 1)]
    large = [m.outputs(True) for _ in order]
    torch.cuda.synchronize()
    for (nu, odd), out in zip(order, large):
        m.call(True, odd, out, nu)
    for key, out in zip(order, large):
        m.check(out, small[key], key)


@pytest.mark.parametrize("P", [4, 5])
def test_bank_in_a_graph(cuda, P):
    """Captured calls of both tables replay to the eager results, also when an eager call with other
    tables comes between two replays."""
    import torch

    m = Copies(cuda, P)
    small = [m.outputs(False) for _ in range(2)]
    large = [m.outputs(True) for _ in range(2)]
    for odd in (0, 1):
        m.call(False, odd, small[odd])
        m.call(True, odd, large[odd])
    torch.cuda.synchronize()
    g, side = torch.cuda.CUDAGraph(), torch.cuda.Stream(device=cuda)
    with torch.cuda.stream(side):
        with torch.cuda.graph(g, stream=side):
            m.call(True, 0, large[0])
            m.call(True, 1, large[1])
    torch.cuda.synchronize()
    for odd in (1, 0):
        for out in large:
            for x in out:
                x.fill_(-7.0)
        m.call(True, odd, m.outputs(True))
        g.replay()
        torch.cuda.synchronize()
        for k in (0, 1):
            m.check(large[k], small[k], ("replay", odd, k))


@pytest.mark.parametrize("P", [1, 4, 5, 7])
def test_one_call_with_other_tables_back_to_back(cuda, P):
    import torch

    m = Copies(cuda, P)
    small = [m.outputs(False) + m.outputs(False) for _ in range(2)]
    for odd in (0, 1):
        m.both(False, odd, small[odd])
    order = [0, 1, 0, 1]
    large = [m.outputs(True) + m.outputs(True) for _ in order]
    torch.cuda.synchronize()
    for odd, out in zip(order, large):
        m.both(True, odd, out)
    for odd, out in zip(order, large):
        m.check(out[:3], small[odd][:3], ("convection", odd))
        m.check(out[3:], small[odd][3:], ("diffusion", odd))
