"""The statistics, estimator and features that start over one another: their norm, and their replay.

The last block of the statistics forms n_eta = max |eta - mean(eta)|, eta = rho / (gamma - 1) log(p /
rho^gamma), for the kernels behind it.  FP32 entropies carry a few roundings of logarithms of order
one each, against n_eta of order 0.1 to 1: 1e-5 relative."""
import numpy as np
import pytest

from minisod2d_gb300 import capi, learn, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,nx", [(4, 12), (2, 5), (7, 4), (1, 40)])
@pytest.mark.parametrize("kind", [capi.MSOD_FIELDS_SMOOTH, capi.MSOD_FIELDS_SHOCK])
def test_normalised_by_the_entropy_norm(cuda, P, nx, kind):
    """nu_E of normalise = 0 over that of normalise = 1 is n_eta in every element."""
    import torch

    dev = workload.DeviceCase(workload.HostCase(workload.custom(P, nx, 0.05, kind=kind, seed=3)))
    r, p = dev.rho.double(), dev.pr.double()
    eta = r / 0.4 * (p.log() - 1.4 * r.log())
    n_eta = float((eta - eta.mean()).abs().max())
    assert abs(n_eta - 1.0) > 0.05
    nu, cap = {}, torch.empty(dev.nelem, device=cuda)
    for norm in (True, False):
        nu[norm] = torch.empty(dev.nelem, device=cuda)
        learn.entropy_viscosity(dev, nu=nu[norm], numax=cap, ce=1e-6, normalise=norm)  # ce small: no cap
    live = (nu[True] < 0.9 * cap) & (nu[False] < 0.9 * cap) & (nu[True] > 0)
    assert int(live.sum()) > dev.nelem // 2
    ratio = nu[False][live].double() / nu[True][live].double()
    assert float((ratio / n_eta - 1.0).abs().max()) < 1e-5, (n_eta, float(ratio.median()))


@pytest.mark.parametrize("nx", [6, 24])
def test_chain_in_a_graph(cuda, nx):
    """Entropy viscosity and learned viscosity replay from a graph to the eager results, on the captured
    fields and on others (24^3 elements: the features start over the statistics; 6^3: behind them)."""
    import torch

    cfg = workload.custom(4, nx, 0.0, kind=capi.MSOD_FIELDS_SHOCK, seed=1)
    host = workload.HostCase(cfg)
    dev = workload.DeviceCase(host)
    mlp = learn.Mlp()
    mlp.load(learn.shipped_weights("learned_48"))
    n = dev.nelem
    mu, nu, cap, net = (torch.empty(k, device=cuda) for k in (n * cfg.nnode, n, n, n))
    flag = torch.empty(n, dtype=torch.int32, device=cuda)

    def step():
        learn.entropy_viscosity(dev, mu, nu, cap)
        learn.learned_viscosity(mlp, dev, net, flag)

    def results():
        torch.cuda.synchronize()
        return [x.clone() for x in (mu, nu, cap, net, flag)]

    hosts = (host, host.with_seed(7))
    eager = []
    for h in hosts:
        dev.set_fields(h)
        step()
        eager.append(results())
    assert int(eager[0][4].sum()) > 0 and not torch.equal(eager[0][1], eager[1][1])
    g, side = torch.cuda.CUDAGraph(), torch.cuda.Stream(device=cuda)
    with torch.cuda.stream(side):
        with torch.cuda.graph(g, stream=side):
            step()
    torch.cuda.synchronize()
    for h, want in zip(hosts, eager):
        dev.set_fields(h)
        for x in (mu, nu, cap, net):
            x.fill_(-1.0)
        flag.fill_(9)
        for _ in range(2):
            g.replay()
        got = results()
        assert torch.equal(got[4], want[4])
        for a, b in zip(got[:4], want[:4]):
            assert float((a.double() - b.double()).norm() / b.double().norm()) < 1e-6
