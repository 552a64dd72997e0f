"""Tensor-core residuals beside non-finite values: they stay where the formulas take them.

On a mesh whose elements share no node, a node's viscosity or energy enters its own element only: the
viscosity all diffusion residuals but the mass, the energy the convection's energy residual only.  The
blocks are persistent, so with more elements than resident blocks one goes from the bad element to
others: those must give the bits of the clean run, and so must the bad element's other residuals.
(Each node belongs to one element: no sum depends on an order.)"""
import numpy as np
import pytest

from minisod2d_gb300 import fem, workload

pytestmark = pytest.mark.gpu


def _disconnected(cuda, P, nx):
    """A jittered structured case with nodes of its own for every element (node e n + a)."""
    import torch

    host = workload.HostCase(workload.custom(P, nx, 0.05, nmodes=8, seed=5))
    dev = workload.DeviceCase(host, device=cuda)
    n, node = host.cfg.nnode, dev.connec.view(host.cfg.nnode, -1).t().reshape(-1).long() - 1
    for k in ("rho", "u", "q", "pr", "E", "Tem", "mu_fluid"):
        f = getattr(dev, k)
        setattr(dev, k, f.view(-1, dev.npoin)[:, node].reshape(-1).contiguous())
    dev.connec = torch.from_numpy(fem.mesh_disconnected(P, dev.nelem, host.tables, False)[0]).to(cuda)
    dev.npoin = dev.nelem * n
    rng = np.random.default_rng(P)
    for k in ("mu_e", "mu_sgs"):
        setattr(dev, k, torch.from_numpy((1e-3 * rng.random(dev.nelem * n)).astype(np.float32)).to(cuda))
    return dev


@pytest.mark.parametrize("prec", ["fp16", "bf16"])
@pytest.mark.parametrize("P,nx", [(1, 24), (2, 20), (3, 17), (4, 15), (5, 13), (6, 12), (7, 11)])
def test_nonfinite_value_stays_in_its_element(cuda, P, nx, prec):
    import torch

    dev = _disconnected(cuda, P, nx)
    n = dev.cfg.nnode
    clean = dev.diffu_mixed(prec), dev.convec_mixed(prec)
    # Every point of an early element but lattice node (0,0,0), by which the fields are shifted.
    bad = 7
    at = bad * n + dev.invAtoIJK.long()[1:] - 1
    for value in (float("inf"), float("nan")):
        keep = dev.mu_fluid[at].clone(), dev.E[at].clone()
        dev.mu_fluid[at], dev.E[at] = value, value
        got = dev.diffu_mixed(prec), dev.convec_mixed(prec)
        dev.mu_fluid[at], dev.E[at] = keep
        for call, a, b in zip(("diffusion", "convection"), got, clean):
            for name, x, y in zip(("mass", "mom", "ener"), a, b):
                same = (x == y).view(-1, dev.nelem, n)
                hit = name == "ener" or (name, call) == ("mom", "diffusion")
                own = same[:, bad]
                assert not bool(own.all()) if hit else bool(own.all()), (call, name, value)
                others = torch.cat([same[:, :bad], same[:, bad + 1:]], 1)
                assert bool(others.all()), (call, name, value, int((~others).sum()))
