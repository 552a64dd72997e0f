"""The FP64 diffusion (one thread per point) against the FP64 oracle, at every order.

Element counts around a block's (1, 2, 4, 7 and 32 elements) that leave the last block partly empty;
tables whose directions differ; a connec entry that names no node.  Tolerance: the FP64 criterion of
tests/test_gpu_parity.py."""
import numpy as np
import pytest

from minisod2d_gb300 import fem, kernels
from oracle import oracle as O
from tests.test_gpu_groups import _tables
from tests.test_gpu_parity import NTH, TOL64, _compare

pytestmark = pytest.mark.gpu


def _case(P, dims, odd):
    t32, t = _tables(P, odd), fem.element_tables(P, np.float64)
    t["dlxigp_ip"] = t32["dlxigp_ip"].astype(np.float64)
    connec, coord, ne, npn = fem.structured_mesh(P, *dims, t32, 0.1, P)
    He, gp = O.elem_jacobian(P, ne, npn, connec, coord.astype(np.float64), t["dNgp"], t["wgp"], np.float64)
    rng = np.random.default_rng(P)
    f = {k: 1.0 + 0.3 * rng.random(npn) for k in ("rho", "Tem", "mu_fluid")}
    f["u"] = rng.standard_normal(3 * npn)
    mu = [rng.random(ne * (P + 1) ** 3) for _ in range(2)]
    return t, connec, He, gp, f, mu, ne, npn


def _run(cuda, t, connec, He, gp, f, mu, ne, npn):
    import torch

    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    out = [torch.full((k * npn,), 7.0, dtype=torch.float64, device=cuda) for k in (1, 3, 1)]
    kernels.full_diffusion_ijk(ne, npn, up(connec), None, None, up(He), up(gp), up(t["dlxigp_ip"]), None,
                               *[up(t[k]) for k in ("invAtoIJK", "AtoI", "AtoJ", "AtoK")], 1004.5, 0.71, up(f["rho"]),
                               up(f["u"]), up(f["Tem"]), up(f["mu_fluid"]), *[up(m) for m in mu], *out)
    return [x.cpu().numpy() for x in out]


@pytest.mark.parametrize("P,dims", [(1, (31, 1, 1)), (1, (11, 3, 1)), (2, (1, 1, 1)), (2, (4, 2, 1)), (3, (5, 1, 1)),
                                    (4, (1, 1, 1)), (4, (3, 1, 1)), (5, (2, 2, 1)), (6, (3, 1, 1)), (7, (1, 1, 1)),
                                    (7, (2, 1, 1)), (8, (2, 1, 1))])
@pytest.mark.parametrize("odd", [False, True])
def test_against_the_oracle(cuda, P, dims, odd):
    t, connec, He, gp, f, mu, ne, npn = _case(P, dims, odd)
    ref = O.full_diffusion_ijk(P, ne, npn, dict(t, connec=connec, He=He, gpvol=gp), 1004.5, 0.71, f["rho"], f["u"],
                               f["Tem"], f["mu_fluid"], *mu, np.float64, nthreads=NTH)
    _compare(_run(cuda, t, connec, He, gp, f, mu, ne, npn), ref, TOL64, "diffu64 P=%d" % P)


@pytest.mark.parametrize("P", [1, 4, 7, 8])
def test_missing_node(cuda, P):
    """An entry outside 1..npoin reads as a node of zeros and is not assembled: the residuals of the
    mesh in which such a node exists."""
    t, connec, He, gp, f, mu, ne, npn = _case(P, (2, 1, 1), True)
    at = (5 * ne + 1, 2 * ne)  # (a * nelem + e)
    bad, more = connec.copy(), connec.copy()
    bad[list(at)] = (0, npn + 7)
    more[list(at)] = npn + 1
    g = {k: np.concatenate([np.append(x, 0.0) for x in v.reshape(-1, npn)]) for k, v in f.items()}
    a = _run(cuda, t, bad, He, gp, f, mu, ne, npn)
    b = _run(cuda, t, more, He, gp, g, mu, ne, npn + 1)
    for k, x, y in zip((1, 3, 1), a, b):
        y = y.reshape(k, npn + 1)[:, :npn].reshape(-1)
        assert np.linalg.norm(x - y) <= TOL64 * np.linalg.norm(y)
