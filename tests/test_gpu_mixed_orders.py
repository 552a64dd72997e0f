"""Tensor-core residuals at the orders whose tiles are far from 8 x 8 lines, on meshes with more
elements than resident blocks (each block goes on to further elements with the node ids it loaded
ahead) and not a multiple of them.  Reference and bounds as in tests/test_gpu_mixed.py."""
import pytest

from tests import test_gpu_mixed as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,nx", [(1, 19), (2, 15), (3, 11), (6, 9)])
def test_mixed_orders(cuda, P, nx):
    host, dev = M._diffu_case(cuda, P, nx, 0, 8)
    conv, diff = M._oracle64(host, dev), M._diffu_oracle64(host, dev)
    floor = M._errs(dev.diffu(), diff)
    for prec in ("fp16", "bf16"):
        for e in M._errs(dev.convec_mixed(prec), conv):
            assert e <= (M.TOL_FP16 if prec == "fp16" else M.TOL), (prec, e)
        for e, fl in zip(M._errs(dev.diffu_mixed(prec), diff), floor):
            assert e <= (M.TOL if prec == "fp16" else max(M.BF16_DIFFU_TOL, M.DIFFU_FLOOR_FACTOR * fl)), (prec, e, fl)
