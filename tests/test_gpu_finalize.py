"""msod_finalize gives every library-owned buffer back, and the library then starts anew.

What the library keeps between calls belongs to the context it was made in.  After msod_finalize a host
may destroy that context and go on in another one, as a coupled code does that owns its contexts.  Each
test is a process of its own, on contexts of its own (driver API), without torch."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r'''
import ctypes as C
import numpy as np
from minisod2d_gb300 import capi, workload

cu = C.CDLL("libcuda.so.1")

def drv(name, *a):
    rc = getattr(cu, name)(*a)
    assert rc == 0, (name, rc)

def context():
    ctx = C.c_void_p()
    drv("cuCtxCreate_v2", C.byref(ctx), C.c_uint(0), C.c_int(0))
    return ctx

held = []

def buf(nbytes, src=None):
    p = C.c_void_p()
    capi.call("msod_malloc", C.byref(p), nbytes)
    held.append(p)
    if src is not None:
        src = np.ascontiguousarray(src)
        capi.call("msod_h2d", p, src.ctypes.data_as(C.c_void_p), src.nbytes, None)
        capi.call("msod_stream_synchronize", None)
    return p

def calls(P, nx):
    """Convection, diffusion and entropy viscosity of a small mesh: their results as one list."""
    host = workload.HostCase(workload.custom(P, nx, 0.05, seed=2))
    t, f, n, ne, npn = host.tables, host.fields, host.cfg.nnode, host.nelem, host.npoin
    up = lambda a: buf(a.nbytes, a)
    con, He, gp = up(host.connec), buf(36 * ne * n), buf(4 * ne * n)
    capi.call("msod_elem_jacobian", P, ne, npn, con, up(host.coord), up(t["dNgp"]), up(t["wgp"]), gp, He, None)
    geo = [con, He, gp] + [up(t[k]) for k in ("dlxigp_ip", "invAtoIJK", "AtoI", "AtoJ", "AtoK")]
    g = [P, ne, npn, con, None, None, He, gp, geo[3], None, *geo[4:]]
    d = {k: up(v) for k, v in f.items()}
    mu = up(np.full(ne * n, 1e-3, np.float32))
    R = [buf(4 * k * npn) for k in (1, 3, 1)]
    nu = buf(4 * ne)
    out = []

    def get(p, count):
        a = np.empty(count, np.float32)
        capi.call("msod_d2h", a.ctypes.data_as(C.c_void_p), p, a.nbytes, None)
        capi.call("msod_stream_synchronize", None)
        out.append(a)

    capi.call("msod_convec_ijk", *g, d["u"], d["q"], d["rho"], d["pr"], d["E"], *R, None)
    for p, k in zip(R, (1, 3, 1)):
        get(p, k * npn)
    capi.call("msod_diffusion_ijk", *g, 1004.5, 0.71, d["rho"], d["u"], d["Tem"], d["mu_fluid"], mu, mu, *R, None)
    for p, k in zip(R, (1, 3, 1)):
        get(p, k * npn)
    capi.call("msod_entropy_viscosity", P, ne, npn, *geo, d["rho"], d["u"], d["pr"], 1.4, 0.1, 0.5, 1, None, nu, None, None)
    get(nu, ne)
    while held:
        capi.call("msod_free", held.pop())
    return out

drv("cuInit", C.c_uint(0))
'''


def _child(code):
    r = subprocess.run([sys.executable, "-c", CHILD + code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


def test_library_starts_again_in_another_context(msod_lib):
    """The same results from a context made after msod_finalize and the end of the first one."""
    _child(r'''
for P, nx in ((1, 9), (4, 5), (7, 3)):
    res = []
    for k in range(2):
        ctx = context()
        res.append(calls(P, nx))
        capi.call("msod_finalize")
        drv("cuCtxDestroy_v2", ctx)
    for a, b in zip(*res):
        assert np.isfinite(a).all() and np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(a), P
''')


def test_finalize_keeps_the_callers_context(msod_lib):
    _child(r'''
ctx, now = context(), C.c_void_p()
calls(4, 3)
capi.call("msod_finalize")
drv("cuCtxGetCurrent", C.byref(now))
assert now.value == ctx.value
''')
