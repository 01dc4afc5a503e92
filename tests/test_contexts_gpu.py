"""The C ABI in CUDA contexts that a host makes and destroys one after the other
(their handles are given again): ungridding, whose kernels need their shared-memory
limit set in each, and gridding in the library's fixed buffer, which lies elsewhere
in each. In a child process, without torch's context."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r'''
import ctypes, sys
import numpy as np
from torchlinops_gb300 import _ext, interp
cu = ctypes.CDLL("libcuda.so.1")
P, ck = ctypes.c_void_p, lambda r: (_ for _ in ()).throw(RuntimeError(str(r))) if r else None
L = _ext.lib()
rng = np.random.default_rng(0)
n, npts, nb = (24, 20, 28), 3000, 2
locs = (rng.random((npts, 3)) * n).astype(np.float32)
img = rng.standard_normal((nb, *n, 2)).astype(np.float32)
vals = rng.standard_normal((nb, npts, 2)).astype(np.float32)
desc = lambda b: interp._desc(3, n, (4.0,) * 3, "kaiser_bessel", 1, "circular", 7.0, True, b, npts)
ck(cu.cuInit(0))
results, handles = [], set()
for _ in range(4):
    ctx = P()
    ck(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0))
    handles.add(ctx.value)

    def alloc(nbytes):
        p = P()
        ck(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(max(nbytes, 16))))
        return p

    def up(a):
        p = alloc(a.nbytes)
        ck(cu.cuMemcpyHtoD_v2(p, a.ctypes.data_as(P), ctypes.c_size_t(a.nbytes)))
        return p

    pad = alloc(1 << 20)  # another layout of the context's memory each time
    pb, tb = ctypes.c_size_t(0), ctypes.c_size_t(0)
    d = desc(nb)
    assert L.tlgb_interp_plan_size(ctypes.byref(d), ctypes.byref(pb), ctypes.byref(tb)) == 0
    plan, tmp, dl, dv, di = alloc(pb.value), alloc(tb.value), up(locs), up(vals), up(img)
    info = _ext.PlanInfo()
    assert L.tlgb_interp_plan_build(ctypes.byref(d), dl, plan, pb, tmp, tb, ctypes.byref(info), None) == 0, L.tlgb_last_error()
    out, grid = alloc(vals.nbytes), alloc(img.nbytes)
    assert L.tlgb_interp_forward(ctypes.byref(d), ctypes.byref(info), plan, dl, di, out, None) == 0, L.tlgb_last_error()
    assert L.tlgb_interp_adjoint_fixed(ctypes.byref(d), ctypes.byref(info), plan, dl, dv, grid, None) == 0, L.tlgb_last_error()
    y, g = np.empty_like(vals), np.empty_like(img)
    ck(cu.cuMemcpyDtoH_v2(y.ctypes.data_as(P), out, ctypes.c_size_t(y.nbytes)))
    ck(cu.cuMemcpyDtoH_v2(g.ctypes.data_as(P), grid, ctypes.c_size_t(g.nbytes)))
    results.append((y, g))
    ck(cu.cuCtxDestroy_v2(ctx))
assert all(np.array_equal(r[0], results[0][0]) and np.array_equal(r[1], results[0][1]) for r in results)
assert np.abs(results[0][0]).max() > 0 and np.abs(results[0][1]).max() > 0
inner = [(results[0][0].astype(np.float64) * vals).sum(), (img.astype(np.float64) * results[0][1]).sum()]
assert abs(inner[0] - inner[1]) < 1e-4 * (np.abs(results[0][0]) * np.abs(vals)).sum()  # adjoint
print("handles", len(handles), "of", len(results))
'''


def test_contexts_made_one_after_the_other():
    pkg = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torch-named-linops_gb300")
    r = subprocess.run([sys.executable, "-c", CHILD], env=dict(os.environ, PYTHONPATH=pkg), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
