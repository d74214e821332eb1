"""Operator calls from two contexts of one device, in turn: the library keeps one
pool of device memory for the device, not another one at every switch."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# the driver API alone: every buffer belongs to the context that uses it
SCRIPT = r"""
import sys, ctypes as C
sys.path.insert(0, %r)
import numpy as np
from ct_b200 import _lib as L
cu = C.CDLL("libcuda.so.1")
def ck(r): assert r == 0, r
ck(cu.cuInit(0))
ctxs = []
p = C.c_void_p(); ck(cu.cuDevicePrimaryCtxRetain(C.byref(p), 0)); ctxs.append(p)
p = C.c_void_p(); ck(cu.cuCtxCreate_v2(C.byref(p), 0, 0)); ctxs.append(p)
det = L.Detector(64, 48, 200.0, 0.0, 1.0, 0.0); g = L.Grid()
L.check(L.lib().ctb_reference_grid(C.byref(det), None, C.byref(g)))
N, Z = 512, 160
grid = L.Grid(N, N, Z, 0, N, 0, N, 0, Z, 0.1)
ang = np.arange(2) * 90.0
n_vol, n_proj = 4 * N * N * Z, 4 * 2 * 64 * 48      # a volume of 168 MB: the call's scratch is its copy
bufs, outs, free = [], [], []
for c in ctxs:
    ck(cu.cuCtxSetCurrent(c))
    v, q = C.c_void_p(), C.c_void_p()
    ck(cu.cuMemAlloc_v2(C.byref(v), C.c_size_t(n_vol))); ck(cu.cuMemAlloc_v2(C.byref(q), C.c_size_t(n_proj)))
    ck(cu.cuMemsetD32_v2(v, 0x3f800000, C.c_size_t(n_vol // 4)))
    bufs.append((v, q))
for rep in range(8):
    for c, (v, q) in zip(ctxs, bufs):
        ck(cu.cuCtxSetCurrent(c))
        L.check(L.lib().ctb_forward_project(v, ang.ctypes.data, None, 2, C.byref(det), C.byref(grid), 0, Z, q, 0, None))
        ck(cu.cuCtxSynchronize())
        out = np.zeros((2, 48, 64), np.float32)
        ck(cu.cuMemcpyDtoH_v2(out.ctypes.data_as(C.c_void_p), q, C.c_size_t(n_proj)))
        outs.append(out)
    f, t = C.c_size_t(), C.c_size_t()
    ck(cu.cuMemGetInfo_v2(C.byref(f), C.byref(t)))
    free.append(f.value >> 20)
assert outs[0].sum() > 0 and all((o == outs[0]).all() for o in outs)
print("free MB", free)
assert free[0] - free[-1] < 64, free
"""


def test_switching_contexts_does_not_take_more_memory():
    r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]
