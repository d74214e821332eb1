"""Views read through global memory from a stack that holds only the detector
rows a slab reaches: the copied rows of widths the TMA loads cannot take, and
the row band the facade keeps of a z sub-box. A tile reaches past such a slab by
up to 31 slices, whose rows the stack does not hold; the bounds-checked build
counts every fetch outside the rows held, and there must be none. The volumes
are those of the gather kernel (ctb_backproject_noalloc) and of the staged boxes.

Each library is loaded in a child process of its own."""
import json
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys, json, ctypes, numpy as np, torch
sys.path.insert(0, %r)
from ct_b200 import CtVolume, ops
from ct_b200 import _lib as L
lib = L.lib()
chk, n, first = ctypes.c_int(), ctypes.c_uint(), ctypes.c_ulonglong()
DT = {"fp32": (L.FP32, torch.float32), "fp16": (L.FP16, torch.float16), "bf16": (L.BF16, torch.bfloat16)}

def status():
    assert lib.ctb_diag_bounds_status(0, ctypes.byref(chk), ctypes.byref(n), ctypes.byref(first), 1) == 0
    return {"checked": chk.value, "violations": n.value, "first": first.value}

def diff(a, b):
    assert float(b.norm()) > 0
    return float((a - b).norm() / b.norm())

def operator(c):
    rng = np.random.default_rng(c["W"] + c["V"])
    det, _ = ops.detector(c["W"], c["H"], c["D"], u_offset=c.get("uoff", 0.0))
    grid = ops.custom_grid(det, tuple(c["size"]), c["vs"])
    X, Y, Z = grid.box
    z0, z1 = c["slab"]
    store, dt = DT[c["store"]]
    proj = torch.from_numpy(rng.standard_normal((c["V"], c["H"], c["W"])).astype(np.float32)).to(dt).cuda()
    ang = np.sort(rng.uniform(0, 360, c["V"]))
    h = rng.uniform(-1.0, 1.0, c["V"]) * c.get("hmax", 0.0)
    out = []
    for name in ("ctb_backproject", "ctb_backproject_noalloc"):
        vol = torch.full((z1 - z0, Y, X), 0.25, device="cuda")
        assert getattr(lib, name)(ctypes.c_void_p(proj.data_ptr()), store, c["V"], ang.ctypes.data, h.ctypes.data,
                                  ctypes.byref(det), ctypes.byref(grid), z0, z1, 1.0,
                                  ctypes.c_void_p(vol.data_ptr()), 0,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == L.CTB_OK
        torch.cuda.synchronize()
        out.append(vol.double())
    return diff(*out)

def facade(c):
    rng = np.random.default_rng(c["W"])
    img = rng.integers(20000, 65535, (c["V"], c["H"], c["W"])).astype(np.uint16)
    v = CtVolume()
    v.setProjectionsPointer(img.ctypes.data, L.U16, c["V"], c["W"], c["H"], np.arange(c["V"]) * (360.0 / c["V"]),
                            pixel_size=0.5, fcd_mm=0.5 * c["D"], keep=img)
    v.setPrecision(c["store"])
    v.setVolumeBounds(0.0, 1.0, 0.0, 1.0, *c["z"])
    if c["slab"]:
        L.check(lib.ctb_set_slab_height(v._ctx, c["slab"]), v._ctx)
    x, y, z = v.grid().box
    out = []
    for every in (1, 0):
        lib.ctb_diag_force_overflow(every)
        vol = np.zeros((z, y, x), np.float32)
        v.reconstructInto(vol.ctypes.data, L.X_FASTEST)
        out.append(torch.from_numpy(vol).double())
    return diff(*out)

status()
report = {}
for name, c in json.loads(sys.argv[1]).items():
    lib.ctb_diag_force_overflow(c.get("every", 1))
    d = (facade if c["op"] == "facade" else operator)(c)
    lib.ctb_diag_force_overflow(0)
    report[name] = dict(status(), diff=d)
print(json.dumps(report))
"""

OP = dict(op="operator", W=41, H=64, D=192.0, V=9, size=[30, 30, 64], vs=1.1)
CASES = {
    # one slice near the start of a tile (rows 27 .. 35 held, the tile's last slice at row 23),
    # one at its end, slabs at both ends of the box, one across two tiles of 32
    "one_slice": dict(OP, store="fp32", slab=[33, 34]),
    "one_slice_split": dict(OP, store="fp16", slab=[33, 34], V=40),
    "tile_end": dict(OP, store="bf16", slab=[31, 32]),
    "first_slices": dict(OP, store="fp32", slab=[0, 3], hmax=1.0),
    "last_slices": dict(OP, store="fp16", slab=[50, 64], hmax=1.0, uoff=1.5),
    "two_tiles": dict(OP, store="bf16", slab=[30, 51], V=24),
    "some_views": dict(OP, store="fp32", slab=[40, 45], every=2),
    "facade_middle": dict(op="facade", W=64, H=96, D=200.0, V=30, z=[0.4, 0.55], slab=0, store="fp32"),
    "facade_slabs": dict(op="facade", W=56, H=96, D=200.0, V=30, z=[0.3, 0.6], slab=5, store="fp16"),
}


@pytest.mark.parametrize("library", ["checked", "normal"])
def test_global_reads_stay_in_the_rows_held(library):
    """2e-6 rel-L2: the bar of the kernels' own comparison (the same row and column
    decisions, other roundings)."""
    env = dict(os.environ, CTB_LIBRARY=library)
    r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT, json.dumps(CASES)], env=env, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    report = json.loads(r.stdout.strip().splitlines()[-1])
    for k in CASES:
        assert report[k]["checked"] == (library == "checked")
        assert report[k]["violations"] == 0, (k, report[k])
        assert report[k]["diff"] < 2e-6, (k, report[k])
