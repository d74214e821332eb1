"""The bounds-checked build on the forward projector: no voxel is read outside the
copy of the slab, at the edges of its row blocks and windows, on thin slabs, rows
the detector cuts, height offsets, and in volumes with infinities; and the
projections are those of the normal library. Each library runs in a child process."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys, json, ctypes, numpy as np, torch
sys.path.insert(0, %r)
from ct_b200 import ops
from ct_b200 import _lib as L
chk, n, first = ctypes.c_int(), ctypes.c_uint(), ctypes.c_ulonglong()
def status():
    assert L.lib().ctb_diag_bounds_status(0, ctypes.byref(chk), ctypes.byref(n), ctypes.byref(first), 1) == 0
    return [chk.value, n.value, first.value]
status()
report = {}
for i, (W, H, size, vs, slab, hmax, inf) in enumerate(json.loads(sys.argv[1])):
    rng = np.random.default_rng(i)
    det, _ = ops.detector(W, H, 6.0 * max(W, 20), u_offset=0.4)
    grid = ops.custom_grid(det, tuple(size), vs)
    z0, z1 = slab
    x = torch.from_numpy(rng.standard_normal((z1 - z0, size[1], size[0])).astype(np.float32)).cuda()
    if inf:
        x[(z1 - z0) // 2, size[1] // 2, size[0] // 2] = float("inf")
    p = ops.forward_project(x, np.sort(rng.uniform(0, 360, 12)), rng.uniform(-1, 1, 12) * hmax, det, grid, z0, z1)
    torch.cuda.synchronize()
    report[i] = status()
    np.save(sys.argv[2] + "_%%d.npy" %% i, p.cpu().numpy())
print(json.dumps(report))
"""

# W, H, volume, voxel pitch, slab, largest height offset, an infinite voxel
CASES = [
    [30, 129, [24, 20, 90], 1.4, [0, 90], 2.0, False],
    [30, 129, [24, 20, 90], 1.4, [0, 90], 2.0, True],
    [17, 40, [16, 16, 300], 0.21, [0, 300], 0.0, False],
    [17, 40, [16, 16, 300], 0.21, [120, 122], 0.0, True],
    [24, 20, [20, 21, 64], 0.9, [30, 31], 1.0, False],
    [24, 200, [20, 21, 30], 2.7, [3, 30], 90.0, False],    # volume off the detector in some views
    [24, 64, [12, 12, 16], 0.5, [0, 16], 40.0, True],
    [64, 64, [40, 30, 64], 1.0, [60, 64], 0.0, False],
]


def run(tmp_path, library):
    prefix = str(tmp_path / library)
    r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT, json.dumps(CASES), prefix],
                       env=dict(os.environ, CTB_LIBRARY=library), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1]), [np.load(prefix + f"_{i}.npy") for i in range(len(CASES))]


def test_no_voxel_outside_the_slab(tmp_path):
    rep_c, p_c = run(tmp_path, "checked")
    rep_n, p_n = run(tmp_path, "normal")
    for i in range(len(CASES)):
        assert rep_c[str(i)] == [1, 0, 0], (CASES[i], rep_c[str(i)])
        assert rep_n[str(i)] == [0, 0, 0]
        assert np.array_equal(p_c[i], p_n[i], equal_nan=True), CASES[i]
    assert all(np.abs(p[np.isfinite(p)]).max() > 0 for p in p_n)
