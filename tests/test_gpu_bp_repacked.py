"""Backprojection from rows the TMA loads cannot take (pitch or base off 16
bytes), which are copied to padded rows first, against the gather kernel on the
same rows (ctb_backproject_noalloc, which may not copy): odd widths of every
storage type, bases one to seven samples past an aligned one, slabs that reach
a band of rows, accumulation, and more views than one run of the copy holds."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402
from ct_b200 import _lib as L  # noqa: E402

DT = {L.FP32: torch.float32, L.FP16: torch.float16, L.BF16: torch.bfloat16}


def both(W, H, V, size, vs, store, slab=None, shift=0, accumulate=0, uoff=0.0, hmax=0.0, D=None):
    rng = np.random.default_rng(W + H + V)
    det, _ = ops.detector(W, H, D or 3.0 * max(W, H), u_offset=uoff)
    grid = ops.custom_grid(det, size, vs)
    X, Y, Z = grid.box
    z0, z1 = slab or (0, Z)
    g = torch.Generator(device="cuda")
    g.manual_seed(W * H)
    flat = torch.randn(V * H * W + shift, generator=g, device="cuda", dtype=torch.float32).to(DT[store])
    proj = flat[shift:]   # nothing of the test's own follows the last sample
    ang = np.sort(rng.uniform(0, 360, V))
    h = rng.uniform(-hmax, hmax, V)
    out = []
    for name in ("ctb_backproject", "ctb_backproject_noalloc"):
        vol = torch.full((z1 - z0, Y, X), 0.25, device="cuda")
        st = getattr(L.lib(), name)(ctypes.c_void_p(proj.data_ptr()), store, V, ang.ctypes.data, h.ctypes.data,
                                    ctypes.byref(det), ctypes.byref(grid), z0, z1, 1.0,
                                    ctypes.c_void_p(vol.data_ptr()), accumulate,
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == L.CTB_OK
        torch.cuda.synchronize()
        out.append(vol.double())
    return out


@pytest.mark.parametrize("store", [L.FP32, L.FP16, L.BF16])
@pytest.mark.parametrize("case", [
    dict(W=33, H=20, V=9, size=(20, 22, 16), vs=1.0),
    dict(W=39, H=31, V=11, size=(33, 17, 40), vs=0.8, uoff=1.5, hmax=2.0),
    dict(W=41, H=64, V=8, size=(30, 30, 64), vs=1.1, slab=(50, 61), hmax=1.0),
    dict(W=46, H=24, V=10, size=(24, 24, 24), vs=1.4, accumulate=1),
    dict(W=40, H=24, V=10, size=(24, 24, 24), vs=1.4, shift=1),   # an aligned pitch at an odd base
    dict(W=47, H=24, V=10, size=(24, 24, 24), vs=1.4, shift=3),
])
def test_copied_rows_match_gathered_rows(case, store):
    """The two kernels take the same row and column decisions and differ in the
    rounding of a sample's interpolation: 2e-6 rel-L2, the bar of the two kernels'
    own comparison."""
    a, b = both(store=store, **case)
    assert float(b.norm()) > 0
    assert float((a - b).norm() / b.norm()) < 2e-6


def test_more_views_than_one_run_of_the_copy():
    a, b = both(W=701, H=401, V=280, size=(80, 80, 48), vs=1.5, store=L.FP32)   # 315 MB in runs of 256 MB
    assert float((a - b).norm() / b.norm()) < 2e-6
