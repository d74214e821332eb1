"""Which kernel a backprojection takes: rows on 16 bytes go to the shared-memory
kernel with and without scratch memory (ctb_backproject_noalloc), other rows are
copied by ctb_backproject and gathered by ctb_backproject_noalloc. The two kernels
round differently, so the volumes tell the route; both are the oracle's."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402
from ct_b200 import _lib as L  # noqa: E402

DT = {L.FP32: torch.float32, L.FP16: torch.float16, L.BF16: torch.bfloat16}


@pytest.mark.parametrize("store", [L.FP32, L.FP16, L.BF16])
@pytest.mark.parametrize("W,aligned", [(64, True), (61, False)])
def test_copied_rows_take_the_shared_memory_kernel(oracle, store, W, aligned):
    V, H, D = 20, 48, 200.0
    det, grid = ops.detector(W, H, D)
    X, Y, Z = grid.box
    rng = np.random.default_rng(W)
    proj = torch.from_numpy(rng.standard_normal((V, H, W)).astype(np.float32)).to(DT[store]).cuda()
    ang = np.sort(rng.uniform(0, 360, V))
    h = rng.uniform(-1.0, 1.0, V)
    out = []
    for name in ("ctb_backproject", "ctb_backproject_noalloc"):
        vol = torch.zeros((Z, Y, X), device="cuda")
        assert getattr(L.lib(), name)(ctypes.c_void_p(proj.data_ptr()), store, V, ang.ctypes.data, h.ctypes.data,
                                      ctypes.byref(det), ctypes.byref(grid), 0, Z, 1.0,
                                      ctypes.c_void_p(vol.data_ptr()), 0,
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == L.CTB_OK
        torch.cuda.synchronize()
        out.append(vol.cpu())
    assert torch.equal(*out) == aligned
    ref = oracle.ref_backproject(proj.float().cpu().numpy(), ang, h, oracle.ref_geom(W, H, D))
    for vol in out:
        d = vol.numpy().transpose(2, 1, 0).astype(np.float64) - ref
        assert np.linalg.norm(d) <= 1e-5 * np.linalg.norm(ref)   # the parity bar of a backprojection
