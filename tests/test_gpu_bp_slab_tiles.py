"""Slabs whose ends cut a tile of the shared-memory backprojector: tiles summed whole
(slices past the slab dropped) and group by group, of 32 and of 16 slices, against
the same slices of the whole box. A slice's row decisions and operations are the
same in every tile, only the order of the views differs: 2e-6 rel-L2, the bar of
the kernels' own comparison. Slices off the slab must stay as they are."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402

SLABS = [(0, 17), (0, 24), (0, 25), (0, 31), (0, 33), (0, 41), (0, 49), (0, 57), (16, 48), (16, 36), (8, 32), (24, 56),
         (20, 52), (5, 69), (30, 50), (95, 96), (7, 96)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("vs,D", [(1.3, 600.0), (4.0, 2500.0)])   # boxes of three CTAs an SM, and of one (FP32)
def test_slabs_match_the_whole_box(dtype, vs, D):
    W, H, V = 256, 160, 23
    det, _ = ops.detector(W, H, D, u_offset=0.7)
    grid = ops.custom_grid(det, (40, 37, 96), vs)
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    proj = torch.randn((V, H, W), generator=g, device="cuda").to(dtype)
    ang = np.arange(V) * (360.0 / V) + 1.0
    h = np.random.default_rng(4).uniform(-1.5, 1.5, V)
    whole = ops.backproject(proj, ang, h, det, grid)
    assert float(whole.norm()) > 0
    for z0, z1 in SLABS:
        buf = torch.full((z1 - z0 + 2, 37, 40), -7.0, device="cuda")
        ops.backproject(proj, ang, h, det, grid, z0, z1, out=buf[1:-1])
        ref = whole[z0:z1].double()
        assert float((buf[1:-1].double() - ref).norm()) <= 2e-6 * float(ref.norm()), (z0, z1)
        assert bool((buf[0] == -7.0).all()) and bool((buf[-1] == -7.0).all()), (z0, z1)
