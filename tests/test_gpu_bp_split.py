"""Backprojection launches whose views are split among the CTAs of a cluster
(grids of few tiles), and tiles that reach past their slab: against the same
views added one at a time, which is never split, at the edges of tiles (16
columns, 8 / 16 / 32 slices), of the view counts that allow 2, 4 and 8 CTAs per
tile, and of slabs off a tile boundary."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402

CASES = [
    # X, Y, Z, views, slab, voxel pitch, storage
    (15, 16, 8, 8, None, 1.0, torch.float32),        # one tile, two CTAs
    (16, 17, 9, 15, None, 1.0, torch.float16),
    (17, 33, 31, 16, None, 1.2, torch.bfloat16),     # four CTAs, a tile one slice short
    (33, 15, 33, 31, None, 0.9, torch.float32),      # a second tile of one slice
    (40, 40, 64, 64, None, 1.5, torch.float16),      # eight CTAs, rows cut at both ends
    (40, 24, 70, 65, (5, 69), 1.0, torch.float32),   # a slab off the tiles at both ends
    (24, 40, 70, 100, (33, 34), 1.0, torch.float16),
    (24, 40, 70, 7, (31, 65), 1.0, torch.float32),   # too few views to split
    (100, 90, 20, 40, (2, 19), 0.6, torch.float32),
    (33, 31, 17, 200, None, 2.5, torch.float32),     # wide boxes
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("accumulate", [False, True])
def test_split_views_match_views_added_one_by_one(case, accumulate):
    """Both sum the same V samples per voxel in FP32 in different orders: within
    2 V 2^-24 of the sum of their magnitudes (bounded by the backprojection of the
    absolute values: every weight is positive)."""
    X, Y, Z, V, slab, vs, dt = case
    W, H = 64, 48
    rng = np.random.default_rng(X * Y + V)
    det, _ = ops.detector(W, H, 250.0, u_offset=0.7)
    grid = ops.custom_grid(det, (X, Y, Z), vs)
    z0, z1 = slab or (0, Z)
    ang = np.sort(rng.uniform(0, 360, V))
    h = rng.uniform(-2, 2, V)
    p = torch.from_numpy(rng.standard_normal((V, H, W)).astype(np.float32)).cuda().to(dt)
    start = torch.full((z1 - z0, Y, X), 0.5 if accumulate else float("nan"), device="cuda")
    out = ops.backproject(p, ang, h, det, grid, z0, z1, out=start.clone(), accumulate=accumulate)
    ref = start.clone()
    mag = torch.zeros_like(start)
    for v in range(V):
        one = p[v:v + 1].contiguous()
        ops.backproject(one, ang[v:v + 1], h[v:v + 1], det, grid, z0, z1, out=ref, accumulate=accumulate or v > 0)
        ops.backproject(one.abs(), ang[v:v + 1], h[v:v + 1], det, grid, z0, z1, out=mag, accumulate=v > 0)
    assert float(mag.abs().max()) > 0
    tol = 2 * (V + 1) * 2.0 ** -24 * (mag.double() + (0.5 if accumulate else 0.0))
    assert bool(((out.double() - ref.double()).abs() <= tol + 1e-30).all())
    again = ops.backproject(p, ang, h, det, grid, z0, z1, out=start.clone(), accumulate=accumulate)
    assert torch.equal(out, again)   # the same sums in the same order every time
