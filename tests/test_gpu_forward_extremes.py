"""The forward projector on volumes of values near the largest float: a pixel is
finite where its weighted values and their sum are, although the slices of a voxel
column summed before their weight would not be."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402


@pytest.mark.parametrize("slab", [(0, 200), (100, 103)])   # windows of slices, slabs thinner than one
@pytest.mark.parametrize("top", [1.0e32, 3.0e38])
def test_values_near_the_largest_float(slab, top):
    """Against the same volume scaled down by 2^40, an exact step, whose sums are far
    from the limits: within 308 x 2^-24 (terms of a pixel and roundings of a weight,
    as in the element-wise comparison) where the scaled-up value is a float. One
    voxel column of large values, so that a pixel sees its weighted sum alone."""
    W, H, V = 24, 40, 60
    det, _ = ops.detector(W, H, 200.0, u_offset=0.3)
    grid = ops.custom_grid(det, (16, 16, 200), 0.2)
    z0, z1 = slab
    vol = torch.zeros((z1 - z0, 16, 16), device="cuda")
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    vol[:, 8, 3] = top * (0.5 + 0.5 * torch.rand(z1 - z0, generator=g, device="cuda"))
    ang = np.arange(V) * (360.0 / V)
    out = ops.forward_project(vol, ang, None, det, grid, z0, z1).double()
    ref = ops.forward_project(vol * 2.0 ** -40, ang, None, det, grid, z0, z1).double() * 2.0 ** 40
    assert float(ref.max()) > top
    fits = ref < 3.4e38
    assert bool(torch.isfinite(out[fits]).all())
    assert bool(((out - ref).abs()[fits] <= 308 * 2.0 ** -24 * ref[fits]).all())
    assert not bool(torch.isfinite(out[ref > 3.41e38]).any())
