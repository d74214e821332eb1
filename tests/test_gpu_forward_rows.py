"""The forward projector where its row windows can go wrong: row blocks of 128 and
pairs of 64 at their edges, windows of one to many slices (K = floor(2 / dv) + 1,
unrolled up to 4), slabs thinner than a window, rows the detector's bounds cut,
strips of four columns at odd widths, and volumes with infinities."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402

# W, H, (X, Y, Z), voxel pitch, slab, height offsets
CASES = [
    (7, 63, (5, 4, 40), 1.7, None, False),       # K = 1 and 2, 63 rows
    (8, 64, (6, 5, 30), 2.6, None, True),        # K = 1
    (9, 65, (6, 6, 90), 0.75, None, False),      # K = 3
    (17, 129, (8, 9, 100), 1.4, None, True),     # a second row block of one row, rows cut at both ends
    (16, 128, (9, 8, 260), 0.55, (3, 257), False),   # K = 4
    (5, 131, (4, 4, 400), 0.31, (5, 390), True),     # K of 6 or 7
    (12, 70, (7, 7, 60), 0.9, (20, 22), False),  # slabs thinner than a window
    (12, 70, (7, 7, 60), 0.9, (31, 32), True),
]


def setup(case):
    W, H, size, vs, slab, heights = case
    rng = np.random.default_rng(W * H)
    det, _ = ops.detector(W, H, 6.0 * max(W, 20), u_offset=0.4)
    grid = ops.custom_grid(det, size, vs)
    V = 3
    ang = rng.uniform(0, 360, V)
    h = rng.uniform(-2, 2, V) if heights else np.zeros(V)
    z0, z1 = slab or (0, size[2])
    return det, grid, ang, h, z0, z1, (V, H, W), (z1 - z0, size[1], size[0]), rng


@pytest.mark.parametrize("case", CASES)
def test_rows_match_the_backprojector_element_by_element(case):
    """A x against the sum over the backprojector's matrix in float64: A^T e for every
    pixel e. Each weight is the same to a few roundings, a pixel sums under 300
    terms: within (300 + 8) 2^-24 of the sum of |weight x|."""
    det, grid, ang, h, z0, z1, pshape, vshape, rng = setup(case)
    x = torch.from_numpy(rng.standard_normal(vshape).astype(np.float32)).cuda()
    Ax = ops.forward_project(x, ang, h, det, grid, z0, z1).double()
    e = torch.zeros(pshape, device="cuda")
    xd = x.double()
    ref = torch.zeros(int(np.prod(pshape)), dtype=torch.float64, device="cuda")
    mag = torch.zeros_like(ref)
    used = torch.zeros(vshape, dtype=torch.bool, device="cuda")
    for k in range(ref.numel()):
        e.view(-1)[k] = 1.0
        row = ops.backproject(e, ang, h, det, grid, z0, z1).double()
        e.view(-1)[k] = 0.0
        assert int((row != 0).sum()) < 300
        used |= row != 0
        ref[k] = (row * xd).sum()
        mag[k] = (row * xd).abs().sum()
    assert int(used.sum()) > 0
    assert bool(((Ax.view(-1) - ref).abs() <= 308 * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("case", [CASES[0], CASES[3], CASES[6]])
def test_infinities_stay_on_the_rows_they_touch(case):
    """One infinite voxel: every pixel it does not reach keeps the value it has with
    the voxel at zero, every pixel with a weight for it is infinite or NaN."""
    det, grid, ang, h, z0, z1, pshape, vshape, rng = setup(case)
    x = torch.from_numpy(rng.standard_normal(vshape).astype(np.float32)).cuda()
    at = (vshape[0] // 2, vshape[1] // 2, vshape[2] // 2)
    unit = torch.zeros_like(x)
    unit[at] = 1.0
    touched = ops.forward_project(unit, ang, h, det, grid, z0, z1) != 0
    assert bool(touched.any())
    x[at] = 0.0
    without = ops.forward_project(x, ang, h, det, grid, z0, z1)
    x[at] = float("inf")
    with_inf = ops.forward_project(x, ang, h, det, grid, z0, z1)
    assert not bool(torch.isfinite(with_inf[touched]).any())
    # a weight of exactly zero may still make a NaN on the row next to the voxel's own
    finite = torch.isfinite(with_inf)
    assert int((~finite).sum()) <= int(touched.sum()) + 8
    tol = 308 * 2.0 ** -24 * float(without.abs().max()) * 4
    assert float((with_inf - without)[finite].abs().max()) <= tol
