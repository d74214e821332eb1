"""The register filter takes four detector rows at a time. The views of low detectors
of 4 k + 2 rows are filtered two at a time, so a group may hold rows of two views: the
result is that of each view by itself, bit for bit (pairs of rows, which share a
transform, never cross a view), with an odd number of views too."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402
from ct_b200 import _lib as L  # noqa: E402


@pytest.mark.parametrize("W", [256, 300, 1024])   # whole rows, embedded ones, one group per CTA and several
@pytest.mark.parametrize("H,V", [(2, 1), (2, 2), (2, 7), (2, 8), (2, 8197), (3, 7), (4, 7), (6, 8), (6, 2733), (62, 265),
                                 (66, 4)])
def test_views_together_are_the_views_one_by_one(W, H, V):
    det, _ = ops.detector(W, H, 1.5 * W)   # (weights that differ from row to row)
    g = torch.Generator(device="cuda")
    g.manual_seed(W + H + V)
    raw = torch.randint(1000, 65000, (V, H, W), generator=g, device="cuda", dtype=torch.int32).to(torch.uint16)
    buf = torch.full((V * H * W + 2 * W,), -7.0, device="cuda")
    out = buf[W:-W].view(V, H, W)
    ops.filter_projections(raw, det, L.HANN, 1, L.FP32, out=out)
    for v in list(range(min(V, 8))) + list(range(max(8, V - 4), V)):
        one = ops.filter_projections(raw[v:v + 1], det, L.HANN, 1, L.FP32)
        assert torch.equal(out[v], one[0]), v
    assert bool((buf[:W] == -7.0).all()) and bool((buf[-W:] == -7.0).all())
