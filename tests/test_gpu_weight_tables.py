"""The cache of Feldkamp weight tables gives up tables above its budget (512 MB),
but none that is still to be read: a batch and a graph captured by the caller
read theirs at every launch, long after other geometries have filled the cache."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402
from ct_b200 import _lib as L  # noqa: E402


def raw_images(V, H, W, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(2000, 65000, (V, H, W), generator=g, device="cuda", dtype=torch.int32).to(torch.uint16)


def fill_the_cache():
    """40 geometries of a 2048 x 2048 detector: 16.8 MB of weights each, more than the budget."""
    raw = raw_images(1, 2048, 2048, 1)
    out = torch.empty((1, 2048, 2048), device="cuda")
    for k in range(40):
        det, _ = ops.detector(2048, 2048, 5000.0 + 10.0 * k)
        ops.filter_projections(raw, det, L.HANN, 1, L.FP32, out=out)
    torch.cuda.synchronize()


def test_a_batch_keeps_its_weight_tables():
    scans = []
    for i, W in enumerate((256, 333)):
        det, grid = ops.detector(W, 64, 3.0 * W)
        grid = ops.custom_grid(det, (48, 48, 40), 2.0)
        X, Y, Z = grid.box
        scans.append(dict(raw=raw_images(20, 64, W, 2 + i), angles_deg=np.arange(20) * 18.0, heights_px=None, det=det,
                          grid=grid, filter=L.RAMLAK, pad=1, vol=torch.zeros((Z, Y, X), device="cuda")))
    batch = ops.Batch(scans, L.FP32)
    batch.run()
    torch.cuda.synchronize()
    before = [s["vol"].clone() for s in scans]
    fill_the_cache()
    for s in scans:
        s["vol"].zero_()
    batch.run()
    torch.cuda.synchronize()
    for s, b in zip(scans, before):
        assert float(b.norm()) > 0 and torch.equal(s["vol"], b)


def test_a_captured_graph_keeps_its_weight_table():
    det, _ = ops.detector(512, 96, 1500.0)
    raw = raw_images(12, 96, 512, 5)
    out = torch.empty((12, 96, 512), device="cuda")
    ops.filter_projections(raw, det, L.HANN, 1, L.FP32, out=out)   # builds the tables
    torch.cuda.synchronize()
    expect = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.filter_projections(raw, det, L.HANN, 1, L.FP32, out=out)
    fill_the_cache()
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, expect)
    # released with the graph: another round of geometries finds room again
    del graph
    fill_the_cache()
    free = torch.cuda.mem_get_info()[0]
    fill_the_cache()
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20
