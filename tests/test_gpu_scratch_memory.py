"""Device memory that the operators keep between calls: given back on request, and
in no other allocator's way meanwhile."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402

MB = 1 << 20


def leave_memory_in_the_pool():
    """A forward projection whose scratch is the copy of a 168 MB volume."""
    det, _ = ops.detector(64, 48, 200.0)
    grid = ops.custom_grid(det, (512, 512, 160), 0.1)
    vol = torch.ones((160, 512, 512), device="cuda")
    out = ops.forward_project(vol, np.arange(4) * 90.0, None, det, grid)
    torch.cuda.synchronize()
    del vol
    torch.cuda.empty_cache()
    return out


def test_release_scratch_gives_the_memory_back():
    first = leave_memory_in_the_pool()
    kept = torch.cuda.mem_get_info()[0]
    ops.release_scratch()
    assert torch.cuda.mem_get_info()[0] - kept >= 160 * MB
    assert torch.equal(leave_memory_in_the_pool(), first)   # the next call takes it again
    with pytest.raises(Exception):
        ops.release_scratch(9999)
    torch.cuda.synchronize()


def test_another_allocator_gets_the_memory_kept():
    leave_memory_in_the_pool()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free + 100 * MB, dtype=torch.uint8, device="cuda")
    assert hold.numel() > free
    del hold
    torch.cuda.empty_cache()
