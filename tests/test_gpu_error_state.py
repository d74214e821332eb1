"""A call that a CUDA error refused leaves nothing behind for the next one."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402
from ct_b200 import _lib as L  # noqa: E402


def test_a_wrong_device_does_not_fail_the_next_call():
    det, grid = ops.detector(32, 20, 120.0)
    proj = torch.ones((4, 20, 32), device="cuda")
    free = ctypes.c_size_t()
    assert L.lib().ctb_free_memory(9999, ctypes.byref(free), None) == L.CTB_ERR_CUDA
    assert b"invalid device" in L.lib().ctb_last_error_global()
    assert float(ops.backproject(proj, np.arange(4) * 90.0, None, det, grid).norm()) > 0
