"""The register-transform filter on groups of four detector rows: heights of every
remainder, widths at the edges of its lengths (whole power-of-two rows, rows
embedded in a transform twice as long or more), and samples its own logarithm
does not take."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from ct_b200 import ops  # noqa: E402
from ct_b200 import _lib as L  # noqa: E402


def reference(raw, W, H, D, pad):
    """-ln, cosine weight and the ramlak row filter in float64."""
    M = W if pad == 1 else 1 << (2 * W - 1).bit_length()
    win = np.arange(M // 2 + 1) / (M // 2 + 1) * W
    s = raw.astype(np.float64)
    if raw.dtype == np.uint16:
        s = s / 65535.0 + 1e-6
    u, v = np.arange(W) - W / 2.0, H / 2.0 - np.arange(H)
    p = -np.log(s / (1.0 + 1e-6)) * D / np.sqrt(D * D + u[None, :] ** 2 + v[:, None] ** 2)
    return np.fft.irfft(np.fft.rfft(p, n=M) * win, n=M)[..., :W]


@pytest.mark.parametrize("H", [2, 3, 4, 5, 7, 33])
@pytest.mark.parametrize("W,pad", [(256, 1), (65, 1), (128, 2), (129, 1), (200, 2), (512, 1), (511, 1), (700, 1),
                                   (1024, 1), (2048, 1), (2047, 1), (4096, 1)])
def test_rows_match_float64(W, pad, H):
    """Within 1e-5 per projection, the filter's bar at every length."""
    rng = np.random.default_rng(W + H)
    V = 3
    raw = rng.integers(9000, 60000, (V, H, W)).astype(np.uint16)
    D = float(np.float32(2.5 * max(W, H)))
    det, _ = ops.detector(W, H, D)
    out = ops.filter_projections(torch.from_numpy(raw.astype(np.int32)).to(torch.uint16).cuda(), det, L.RAMLAK, pad,
                                 L.FP32).double().cpu().numpy()
    ref = reference(raw, W, H, D, pad)
    for v in range(V):
        assert np.linalg.norm(out[v] - ref[v]) <= 1e-5 * np.linalg.norm(ref[v])


def test_logarithm_over_its_range():
    """Float samples over 60 decades (negative powers of two to large ones), one constant
    row pair each: the filtered row of a constant is its -ln times the window's zero
    bin response; compared with float64 through the whole filter."""
    W, V = 256, 120
    rng = np.random.default_rng(5)
    raw = np.exp(rng.uniform(-60.0, 60.0, (V, 4, W))).astype(np.float32)
    det, _ = ops.detector(W, 4, 700.0)
    out = ops.filter_projections(torch.from_numpy(raw).cuda(), det, L.RAMLAK, 1, L.FP32).double().cpu().numpy()
    ref = reference(raw, W, 4, 700.0, 1)
    assert np.linalg.norm(out - ref) <= 2e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("value", [0.0, -1.0, float("inf"), float("nan")])
@pytest.mark.parametrize("W", [256, 700])
def test_samples_without_a_logarithm_spoil_only_their_row_pair(W, value):
    """As logf gives them: infinities and NaN in the row, and in its partner of the
    complex transform; every other row keeps its values bit for bit."""
    H = 9
    rng = np.random.default_rng(W)
    raw = rng.uniform(0.2, 0.9, (2, H, W)).astype(np.float32)
    det, _ = ops.detector(W, H, 3.0 * W)
    clean = ops.filter_projections(torch.from_numpy(raw).cuda(), det, L.HANN, 1, L.FP32).cpu().numpy()
    raw[1, 6, 11] = value
    out = ops.filter_projections(torch.from_numpy(raw).cuda(), det, L.HANN, 1, L.FP32).cpu().numpy()
    assert not np.isfinite(out[1, 6]).any()
    keep = np.ones((2, H), bool)
    keep[1, 6:8] = False
    assert np.isfinite(clean).all()
    assert np.array_equal(out[keep], clean[keep])


def test_tiny_samples_match_float64():
    W = 256
    raw = np.full((1, 4, W), 0.5, np.float32)
    raw[0, 1, 3], raw[0, 2, 5] = 1e-39, 1e-45   # below the normal range
    det, _ = ops.detector(W, 4, 700.0)
    out = ops.filter_projections(torch.from_numpy(raw).cuda(), det, L.RAMLAK, 1, L.FP32).double().cpu().numpy()
    ref = reference(raw, W, 4, 700.0, 1)
    assert np.linalg.norm(out - ref) <= 1e-5 * np.linalg.norm(ref)


def test_extreme_base_intensity_takes_the_general_kernel():
    """A base intensity of 1e-31 puts the logarithm's arguments beyond the register
    kernel's range for whole-number samples. p is near -71 with a spread of about
    0.4; half a unit in its last place from the logarithm and from the weight is
    3e-6, 8e-6 of the spread the ramp keeps: 5e-5 covers it and the transform."""
    W, H, base = 256, 6, 1e-31
    rng = np.random.default_rng(3)
    raw = rng.integers(9000, 60000, (2, H, W)).astype(np.uint16)
    det, _ = ops.detector(W, H, 700.0, base_intensity=base)
    out = ops.filter_projections(torch.from_numpy(raw.astype(np.int32)).to(torch.uint16).cuda(), det, L.RAMLAK, 1,
                                 L.FP32).double().cpu().numpy()
    u, v = np.arange(W) - W / 2.0, H / 2.0 - np.arange(H)
    p = -np.log((raw / 65535.0 + 1e-6 * base) / (base + 1e-6 * base))
    p = p * 700.0 / np.sqrt(700.0 ** 2 + u[None, :] ** 2 + v[:, None] ** 2)
    ref = np.fft.irfft(np.fft.rfft(p) * (np.arange(W // 2 + 1) / (W // 2 + 1) * W), n=W)
    assert np.linalg.norm(out - ref) <= 5e-5 * np.linalg.norm(ref)
