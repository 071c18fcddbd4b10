"""Median background of whole-number frames at the edges of its tiles (GPU)."""
import numpy as np
import pytest

from lauematching_b200 import preprocess as PP

ndimage = pytest.importorskip("scipy.ndimage")
pytestmark = pytest.mark.gpu


def _frames(ny, nx, rng):
    ramp = np.add.outer(np.arange(ny) * 3, np.arange(nx) * 2)
    noise = rng.poisson(120 + 0.05 * ramp)
    step = np.where(ramp > ramp.max() // 2, 60000, 3)
    wild = rng.integers(0, 65536, (ny, nx))
    return {"flat": np.full((ny, nx), 65535), "zero": np.zeros((ny, nx)), "noise": noise,
            "step": step, "steep": np.clip(ramp * 97, 0, 65535), "wild": wild}


# tiles are 64 x 32 pixels; sizes even and odd, as wide as the frame and wider, the
# largest the tiles take (255) and the first beyond
@pytest.mark.parametrize("shape,size,passes", [((32, 64), 3, 1), ((33, 65), 4, 2), ((31, 63), 31, 1),
                                               ((70, 130), 17, 2), ((1, 90), 5, 1), ((90, 1), 6, 1),
                                               ((40, 50), 101, 1), ((36, 34), 255, 1),
                                               ((36, 34), 256, 1)])
def test_whole_number_frames_match_scipy(shape, size, passes):
    rng = np.random.default_rng(size)
    h = PP.DevicePreprocessor(*shape)
    for name, f in _frames(*shape, rng).items():
        want = f.astype(np.float64)
        for _ in range(passes):
            want = ndimage.median_filter(want, size)
        for dt in (np.uint16, np.float64):
            got = h.median(f.astype(dt), size, passes)
            assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), (name, dt)
    # a value that is no whole number (or a negative zero) takes the other path
    for bad in (0.5, -0.0, 70000.0):
        f = rng.poisson(50, shape).astype(np.float64)
        f[shape[0] // 2, shape[1] // 2] = bad
        want = ndimage.median_filter(f, size)
        assert np.array_equal(h.median(f, size, 1), want)
    h.close()


def test_a_detector_frame_matches_scipy_on_a_strip():
    """A 2048-wide frame, radius 101, against scipy on rows whose windows it holds."""
    rng = np.random.default_rng(0)
    x = np.linspace(0, 1, 2048)[None, :]
    f = rng.poisson(105 + 60 * x + np.zeros((300, 1))).astype(np.float64)
    f[rng.integers(0, 300, 500), rng.integers(0, 2048, 500)] = 4000
    h = PP.DevicePreprocessor(300, 2048)
    got = h.median(f.astype(np.uint16), 101, 1)
    h.close()
    cut = f[:, 900:1100]
    assert np.array_equal(got[:, 950:1050], ndimage.median_filter(cut, 101)[:, 50:150])


@pytest.mark.parametrize("size,passes", [(5, 1), (9, 2)])
def test_frames_given_up_part_of_the_way_match_scipy(size, passes):
    """More tiles than run at once, of which the first, the last or all are beyond the
    tiles' thresholds, and values with gaps above and below the first threshold."""
    ny, nx = 1250, 1500
    rng = np.random.default_rng(size)
    smooth = rng.poisson(30, (ny, nx))
    first, last, second = smooth.copy(), smooth.copy(), smooth.copy()
    first[:40, :70] = rng.integers(0, 65536, (40, 70))
    last[-40:, -70:] = rng.integers(0, 65536, (40, 70))
    second[600:640, ::2] = 50000  # half of the values, then none
    frames = {"first": first, "last": last, "second": second, "gaps": 16 * smooth,
              "noise": rng.normal(20000, 1000, (ny, nx)).astype(int),
              "below": np.where(rng.random((ny, nx)) < 0.5, 3, 60000),
              "ramp": smooth + 8 * np.arange(nx)}
    h = PP.DevicePreprocessor(ny, nx)
    for name, f in frames.items():
        want = f.astype(np.uint16)
        for _ in range(passes):
            want = ndimage.median_filter(want, size)
        got = h.median(f.astype(np.uint16), size, passes)
        assert np.array_equal(got, want.astype(np.float64)), name
    h.close()
