"""Closest pair of component centres (the blur width), of few and of many centres (GPU)."""
import numpy as np
import pytest

from lauematching_b200 import preprocess as PP

pytestmark = pytest.mark.gpu


def _isolated(n, spacing, close=False):
    """n bright 4 x 4 spots, every two at least ``spacing`` apart; with ``close`` the
    last one 12 pixels from the first."""
    side = int(np.ceil(np.sqrt(max(n, 1))))
    img = np.zeros((side * spacing + 24, side * spacing + 24), np.uint16)
    at = [(8 + spacing * (i // side), 8 + spacing * (i % side)) for i in range(n)]
    if close:
        at[-1] = (at[0][0], at[0][1] + 12)
    for k, (y, x) in enumerate(at):
        img[y:y + 4, x:x + 4] = 1000
        img[y + k % 4, x + k // 4 % 4] += k % 7  # centres off the lattice
    return img


@pytest.mark.parametrize("n", [0, 1, 2, 33, 64, 2047, 2048, 2049, 2600])
@pytest.mark.parametrize("close", [False, True])
def test_closest_pair_of_few_and_many_centres(n, close):
    """All pairs of up to 2048 centres, the cells beyond, and every pair again where no
    two are within a cell (32 pixels) of one another."""
    if close and n < 3:
        pytest.skip("needs three spots")
    img = _isolated(n, 36, close)
    h = PP.DevicePreprocessor(*img.shape)
    for _ in range(2):
        cnt = h.segment(img, override_thresh=10.0, min_area=1)
        assert cnt.n_centres == n
        c = np.array([p[1] for p in h.centres(n)], np.float64).reshape(n, 2)
        want = np.inf
        for i in range(n - 1):
            d = c[i + 1:] - c[i]
            want = min(want, float((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]).min()))
        assert cnt.min_dist2 == want
    h.close()


def test_isolated_centres_do_not_wait_for_one_block():
    """The component stage of 3500 spots, none within a cell of another, against the
    same with one close pair: all pairs by a single block made it 30 times as long."""
    took = []
    for close in (False, True):
        img = _isolated(3500, 34, close)
        h = PP.DevicePreprocessor(*img.shape)
        t = []
        for _ in range(9):
            h.segment(img, override_thresh=10.0, min_area=1)
            t.append(h.timings()["components"])
        took.append(min(t))
        h.close()
    assert took[0] < 8 * took[1], took
