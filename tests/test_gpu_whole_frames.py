"""Whole-number frames minus a whole-number background at the edges of the eight-pixel
loads (GPU)."""
import numpy as np
import pytest

from lauematching_b200 import preprocess as PP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("shape", [(1, 1), (1, 7), (2, 4), (3, 3), (33, 65), (64, 96), (211, 1031)])
def test_integer_differences_give_the_float64_thresholds(shape, dtype):
    rng = np.random.default_rng(shape[1])
    top = int(np.iinfo(dtype).max)
    h = PP.DevicePreprocessor(*shape)
    for kind in ("noise", "wild", "flat"):
        f = {"noise": rng.poisson(60, shape), "wild": rng.integers(0, top + 1, shape),
             "flat": np.full(shape, top)}[kind].clip(0, top).astype(dtype)
        for bg in (np.zeros(shape), rng.poisson(55, shape).astype(np.float64),
                   np.full(shape, 65535.0), rng.poisson(55, shape) + 0.5):
            h.set_background(bg)
            d = np.maximum(f.astype(np.float64) - bg, 0.0)
            nz = d[d > 0]
            med = np.median(nz) if nz.size else 0.0
            floor = max(med + 4 * (1.4826 * np.median(np.abs(nz - med))), 1.0) if nz.size else 1.0
            for method, want in (("adaptive", floor), ("percentile", np.percentile(d, 97.3))):
                cnt = h.segment(f, method, 0.0, 97.3, 1)
                assert cnt.threshold == want, (kind, method)
                got = h.images(thresholded=True)["thresholded"]
                assert np.array_equal(got, np.where(d <= want, 0.0, d).astype(np.uint16)), (kind, method)
