"""Survivor lists around the rooms that a pass writes them to (GPU)."""
import numpy as np
import pytest

from lauematching_b200 import params as P
from lauematching_b200 import synth
from test_gpu_parity import engine_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [0, 300, 100])
def test_lists_read_late_and_of_every_length(cap):
    """Record i has one spot on pixel i and a frame of m positive pixels m survivors:
    lists of up to 256 and of up to 4096 in host memory, longer ones on the device.
    Lists of earlier passes are read after the larger room was made, eager passes and
    replayed ones."""
    n = 6000
    p = P.parse_params_text(synth.params_text(nr_px=(100, 60), max_nr_spots=1, min_nr_spots=1,
                                              min_intensity=0.0))
    rec = np.zeros((n, 3), np.uint16)
    rec[:, 0], rec[:, 1], rec[:, 2] = 1, np.arange(n) % 100, np.arange(n) // 100
    lengths = [m for m in (3, 255, 256, 257, 300, 4095, 4096, 4097, 6000, 100) if not cap or m <= cap]
    rng = np.random.default_rng(1)
    on = [np.sort(rng.choice(n, m, replace=False)) for m in lengths]
    u8 = [1 + at % 255 for at in on]  # as loaded: scaled to a maximum of 255
    u8 = [np.clip(np.floor(v * (255.0 / v.max())), 1, 255) for v in u8]
    with engine_for(p, cap) as e:
        e.upload_db(rec)
        for k, at in enumerate(on):
            img = np.zeros(n, np.uint8)
            img[at] = 1 + at % 255
            e.load_image(k, img)
        slots = list(range(len(on)))

        def check(k, got):
            assert got[1] == lengths[k]
            assert np.array_equal(got[0]["id"], on[k]), lengths[k]
            assert np.array_equal(got[0]["sum_u8"], u8[k])

        for turn in range(3):
            for k in slots:  # one pass a slot, all before the first is read
                e.match([k], 1, 0.0)
            for k in reversed(slots):
                check(k, e.results(k))
            e.match(slots, 1, 0.0)
            got = e.results_batch(slots)
            for k in slots:
                check(k, got[k])
                check(k, e.results(k))
