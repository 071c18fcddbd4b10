"""The group filter where its warps take several chunks of a run (GPU).

The filter's grid has 32 warps on each SM and a chunk is 32 records, so on 148 SMs a
warp takes a second chunk of a run beyond 151,552 records of one number of units (two
spots each): the loads ahead, the strides and the candidates of several chunks start
there."""
import numpy as np
import pytest

from lauematching_b200 import params as P
from lauematching_b200 import synth
from lauematching_b200._lib import device_info
from test_gpu_parity import engine_for

pytestmark = pytest.mark.gpu


# spots per record (one or several runs), chunks per warp of the first run, slots
@pytest.mark.parametrize("counts,rounds,K", [((1,), 2.03, 3), ((2,), 3.5, 16), ((3, 1), 4.0, 64),
                                             ((4, 3), 1.97, 17), ((5,), 2.5, 5), ((6, 5), 3.02, 33),
                                             ((8, 2), 2.0, 7), ((11,), 1.4, 64), ((16,), 2.3, 2),
                                             ((31, 32), 1.6, 9), ((34,), 2.2, 20), ((61, 33, 4), 1.1, 4)])
def test_filtered_passes_of_several_chunks_per_warp(counts, rounds, K):
    rng = np.random.default_rng(sum(counts) + K)
    W, H, S = 256, 192, max(counts)
    warp_round = device_info()["sms"] * 1024
    n = int(rounds * warp_round) + 7 * len(counts)
    p = P.parse_params_text(synth.params_text(nr_px=(W, H), max_nr_spots=S, min_nr_spots=1,
                                              min_intensity=1.0))
    rec = np.zeros((n * len(counts), 1 + 2 * S), np.uint16)
    rec[:, 0] = np.repeat(counts, n)
    rng.shuffle(rec[:, 0])
    rec[:, 1::2] = rng.integers(0, W, (len(rec), S), dtype=np.uint16)
    rec[:, 2::2] = rng.integers(0, H, (len(rec), S), dtype=np.uint16)
    slots = list(range(K))
    with engine_for(p, len(rec)) as e:
        e.upload_db(rec)
        for k in slots:  # corners of different size, so that cells of some slots stay unmarked
            img = np.zeros((H, W), np.uint8)
            img[: 20 + k % 30, : 15 + 2 * k % 60] = 1 + k
            e.load_image(k, img)
        found = 0
        for need in sorted({1, (min(counts) + 1) // 2, max(1, S // 3), S}):
            got = {}
            for variant in (1, 5):
                e.set_tuning(variant=variant)
                e.match(slots, need, 1.0)
                got[variant] = e.results_batch(slots)
                assert e.get_tuning()["last_form"] == (2 if variant == 5 else 0)
            for k in slots:
                assert got[5][k][1] == got[1][k][1], (need, k)
                assert np.array_equal(got[5][k][0], got[1][k][0]), (need, k)
                found += len(got[5][k][0])
        assert found > warp_round // 100
