"""Passes over the records grouped by spot count, and the DB build's screens, at
the sizes where they can go wrong (GPU)."""
import numpy as np
import pytest

import oracle as O
from lauematching_b200 import params as P
from lauematching_b200 import synth
from test_gpu_parity import assert_same_survivors, engine_for

pytestmark = pytest.mark.gpu


def _random_db(rng, n, S, W, H):
    """Counts 0..S+1 (one above the clamp), every 16th pixel off the detector."""
    rec = np.zeros((n, 1 + 2 * S), np.uint16)
    rec[:, 0] = rng.integers(0, S + 2, n)
    x, y = rng.integers(0, W, (n, S)), rng.integers(0, H, (n, S))
    off = rng.random((n, S)) < 1 / 16
    rec[:, 1::2] = np.where(off, W + x % 7, x)
    rec[:, 2::2] = y
    return rec


# 4 spots a group and 32 in registers; 5 and 8 counter bits; 1 to 64 slots in up to
# 16 groups; detectors whose cells are 1 x 1, uneven and larger than a frame's edge
@pytest.mark.parametrize("S,K,nr_px,need", [(1, 1, (64, 48), 1), (5, 2, (61, 67), 2),
                                            (31, 16, (300, 257), 6), (32, 17, (300, 257), 9),
                                            (33, 5, (257, 300), 12), (40, 33, (640, 480), 12),
                                            (7, 64, (2048, 1100), 3), (255, 3, (256, 256), 30)])
@pytest.mark.parametrize("n", [1, 31, 33, 4097, 40000])
def test_filter_keeps_every_record_that_can_pass(S, K, nr_px, need, n):
    """Variant 5 (filtered) and the automatic variant (listed at these sizes) give
    the oracle's survivors in every slot."""
    rng = np.random.default_rng(100 * S + n)
    W, H = nr_px
    p = P.parse_params_text(synth.params_text(nr_px=nr_px, max_nr_spots=S, min_nr_spots=need,
                                              min_intensity=3.0))
    rec = _random_db(rng, n, S, W, H)
    imgs = []
    for k in range(K):
        img = np.zeros((H, W))
        img[rng.integers(0, H, 400), rng.integers(0, W, 400)] = rng.integers(1, 256, 400)
        if k % 3 == 0:  # a slot whose frame covers a quarter of the detector
            img[: H // 2, : W // 2] = 7.0
        imgs.append(img.ravel())
    slots = rng.permutation(64)[:K].tolist()
    with engine_for(p) as e:
        e.upload_db(rec)
        for s, img in zip(slots, imgs):
            e.load_image(s, img)
        for variant in (5, 3):
            e.set_tuning(variant=variant)
            for ms in (need, max(1, need - 1), S):
                e.match(slots, ms, 3.0)
                got = e.results_batch(slots)
                for s, img in list(zip(slots, imgs))[:6]:
                    ref = O.compare(rec, S, img, W, H, ms, 3.0)
                    assert got[s][1] == ref.n_pass, (variant, ms, s)
                    assert_same_survivors(got[s][0], ref)


@pytest.mark.parametrize("elo,px,shuffle", [(5.0, 0.0002, False), (0.0, 0.0002, True),
                                            (12.0, -0.0002, True)])
def test_build_screens_keep_every_spot(elo, px, shuffle):
    """Records of the screened build equal those of the all-FP64 one: a triclinic
    cell, an energy band from zero, a negative pixel pitch, HKLs in any order with
    repeats, 000 and some without their -h, and matrices that are no rotations."""
    rng = np.random.default_rng(7)
    txt = synth.params_text(lattice=(0.41, 0.52, 0.73, 81.0, 97.0, 112.0), space_group=2,
                            p=(0.03, -0.02, 0.4), r=(-0.9, 0.4, -0.3), px=px, nr_px=(1100, 1001),
                            elo=elo, ehi=25.0, max_nr_spots=12)
    p = P.parse_params_text(txt)
    hk = synth.hkls_cubic(5, "P")
    hk = np.concatenate([hk, hk[5:40], [[0, 0, 0]], hk[100:103]]).astype(np.int32)
    if shuffle:
        hk = hk[rng.permutation(len(hk))][: len(hk) - 200]
    om = synth.shoemake_orientations(3000, 11)
    om[7] *= 1.3
    om[8, 4] = np.nan
    om[9] = 0.0
    om[10] += 2e-5 * rng.standard_normal(9)  # as rounded in a file
    with engine_for(p) as e:
        e.build_db(om, hk)
        got = e.download_db()
        e.build_db(om, hk, exact_fp64=True)
        want = e.download_db()
    assert want[:, 0].max() == 12 and (want[:, 0] < 12).any()
    assert np.array_equal(got, want)
