"""Copies through the page-locked pieces and the build's chunks at their edges (GPU)."""
import numpy as np
import pytest

from lauematching_b200 import params as P
from lauematching_b200 import synth
from lauematching_b200.engine import PinnedBuffer
from test_gpu_parity import engine_for

pytestmark = pytest.mark.gpu


# 1 + 2 S uint16 = 64 bytes a record; 2 MiB go directly, pieces are 8 MiB, four in the ring
@pytest.mark.parametrize("mib,extra", [(2, 0), (2, 1), (8, -1), (8, 0), (8, 1), (32, 0), (32, 1), (45, 7)])
def test_records_go_up_and_down_unchanged(mib, extra):
    p = P.parse_params_text(synth.params_text(nr_px=(64, 64), max_nr_spots=15))
    rng = np.random.default_rng(mib)
    n = (mib << 20) // 62 + extra
    rec = rng.integers(0, 65536, (n, 31), dtype=np.uint16)
    pin = PinnedBuffer(rec.shape, np.uint16)
    pin.array[...] = rec
    with engine_for(p) as e:
        e.upload_db(rec)
        assert np.array_equal(e.download_db(), rec)
        assert np.array_equal(e.download_db(5, n - 11), rec[5:n - 6])
        e.upload_db(pin.array[:n - 3])  # page-locked, into the same memory
        assert np.array_equal(e.download_db(), rec[:n - 3])
    pin.free()


@pytest.mark.parametrize("n", [1, 127, 32768, 98305, 200_000, (256 << 10) * 2 + 1])
def test_chunked_build_equals_its_parts(n):
    """A build over several chunks gives each orientation the record that a build of
    a short list around it gives; the synthetic build of the same matrices too."""
    p = P.parse_params_text(synth.params_text(max_nr_spots=10))
    hk = synth.hkls_cubic(4)
    with engine_for(p) as e:
        om = e.build_db_synthetic(seed=5, n=n, hkls=hk, return_orients=True)
        synthetic = e.download_db()
        e.build_db(om, hk)
        got = e.download_db()
        assert np.array_equal(got, synthetic)
        for at in {0, n // 3, n // 2, max(0, n - 300)}:
            e.build_db(om[at:at + 300], hk)
            assert np.array_equal(e.download_db(), got[at:at + 300])


def test_float64_copies_survive_the_growth_of_their_room():
    """keep_f64 loads into slots that make the room grow: each slot's float64 pass
    gives what it gave alone."""
    rng = np.random.default_rng(2)
    p = P.parse_params_text(synth.params_text(nr_px=(300, 200), max_nr_spots=7, min_nr_spots=2))
    rec = np.zeros((5000, 15), np.uint16)
    rec[:, 0] = 7
    rec[:, 1::2] = rng.integers(0, 300, (5000, 7))
    rec[:, 2::2] = rng.integers(0, 200, (5000, 7))
    slots = [0, 3, 1, 40, 63]
    imgs = {s: np.where(rng.random(60000) < 0.2, rng.random(60000) * 50, 0.0) for s in slots}

    def one(e, s):
        e.match([s], 2, 3.0, value_mode=1)
        return e.results(s)

    alone = {}
    for s in slots:
        with engine_for(p) as e:
            e.upload_db(rec)
            e.load_image(s, imgs[s], keep_f64=True)
            alone[s] = one(e, s)
    with engine_for(p) as e:
        e.upload_db(rec)
        for i, s in enumerate(slots):
            e.load_image(s, imgs[s], keep_f64=True)
            for t in slots[:i + 1]:  # eager, then from a graph, then over new room
                for _ in range(2):
                    got, n_pass = one(e, t)
                    assert n_pass == alone[t][1] and np.array_equal(got, alone[t][0])


@pytest.mark.parametrize("dtype", [np.uint8, np.float32, np.float64])
def test_pairs_read_in_place_and_pairs_copied_give_the_dense_slots(dtype):
    """Pairs of one frame are read from page-locked memory up to 128 KiB and copied
    beyond: both sides of that line, more frames in a row than staging buffers."""
    rng = np.random.default_rng(11)
    nx, ny = 800, 700
    p = P.parse_params_text(synth.params_text(nr_px=(nx, ny), max_nr_spots=7, min_nr_spots=1))
    rec = np.zeros((4000, 15), np.uint16)
    rec[:, 0] = 7
    rec[:, 1::2] = rng.integers(0, nx, (4000, 7))
    rec[:, 2::2] = rng.integers(0, ny, (4000, 7))
    size = np.dtype(dtype).itemsize
    bytes_of = lambda n: -(-4 * n // 16) * 16 + n * size
    last = max(n for n in range(1, 40000) if bytes_of(n) <= 128 << 10)
    frames = []
    for n in (1, last, last + 1, last - 1, last + 2000, 100, last):
        f = np.zeros(nx * ny, dtype)
        f[rng.choice(nx * ny, n, replace=False)] = rng.integers(1, 256, n)
        frames.append(f)
    slots = list(range(len(frames)))
    got = {}
    for sparse in (True, False):
        with engine_for(p) as e:
            e.upload_db(rec)
            e.set_sparse_uploads(sparse)
            for s in slots:
                e.load_image(s, frames[s])
            e.match(slots, 1, 0.0)
            got[sparse] = [e.results(s) for s in slots]
    for a, b in zip(got[True], got[False]):
        assert a[1] == b[1] and np.array_equal(a[0], b[0])
