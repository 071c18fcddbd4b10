"""What the library does when a call of the CUDA runtime fails (CPU).

The library's objects are linked against a runtime on the host (fake_cudart.cu) in
which allocations, copies and launches fail on request; no GPU takes part."""
import concurrent.futures
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from lauematching_b200 import _lib, build
from lauematching_b200 import params as P
from lauematching_b200 import synth
from lauematching_b200.engine import Engine
from lauematching_b200.preprocess import DevicePreprocessor

HERE = os.path.dirname(os.path.abspath(__file__))
MIB = 1 << 20


def _run(cmd):
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    tmp = str(tmp_path_factory.mktemp("fake"))
    objdir = os.path.join(build.HERE, "_build")
    headers = [os.path.join(build.CSRC, f) for f in os.listdir(build.CSRC) if f.endswith(("h",))]
    newest = max(os.path.getmtime(h) for h in headers)
    inc = ["-I", os.path.join(build.ROOT, "include")]
    objs, jobs = [], []
    for src in build.sources():
        obj = os.path.join(objdir, os.path.basename(src) + ".o")
        if not os.path.exists(obj) or os.path.getmtime(obj) < max(newest, os.path.getmtime(src)):
            obj = os.path.join(tmp, os.path.basename(src) + ".o")
            jobs.append([build.nvcc(), *build.NVCC_FLAGS, *inc, "-dc", "-c", src, "-o", obj])
        objs.append(obj)
    fake = os.path.join(tmp, "fake_cudart.o")
    jobs.append([build.nvcc(), *build.NVCC_FLAGS, *inc, "-c", os.path.join(HERE, "fake_cudart.cu"),
                 "-o", fake])
    with concurrent.futures.ThreadPoolExecutor(8) as ex:
        list(ex.map(_run, jobs))
    link = os.path.join(tmp, "dlink.o")
    _run([build.nvcc(), *build.NVCC_FLAGS[:2], "-dlink", "-Xcompiler", "-fPIC", *objs, "-o", link])
    so = os.path.join(tmp, "libfake.so")
    _run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, *objs, link, fake, "-lgomp"])
    return so


@pytest.fixture
def fake(fake_path, monkeypatch):
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", fake_path)
    f = C.CDLL(fake_path)
    f.fake_limits.argtypes = [C.c_size_t, C.c_size_t]
    f.fake_counts.argtypes = [C.c_int, C.c_ulonglong]
    for name in ("fake_device_used", "fake_host_used"):
        getattr(f, name).restype = C.c_size_t
    f.fake_fail_copies.argtypes = [C.c_long]
    for name in ("fake_device_mallocs", "fake_launched"):
        getattr(f, name).restype = C.c_long
    f.fake_reset()
    yield f
    f.fake_reset()


def _engine(max_nr_spots=15, **kw):
    return Engine(P.parse_params_text(synth.params_text(nr_px=(64, 64), max_nr_spots=max_nr_spots, **kw)))


def _db_size(e):
    n, s = C.c_uint64(0), C.c_int32(0)
    _lib.check(_lib.lib().lmb_db_info(e._h, C.byref(n), C.byref(s)))
    return n.value


def _records(n, S=15):
    return np.random.default_rng(n).integers(0, 60, (n, 1 + 2 * S), dtype=np.uint16)


def test_failed_upload_leaves_no_records(fake):
    with _engine() as e:
        e.upload_db(_records(100_000))
        assert _db_size(e) == 100_000
        fake.fake_fail_copies(MIB)
        with pytest.raises(_lib.LmbError):
            e.upload_db(_records(90_000))
        assert _db_size(e) == 0
        fake.fake_fail_copies(0)
        rec = _records(80_000)
        e.upload_db(rec)
        assert _db_size(e) == 80_000 and np.array_equal(e.download_db(), rec)


@pytest.mark.parametrize("what", ["spots", "copy", "kernel"])
def test_failed_build_leaves_no_records(fake, what):
    """More spots per record than a build takes, a failing copy, a failing launch."""
    om, hk = synth.shoemake_orientations(50_000, 1), synth.hkls_cubic(4)
    with _engine(1281 if what == "spots" else 15) as e:
        if what != "spots":
            e.build_db(om[:30_000], hk)
            assert _db_size(e) == 30_000
        else:
            e.upload_db(_records(1000, 1281))
        fake.fake_fail_copies(MIB if what == "copy" else 0)
        fake.fake_fail_kernel(b"dbbuild_kernel" if what == "kernel" else b"")
        with pytest.raises(_lib.LmbError):
            e.build_db(om, hk)
        assert _db_size(e) == 0


def test_failed_pass_leaves_no_counts(fake):
    """A pass whose ordering cannot be launched: what its counting kernel found is not
    added to by the next pass."""
    fake.fake_counts(9, 1000)
    with _engine(min_nr_spots=5) as e:
        e.upload_db(_records(1000))
        e.load_image(0, np.ones(64 * 64))
        fake.fake_survivors(3)
        fake.fake_fail_kernel(b"order_kernel")
        with pytest.raises(_lib.LmbError):
            e.match([0], 5, 1.0)
        fake.fake_fail_kernel(b"")
        e.match([0], 5, 1.0)
        assert fake.fake_launched(b"listed_kernel") == 2
        assert len(e.results(0)[0]) == 3


def _filtered(fake, e, n):
    """A DB of n records of 15 spots each and a filtered pass over it."""
    fake.fake_reset()
    fake.fake_counts(15, n)
    e.upload_db(_records(n))
    e.load_image(0, np.ones(64 * 64))
    e.match([0], 5, 1.0)
    assert fake.fake_launched(b"group_filter_kernel") == 1


@pytest.mark.parametrize("how", ["upload", "build", "first pass", "tiled layout"])
def test_memory_kept_for_the_next_db_is_given_back_when_it_does_not_fit(fake, how):
    """List, codes and candidates of the old DB (some 40 of its 62 bytes a record) are
    no reason for a new one not to fit, nor for a build's matrices, a new list or a
    tiled layout."""
    n = 1_000_000
    with _engine(min_nr_spots=5) as e:
        base = fake.fake_device_used()
        _filtered(fake, e, n if how != "first pass" else n // 3)
        if how == "upload":
            rec = _records(n * 6 // 5)
            fake.fake_limits(base + rec.nbytes + MIB, 1 << 40)
            e.upload_db(rec)
            assert _db_size(e) == len(rec) and np.array_equal(e.download_db(), rec)
        elif how == "build":
            fake.fake_limits(fake.fake_device_used() + 10 * MIB, 1 << 40)
            e.build_db(synth.shoemake_orientations(n - 5, 1), synth.hkls_cubic(2))
            assert _db_size(e) == n - 5
        elif how == "tiled layout":  # chunk counts: 16 bytes per 32 records
            e.upload_db(_records(n))
            fake.fake_limits(fake.fake_device_used(), 1 << 40)
            e.set_tuning(variant=2)
            e.match([0], 5, 1.0)
            assert e.get_tuning()["last_variant"] == 2
        else:  # the list of a longer DB, the old one's codes in its way
            e.upload_db(_records(n))
            fake.fake_limits(fake.fake_device_used() + MIB, 1 << 40)
            fake.fake_counts(15, 0)
            fake.fake_counts(1, n)
            e.match([0], 5, 1.0)
            assert e.layout_info()["compact"] == 1 and e.layout_info()["tiles"] == 0


def test_filter_without_memory_is_tried_once(fake):
    """No room for the codes: the passes run over the list, without asking again and
    without holding the candidates' memory; the next DB is tried anew."""
    n = 1_000_000
    with _engine(min_nr_spots=5) as e:
        fake.fake_counts(15, n)
        e.upload_db(_records(n))
        e.load_image(0, np.ones(64 * 64))
        before = fake.fake_device_used()
        fake.fake_limits(before + 12 * MIB, 1 << 40)
        e.match([0], 5, 1.0)
        used, tried = fake.fake_device_used(), fake.fake_device_mallocs()
        for ms in (5, 5, 5, 6):
            e.match([0], ms, 1.0)
        assert fake.fake_device_mallocs() == tried and fake.fake_launched(b"group_filter") == 0
        assert fake.fake_launched(b"listed_kernel") >= 3
        fake.fake_limits(fake.fake_device_used() + 100 * MIB, 1 << 40)
        e.upload_db(_records(n))
        e.match([0], 5, 1.0)
        assert fake.fake_launched(b"group_filter_kernel") == 1
        assert used - before < 6 * MIB  # list and counts 5.3 MB, candidates 4.2 MB


@pytest.mark.parametrize("pieces", [0, 1, 3])
def test_large_copies_go_directly_without_page_locked_pieces(fake, pieces):
    """Room for none, one or three of the four 8 MiB pieces: records, a background and
    a preprocessed frame move all the same."""
    with _engine() as e:
        fake.fake_limits(1 << 50, fake.fake_host_used() + pieces * 8 * MIB)
        rec = _records(700_000)
        e.upload_db(rec)
        assert np.array_equal(e.download_db(), rec)
    fake.fake_reset()
    ny, nx = 1100, 1001
    h = DevicePreprocessor(ny, nx)
    fake.fake_limits(1 << 50, fake.fake_host_used() + pieces * 8 * MIB)
    bg = np.random.default_rng(1).random((ny, nx))
    h.set_background(bg)
    assert np.array_equal(h.background(), bg)
    h.close()


@pytest.mark.parametrize("room", [True, False])
def test_room_for_long_lists_comes_when_one_is_read(fake, room):
    """An engine that only builds, and one whose passes find few survivors, lock no 8
    MiB of host memory; without them a long list is fetched from the device."""
    fake.fake_counts(9, 1000)
    host = fake.fake_host_used()
    with _engine(min_nr_spots=5) as e:
        e.build_db(synth.shoemake_orientations(1000, 1), synth.hkls_cubic(2))
        e.download_db()
        e.load_image(0, np.ones(64 * 64))
        for need, n in enumerate((3, 256, 257, 4096, 4097, 30), 1):  # each pass eager
            fake.fake_survivors(n)
            if not room:
                fake.fake_limits(1 << 50, fake.fake_host_used())
            launched = fake.fake_launched(b"gather")
            e.match([0], need, 1.0)
            assert len(e.results(0)[0]) == n and len(e.results_batch([0])[0][0]) == n
            fetched = n > (4096 if room and n > 257 else 256)
            assert fake.fake_launched(b"gather") - launched == fetched
            assert (fake.fake_host_used() - host > 8 * MIB) == (room and n in (4096, 4097, 30))
            fake.fake_limits(1 << 50, 1 << 50)


@pytest.mark.parametrize("method", ["adaptive", "percentile"])
@pytest.mark.parametrize("dtype,fractional_bg", [(np.uint16, 0), (np.uint16, 1), (np.uint8, 1),
                                                 (np.float32, 0), (np.float64, 1)])
def test_components_are_found_once(fake, method, dtype, fractional_bg):
    """A frame whose differences are no whole numbers goes to the radix selection
    before its components are looked for, and over a fractional background without
    a value histogram."""
    h = DevicePreprocessor(100, 80)
    fake.fake_fractional(fractional_bg)
    h.set_background(np.full((100, 80), 0.5 * fractional_bg))
    fake.fake_fractional(0)
    h.segment(np.ones((100, 80), dtype), method=method)
    assert fake.fake_launched(b"label_kernel") == 1
    assert fake.fake_launched(b"foreground_kernel") == 1
    assert fake.fake_launched(b"value_hist_kernel") == 1 - fractional_bg
    radix = fractional_bg or dtype is np.float32  # the fake leaves the value path unset
    assert (fake.fake_launched(b"sel_hist_kernel") > 0) == bool(radix)
    h.close()


@pytest.mark.parametrize("n,spots,variant,form", [(1000, 15, 5, 1), (1_000_000, 3, 2, 2),
                                                  (1_000_000, 15, 5, 2), (1000, 2, 2, 1)])
def test_the_form_of_the_pass_is_reported(fake, n, spots, variant, form):
    """What a pass ran over goes by the number of spots to look at, ``last_variant`` by
    the number per record."""
    fake.fake_counts(spots, n)
    with _engine(min_nr_spots=2) as e:
        e.upload_db(_records(n))
        e.load_image(0, np.ones(64 * 64))
        e.match([0], 2, 1.0)
        assert fake.fake_launched(b"group_filter_kernel") == form - 1
        assert e.get_tuning()["last_variant"] == variant and e.get_tuning()["last_form"] == form
        e.set_tuning(variant=1)
        e.match([0], 2, 1.0)
        assert e.get_tuning()["last_form"] == 0
