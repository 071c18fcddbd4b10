"""The DB build's screens against FP64 for every HKL, for matrices at the edge of what
counts as a rotation and beyond it (GPU)."""
import numpy as np
import pytest

from lauematching_b200 import params as P
from lauematching_b200 import synth
from test_gpu_parity import engine_for

pytestmark = pytest.mark.gpu

GEOMETRIES = {
    "normal": {},
    "tilted": dict(p=(0.028745, 0.002788, 0.513115), r=(-1.20131258, -1.21399082, -1.21881158)),
    "back": dict(p=(0.01, -0.02, 0.2), r=(0.1, 2.8, -0.2)),  # 2 theta from about 110 degrees
    "near": dict(p=(0.0, 0.05, 0.08), r=(0.3, -0.4, 0.1)),   # wide, off centre
}


def _off(om):
    m = om.reshape(-1, 3, 3)
    return np.abs(np.einsum("nki,nkj->nij", m, m) - np.eye(3)).max((1, 2))


def _at_tolerance(rot, rng, limit):
    """Rotations with a random strain that brings the largest entry of |M^T M - 1| to
    ``limit`` (a fraction of each matrix's own)."""
    noise = rng.standard_normal(rot.shape)
    lo, hi = np.zeros(len(rot)), np.full(len(rot), 1.0)
    for _ in range(60):
        mid = (lo + hi) / 2
        over = _off(rot + mid[:, None] * noise) > limit
        lo, hi = np.where(over, lo, mid), np.where(over, mid, hi)
    return rot + lo[:, None] * noise


@pytest.mark.parametrize("geometry", sorted(GEOMETRIES))
@pytest.mark.parametrize("hexagonal", [False, True])
def test_screened_records_equal_fp64_ones(geometry, hexagonal):
    rng = np.random.default_rng(17)
    lat = dict(lattice=(0.295, 0.295, 0.468, 90.0, 90.0, 120.0), space_group=194) if hexagonal else {}
    p = P.parse_params_text(synth.params_text(max_nr_spots=20, **lat, **GEOMETRIES[geometry]))
    hk = synth.hkls_hexagonal(6) if hexagonal else synth.hkls_cubic(8)
    rot = synth.shoemake_orientations(6000, 23)
    lists = {"just inside 1e-4": _at_tolerance(rot, rng, 0.9999e-4),
             "just outside 1e-4": _at_tolerance(rot, rng, 1.0001e-4),
             "4 digits": np.round(rot, 4), "2 digits": np.round(rot, 2),
             "strained": rot + 0.2 * rng.standard_normal(rot.shape),
             "scaled": rot * 10.0 ** rng.uniform(-3, 3, (len(rot), 1)),
             "left-handed": -rot,
             "flat": np.concatenate([rot[:, :6], rot[:, 3:6] * (1 + 1e-9)], 1)}
    odd = rot[:64].copy()
    for i, v in enumerate((0.0, np.nan, np.inf, -np.inf, 1e200, 1e30, 1e-30, 1e-200)):
        odd[8 * i] = v
        odd[8 * i + 1, i] = v
        odd[8 * i + 2] *= v if np.isfinite(v) else 1.0
    lists["odd"] = odd
    with engine_for(p) as e:
        found = 0
        for name, om in lists.items():
            e.build_db(om, hk)
            got = e.download_db()
            e.build_db(om, hk, exact_fp64=True)
            want = e.download_db()
            bad = np.flatnonzero((got != want).any(1))
            assert not len(bad), (name, len(bad), om[bad[0]])
            found += int(want[:, 0].sum())
    assert found > 1000


def test_lists_of_coarse_matrices_build_about_as_fast_as_rotations():
    """2e5 matrices of three digits, none a rotation: within five times the rotations'
    time (FP64 for every HKL took seven, the screens 2.7)."""
    import time
    p = P.parse_params_text(synth.params_text())
    om, hk = synth.shoemake_orientations(200_000, 3), synth.hkls_cubic(8)
    took = []
    with engine_for(p) as e:
        for m in (om, np.round(om, 3)):
            ts = []
            for _ in range(6):
                t = time.perf_counter()
                e.build_db(m, hk)
                ts.append(time.perf_counter() - t)
            took.append(min(ts))
    assert took[1] < 5 * took[0], took
