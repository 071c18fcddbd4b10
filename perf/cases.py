"""Timed cases of the framework: what its users have it do, through its public entry points.

A user indexes Laue frames against an orientation DB.  The cases are that work from the raw frame and
the orientation list to the survivors, at the sizes of this repository's configurations, tests and
benchmark: detectors of 1024^2, 1100 x 1001 and 2048^2 pixels, DBs of 1e5 to 1e8 orientations, 1 to 64
frames per pass, fcc (1240 HKLs) and hexagonal (7790 HKLs) crystals, the detector normal to the beam
(about 1.25 on-detector spots per orientation; hexagonal 3.3) and the tilted 34-ID-E detector (15).
Frames of fewer pixels are binned ones: the detector keeps its size.  Kinds:

  match       frames against a resident DB: ``Engine.match`` + ``results``; with ``load`` the frames
              come from host memory in the given dtype in every pass, otherwise they lie in their slots
              (the throughput form: several parameter sets or DB ranges over one batch)
  cache       DB build from orientations in host memory and the download of its records (the forward
              cache that the command line writes)
  fresh       DB build and the first pass over it (the command line with DoFwd 1)
  raw         raw uint16 detector frames -> preprocessing on the device -> image slots -> pass
  preprocess  one raw frame with its own median background to host arrays (``preprocess_image``)

DBs of up to ``HOST_ORIENTS`` orientations are built from host matrices, larger ones by the device's
own generator.  Refinement and duplicate merge follow a pass on the host and are not timed here.
"""
import math

import numpy as np
import torch

from lauematching_b200 import params as P
from lauematching_b200 import preprocess as PP
from lauematching_b200 import synth
from lauematching_b200.engine import SURVIVOR_DTYPE, Engine, PinnedBuffer

_DEV = "cuda"
HOST_ORIENTS = 10_000_000
SCAN = 200_000  # records searched for the grains of the frames
TILTED = dict(p=(0.028745, 0.002788, 0.513115), r=(-1.20131258, -1.21399082, -1.21881158))
HEX_LATTICE = (0.295, 0.295, 0.468, 90.0, 90.0, 120.0)
# on-detector spots per DB orientation that belong to orientations with at least MinNrSpots of them
# (the others cannot match): counted on 10,000 to 40,000 orientations
SPOTS = {"normal": {3: 0.37, 4: 0.071, 5: 0.0105}, "tilted": {5: 14.8, 8: 14.7, 12: 12.8},
         "hex": {4: 2.0, 5: 1.13, 6: 0.51}}


def _case(kind, name=None, **kw):
    c = dict(kind=kind, geometry="normal", n=100_000, frames=1, nx=2048, ny=2048, min_spots=5,
             min_intensity=200.0, load="", pinned=True, background=False, exact_fp64_values=False,
             method="adaptive")
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest use: one frame against a small grid of orientations (a quick look, a test set-up)
        _case("match", "plain_100k_1", load="u8"),
        # one wire frame at a time against the full DB, as the daemon serves a lone request
        _case("match", "plain_100M_1", n=100_000_000, load="f32"),
        # the batched pass over resident frames: throughput of a scan
        _case("match", "batch_100M_64", n=100_000_000, frames=64),
        # a backlog of wire frames: load, pass, results
        _case("match", "wire_100M_32", n=100_000_000, frames=32, load="f32"),
        # the beamline's own tilted detector: every orientation can match
        _case("match", "tilted_100M_64", geometry="tilted", n=100_000_000, frames=64),
        # the same detector, few float64 frames of an odd size against an odd number of orientations
        _case("match", "tilted_10M_odd_3", geometry="tilted", n=9_999_991, frames=3, nx=1100, ny=1001,
              load="f64", pinned=False),
        # lower symmetry: more reflections, more spots per orientation
        _case("match", "hex_100M_32", geometry="hex", n=100_000_000, frames=32),
        # frames that keep their background: a thousand survivors per frame
        _case("match", "survivors_100M_16", n=100_000_000, frames=16, background=True,
              min_intensity=50.0),
        # the forward cache of a small orientation list, to be written to a file
        _case("cache", "cache_tilted_200k", geometry="tilted", n=200_000),
        # first use with a new crystal: build, lay out, match one frame with its float64 values
        _case("fresh", "fresh_hex_4M_1", geometry="hex", n=4_000_037, load="f64", pinned=False,
              exact_fp64_values=True),
        # raw detector frames to survivors without leaving the device
        _case("raw", "raw_10M_16", n=10_000_000, frames=16),
        # the image server's first frame: median background and every preprocessing step, to the host
        _case("preprocess", "preprocess_2048"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["match"] * 6 + ["cache", "fresh", "raw", "preprocess"])
    geometry = rng.choice(["normal", "tilted", "hex"])
    nx, ny = rng.choice([(2048, 2048), (2048, 2048), (1024, 1024), (1100, 1001),
                         (_log_int(rng, 900, 2048), _log_int(rng, 900, 2048))])
    c = _case(kind, geometry=geometry, nx=nx, ny=ny, frames=_log_int(rng, 1, 64),
              min_spots=rng.choice(sorted(SPOTS[geometry])),
              min_intensity=rng.choice([50.0, 100.0, 200.0]))
    if kind == "match":
        c["n"] = _log_int(rng, 100_000, 30_000_000 if geometry == "hex" else 100_000_000)
        c["load"] = rng.choice(["", "", "u8", "f32", "f64"])
        c["pinned"] = rng.choice([True, False])
        if geometry == "normal" and c["min_spots"] == 5 and c["frames"] <= 16 and (nx, ny) == (2048, 2048):
            c["background"] = rng.choice([True, False])
            if c["background"]:
                c["min_intensity"] = 50.0
    elif kind == "cache":
        c.update(n=_log_int(rng, 50_000, 400_000), frames=1)
    elif kind == "fresh":
        c.update(n=_log_int(rng, 100_000, 4_000_000), frames=1, load="f64", pinned=False,
                 exact_fp64_values=rng.choice([True, False]))
    elif kind == "raw":
        c.update(n=_log_int(rng, 100_000, 10_000_000), frames=_log_int(rng, 1, 16))
        c["method"] = rng.choice(["adaptive", "percentile"])
    else:
        c.update(n=0, frames=1, min_spots=5, method=rng.choice(["adaptive", "percentile"]))
    return c


# ---- inputs -----------------------------------------------------------------------------------
def _params(case):
    geo = TILTED if case["geometry"] == "tilted" else {}
    lat = dict(lattice=HEX_LATTICE, space_group=194) if case["geometry"] == "hex" else {}
    return P.parse_params_text(synth.params_text(
        nr_px=(case["nx"], case["ny"]), px=0.0002 * 2048 / max(case["nx"], case["ny"]),
        max_nr_spots=30, min_nr_spots=case["min_spots"],
        min_intensity=case["min_intensity"], **geo, **lat))


def _hkls(case):
    return synth.hkls_hexagonal(10) if case["geometry"] == "hex" else synth.hkls_cubic(8)


def _generator(seed, salt):
    return torch.Generator(device=_DEV).manual_seed(1_000_003 * seed + salt)


def _rotations(n, seed):
    """(n, 9) uniform random rotations (normalised Gaussian quaternions), float64 on the GPU."""
    q = torch.randn(n, 4, dtype=torch.float64, device=_DEV, generator=_generator(seed, 1))
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1)


def _spot_frame(records, grains, nx, ny, sigma, lo, hi, g):
    """Gaussian spots of the grains' records on a (ny, nx) float32 frame (the larger wins)."""
    pts = np.concatenate([np.zeros((0, 2), np.int64)] +
                         [records[i, 1:1 + 2 * int(records[i, 0])].reshape(-1, 2) for i in grains])
    pts = torch.as_tensor(pts.astype(np.int64), device=_DEV)
    rad = int(math.ceil(4 * sigma))
    off = torch.arange(-rad, rad + 1, device=_DEV)
    amp = lo + (hi - lo) * torch.rand(pts.shape[0], device=_DEV, generator=g)
    px, py = pts[:, 0, None, None] + off[None, None, :], pts[:, 1, None, None] + off[None, :, None]
    v = amp[:, None, None] * torch.exp(-0.5 * (off[None, None, :] ** 2 + off[None, :, None] ** 2) / sigma ** 2)
    ok = ((px >= 0) & (px < nx) & (py >= 0) & (py < ny)).expand(v.shape)
    img = torch.zeros(ny * nx, device=_DEV)
    return img.scatter_reduce_(0, (py * nx + px).expand(v.shape)[ok], v[ok], "amax").reshape(ny, nx)


def _frames(case, records, seed):
    """The case's frames as a (K, ny, nx) GPU tensor of float32 whole numbers: thresholded (or, with
    ``background``, unthresholded) frames of 1-20 grains with maximum 255, or raw detector frames."""
    g, rng = _generator(seed, 2), np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    raw = case["kind"] in ("raw", "preprocess")
    out = torch.empty(case["frames"], ny, nx, device=_DEV)
    for k in range(case["frames"]):
        grains = synth.pick_grains(records, int(rng.integers(1, 21)), case["min_spots"], rng)
        if raw:
            yy = torch.linspace(0, 1, ny, device=_DEV)[:, None]
            xx = torch.linspace(0, 1, nx, device=_DEV)[None, :]
            img = torch.poisson(105.0 + 60.0 * (0.6 * yy + 0.4 * xx), generator=g)
            img = img + _spot_frame(records, grains, nx, ny, 1.2, 300.0, 4000.0, g)
            out[k] = img.round().clamp(0, 65535)
        else:
            img = _spot_frame(records, grains, nx, ny, 2.0, 50.0, 255.0, g)
            img = img + torch.poisson(torch.full((ny, nx), 5.0, device=_DEV), generator=g)
            if not case["background"]:
                img = torch.where(img < 20.0, 0.0, img)
            img = img.round().clamp(0, 255)
            out[k] = (img * (255.0 / img.max().clamp(min=1.0))).round()
    return out


_NP = {"u8": np.uint8, "f32": np.float32, "f64": np.float64, "u16": np.uint16}


def _to_host(frames, dtype, pinned):
    """The frames in host memory, page-locked or not: (owner, list of 2-D arrays)."""
    dt = _NP[dtype]
    if not pinned:
        a = frames.cpu().numpy().astype(dt)
        return a, list(a)
    buf = PinnedBuffer(tuple(frames.shape), dt)
    buf.array[...] = frames.cpu().numpy()
    return buf, list(buf.array)


def _config(case):
    return dict(nr_px_x=case["nx"], nr_px_y=case["ny"], px_x=0.2, px_y=0.2, distance=0.513,
                threshold_method=case["method"], threshold_value=0.0, threshold_percentile=99.0,
                min_area=10, filter_radius=101, median_passes=1, orientation_spacing=0.4,
                background_file="")


def _some_records(case, seed):
    """Records that the frames of a case without a resident DB take their spots from."""
    with Engine(_params(case), survivor_capacity=1024) as e:
        e.build_db(_rotations(SCAN, seed).cpu().numpy(), _hkls(case))
        return e.download_db()


def prepare(case, seed):
    p, hkls = _params(case), _hkls(case)
    k = case["frames"]
    st = dict(case=case, p=p, hkls=hkls, slots=list(range(k)), sv=np.zeros(_room(case), SURVIVOR_DTYPE),
              filled=0, count=np.zeros(k, np.int64), n_pass=np.zeros(k, np.int64))
    if case["kind"] == "preprocess":
        st["hold"], fr = _to_host(_frames(case, _some_records(case, seed), seed), "u16", True)
        return dict(st, frame=fr[0], cfg=_config(case))
    orients = _rotations(case["n"], seed).cpu().numpy() if case["n"] <= HOST_ORIENTS else None
    if case["kind"] == "cache":
        return dict(st, orients=orients, engine=Engine(p))
    if case["kind"] == "fresh":
        records = _some_records(case, seed)
        st["hold"], fr = _to_host(_frames(case, records, seed), case["load"], case["pinned"])
        return dict(st, orients=orients, engine=Engine(p), frames=fr)
    e = Engine(p)
    if orients is not None:
        e.build_db(orients, hkls)
    else:
        e.build_db_synthetic(seed, case["n"], hkls, hex_fz=case["geometry"] == "hex")
    frames = _frames(case, e.download_db(0, min(SCAN, case["n"])), seed)
    if case["kind"] == "raw":
        st["hold"], st["frames"] = _to_host(frames, "u16", True)
        cfg = _config(case)
        st["pool"] = PP.PreprocessPool(cfg, PP.compute_background(st["frames"][0], 101, 1))
    elif case["load"]:
        st["hold"], st["frames"] = _to_host(frames, case["load"], case["pinned"])
    else:
        hold, fr = _to_host(frames, "u8", False)
        e.load_images(st["slots"], fr)
        st["frames"] = None
    return dict(st, engine=e)


# ---- one pass ---------------------------------------------------------------------------------
def _room(case):
    """Entries that the program keeps for the survivors of a pass (4-30 per thresholded frame)."""
    return case["frames"] * (16384 if case["background"] else 4096)


def _survivors(st, res, slots):
    """The lists back to back in the program's own array, the rest of it zero."""
    sv, n = st["sv"], 0
    for i, s in enumerate(slots):
        v, st["n_pass"][i] = res[s]
        sv[n:n + len(v)] = v
        n += len(v)
        st["count"][i] = len(v)
    sv[n:st["filled"]] = 0
    st["filled"] = n
    return {"count": st["count"], "n_pass": st["n_pass"], "id": sv["id"].view(np.int64),
            "n_spots": sv["n_spots"], "sum_u8": sv["sum_u8"], "tot_int": sv["tot_int"],
            "score": sv["score"]}


def run(st):
    case, p, slots = st["case"], st["p"], st["slots"]
    kind = case["kind"]
    if kind == "preprocess":
        blurred, img, labels, centres = PP.preprocess_image(st["frame"], st["cfg"])
        rows = np.zeros((4096, 4))
        rows[:len(centres)] = [(c[0], *c[1], c[2]) for c in centres]
        return {"blurred": blurred, "filt_img": img, "filt_labels": labels, "centres": rows}
    e = st["engine"]
    if kind == "cache":
        e.build_db(st["orients"], st["hkls"])
        return e.download_db()
    mode = 1 if case["exact_fp64_values"] else 0
    if kind == "fresh":
        e.build_db(st["orients"], st["hkls"])
    if kind == "raw":  # a frame without spots leaves its slot as it was
        done = st["pool"].to_slots(e, slots, st["frames"])
        slots = [s for s, n in zip(slots, done) if n is not None]
    elif case["load"] and len(slots) == 1:
        e.load_image(0, st["frames"][0], keep_f64=bool(mode), want_scale=False)
    elif case["load"]:
        e.load_images(slots, st["frames"])
    e.match(slots, p.min_nr_spots, p.min_intensity, value_mode=mode)
    res = {slots[0]: e.results(slots[0])} if len(slots) == 1 else e.results_batch(slots)
    return _survivors(st, res, slots)


def work(case):
    """Bytes a pass cannot do without, each once: the host frames (resident ones: one bit per pixel);
    for a match, 4 bytes per on-detector spot of the orientations that have MinNrSpots of them; for a
    build, its matrices and records; its flops, one rotation (15) per orientation and HKL."""
    px = case["nx"] * case["ny"]
    size = {"u8": 1, "f32": 4, "f64": 8, "": 0.125}[case["load"]]
    if case["kind"] == "preprocess":
        return {"bytes": px * (2 + 8 + 2 + 4), "flops": px * 2 * 9 * 2}
    size = 2 if case["kind"] == "raw" else size
    b = 0 if case["kind"] == "cache" else case["frames"] * px * size
    if case["kind"] != "cache":
        b += case["n"] * 4 * SPOTS[case["geometry"]][case["min_spots"]]
    f = 0
    if case["kind"] in ("cache", "fresh"):
        b += case["n"] * (72 + 2 * 61)
        f = 15.0 * case["n"] * len(_hkls(case))
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, without the framework -------------------------------------------------
def _forward(case, om):
    """Spots of the orientations (n, 9): flat (orientation, pixel) tensors in record order."""
    p, hkls = _params(case), torch.as_tensor(_hkls(case).astype(np.float64), device=_DEV)
    a, b, c = (float(v) for v in p.lattice[:3])
    al, be, ga = (math.radians(float(v)) for v in p.lattice[3:])
    v = math.sqrt(1 - math.cos(al) ** 2 - math.cos(be) ** 2 - math.cos(ga) ** 2 +
                  2 * math.cos(al) * math.cos(be) * math.cos(ga))
    direct = np.array([[a, b * math.cos(ga), c * math.cos(be)],
                       [0, b * math.sin(ga), c * (math.cos(al) - math.cos(be) * math.cos(ga)) / math.sin(ga)],
                       [0, 0, c * v / math.sin(ga)]])
    recip = torch.as_tensor(2 * math.pi * np.linalg.inv(direct).T, device=_DEV)
    r = np.array([float(x) for x in p.r_array])
    t = float(np.linalg.norm(r))
    ax = r / t
    k = np.array([[0, -ax[2], ax[1]], [ax[2], 0, -ax[0]], [-ax[1], ax[0], 0]])
    rot = np.eye(3) + math.sin(t) * k + (1 - math.cos(t)) * (k @ k)
    rt = torch.as_tensor(rot.T.copy(), device=_DEV)
    pos = [float(x) for x in p.p_array]
    spots, step = [], max(1, 40_000_000 // len(hkls))
    for i in range(0, om.shape[0], step):
        m = om[i:i + step].reshape(-1, 3, 3) @ recip
        qz = m[:, 2] @ hkls.T
        q2 = (m[:, 0] @ hkls.T) ** 2 + (m[:, 1] @ hkls.T) ** 2 + qz ** 2
        energy = 1.2398419739 * q2 / (-4 * math.pi * qz)
        o, h = torch.nonzero((energy >= float(p.elo)) & (energy <= float(p.ehi)), as_tuple=True)
        q = (m[o] @ hkls[h][:, :, None])[:, :, 0]
        q = q / q.norm(dim=1, keepdim=True)
        kf = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=_DEV) - 2 * q[:, 2:] * q
        d = kf @ rt.T
        x = ((d[:, 0] * pos[2] / d[:, 2] - pos[0]) / float(p.px_x) + 0.5 * (case["nx"] - 1)).trunc()
        y = ((d[:, 1] * pos[2] / d[:, 2] - pos[1]) / float(p.px_y) + 0.5 * (case["ny"] - 1)).trunc()
        ok = (d[:, 2] > 0) & (x >= 0) & (x < case["nx"]) & (y >= 0) & (y < case["ny"])
        o, pix = o[ok], (y[ok] * case["nx"] + x[ok]).long()
        key, order = torch.sort(o * (case["nx"] * case["ny"]) + pix, stable=True)
        first = torch.ones_like(key, dtype=torch.bool)
        first[1:] = key[1:] != key[:-1]
        at = torch.sort(order[first]).values  # the first of each pixel, in HKL order
        o, pix = o[at], pix[at]
        begin = torch.searchsorted(o, o)
        kept = torch.arange(len(o), device=_DEV) - begin < int(p.max_nr_spots)
        spots.append((o[kept] + i, pix[kept]))
    return torch.cat([s[0] for s in spots]), torch.cat([s[1] for s in spots])


def _records(o, pix, n, case):
    rec = np.zeros((n, 61), np.uint16)
    o, pix = o.cpu().numpy(), pix.cpu().numpy()
    at = np.arange(len(o)) - np.searchsorted(o, o)
    rec[:, 0] = np.bincount(o, minlength=n)
    rec[o, 1 + 2 * at] = pix % case["nx"]
    rec[o, 2 + 2 * at] = pix // case["nx"]
    return rec


def _match_exact(case, o, pix, frames):
    tot_all, score_all = [], []
    for img in frames:
        x = img.double().reshape(-1)
        mx = float(x.max())
        v = x * (255.0 / mx if mx > 0 else 0.0)
        u8 = torch.where(x > 0, torch.where(v < 1, 1.0, v.floor().clamp(max=255.0)), 0.0)
        val = (x.clamp(min=0) if case["exact_fp64_values"] else u8 * (mx / 255.0 if mx > 0 else 1.0))[pix]
        hit = val > 0
        ns = torch.zeros(case["n"], dtype=torch.float64, device=_DEV).index_add_(0, o[hit], torch.ones_like(val[hit]))
        tot = torch.zeros_like(ns).index_add_(0, o[hit], val[hit])
        ok = (ns >= case["min_spots"]) & (tot >= case["min_intensity"])
        tot_all.append(tot[ok])
        score_all.append(tot[ok] * ns[ok].sqrt())
    def padded(lists):
        v = torch.cat(lists)
        return torch.nn.functional.pad(v, (0, _room(case) - len(v)))
    return {"count": None, "n_pass": None, "id": None, "n_spots": None, "sum_u8": None,
            "tot_int": padded(tot_all), "score": padded(score_all)}


def _median_exact(img, size):
    """Square median of a frame of whole numbers with mirrored borders, by counting window values."""
    h = size // 2
    idx = [torch.as_tensor(np.pad(np.arange(n), h, mode="symmetric"), device=_DEV) for n in img.shape]
    wide = img[idx[0]][:, idx[1]]
    # bounds of every window's median from a coarse look at the values, then value by value
    out = torch.full(img.shape, -1.0, dtype=torch.float64, device=_DEV)
    need = size * size // 2 + 1
    for v in torch.unique(wide).tolist():
        s = torch.nn.functional.pad((wide <= v).double().cumsum(0).cumsum(1), (1, 0, 1, 0))
        cnt = s[size:, size:] - s[:-size, size:] - s[size:, :-size] + s[:-size, :-size]
        out = torch.where((out < 0) & (cnt >= need), float(v), out)
        if bool((out >= 0).all()):
            break
    return out


def _blur_exact(case, img, bg):
    """The blurred frame of a raw one: subtraction, threshold, small components removed, Gaussian."""
    sub = (img - bg).clamp(min=0)
    if case["method"] == "percentile":
        s = torch.sort(sub.reshape(-1)).values
        at = 0.99 * (len(s) - 1)
        lo = int(at)
        thr = float(s[lo] + (s[min(lo + 1, len(s) - 1)] - s[lo]) * (at - lo))
    else:
        nz = torch.sort(sub[sub > 0]).values
        def mid(s):
            return float((s[(len(s) - 1) // 2] + s[len(s) // 2]) / 2)
        med = mid(nz)
        thr = max(1.0, med + 4 * 1.4826 * mid(torch.sort((nz - med).abs()).values))
    t = torch.where(sub > thr, sub, 0.0).trunc()
    on = t > 0
    lab = torch.where(on, torch.arange(1, t.numel() + 1, device=_DEV, dtype=torch.float64).reshape(t.shape), 0.0)
    while True:
        new = torch.where(on, torch.nn.functional.max_pool2d(lab[None, None], 3, 1, 1)[0, 0], 0.0)
        if torch.equal(new, lab):
            break
        lab = new
    _, inv, area = torch.unique(lab, return_inverse=True, return_counts=True)
    big = area >= 10
    kept = int(big[torch.unique(inv[on])].sum())
    if kept == 0:
        return None
    t = torch.where(on & big[inv], t, 0.0)
    sigma = 1.0 if kept >= 2 else 3.0  # 0.2 mm pixels at 0.513: the spot spacing never widens it
    r = int(4 * sigma + 0.5)
    w = torch.exp(-0.5 / sigma ** 2 * torch.arange(-r, r + 1, device=_DEV, dtype=torch.float64) ** 2)
    w = w / w.sum()
    for axis in (0, 1):
        n = t.shape[axis]
        idx = torch.as_tensor(np.pad(np.arange(n), r, mode="symmetric"), device=_DEV)
        wide = t.index_select(axis, idx)
        t = sum(w[j] * wide.narrow(axis, j, n) for j in range(2 * r + 1))
    return t


def exact(case, seed):
    if case["kind"] == "cache":
        return None  # whole numbers only
    pairs = case["n"] * len(_hkls(case))
    if case["kind"] != "preprocess" and (case["n"] > HOST_ORIENTS or pairs > 4e10):
        return None  # the forward simulation alone would take longer than half a minute
    if case["kind"] == "preprocess":
        rec = _records(*_forward(case, _rotations(SCAN, seed)), SCAN, case)
        img = _frames(case, rec, seed)[0].double()
        out = _blur_exact(case, img, _median_exact(img, 101))
        out = torch.zeros_like(img) if out is None else out
        return {"blurred": out, "filt_img": None, "filt_labels": None, "centres": None}
    om = _rotations(case["n"], seed)
    o, pix = _forward(case, om)
    if case["kind"] == "fresh":
        rec = _records(*_forward(case, _rotations(SCAN, seed)), SCAN, case)
    else:
        scan = min(SCAN, case["n"])
        first = o < scan
        rec = _records(o[first], pix[first], scan, case)
    frames = _frames(case, rec, seed)
    if case["kind"] == "raw":
        bg = _median_exact(frames[0].double(), 101)
        blurred = [_blur_exact(case, f.double(), bg) for f in frames]
        frames = [b.float() for b in blurred if b is not None]
    return _match_exact(case, o, pix, frames)
