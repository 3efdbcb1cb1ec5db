"""Performance cases of the tracking front-end: the calls a visual-odometry program makes, from one
VGA frame's pyramid to a training step through the differentiable tracker.

Every case draws its scenes on the GPU from a seed (Gaussian blobs, four octaves of value noise, a
similarity warp between the frames, sensor noise, 8-bit quantisation) and takes its corners from
them with a plain Shi-Tomasi measure, so that no input depends on the code that is measured.

kinds of case
  pyramid   ImagePyramid.build / build_f32: image and gradient pyramid of one frame
  select    Selection.compute_gftt_and_select_features: new features beside the alive ones
  lk        LKFeatureTracker.track_points / track_mono on two built pyramids
  frame     one camera's whole frame through the plain calls: build, track, read back, top up
  rig       Batch: every camera's frame in one graph (optionally with retrack and finish filters)
  affine    STFeatureTracker / STFeatureTrackerWithCache
  l2r       StereoMatcher over rectified pairs with epipolar candidates
  diff      DiffTracker forward and backward through torch.autograd
"""

import functools
import math
import types

import numpy as np
import torch
import torch.nn.functional as F

from cuvslam_b200 import _lib
from cuvslam_b200.diff import DiffTracker
from cuvslam_b200.frontend import (Batch, CameraFrame, Context, ImagePyramid, LKFeatureTracker, Selection,
                                   STFeatureTracker, STFeatureTrackerWithCache, TrackFinish, track_mono,
                                   tracks_from_device, tracks_to_device)
from cuvslam_b200.stereo import EpipolarCurves, StereoMatcher, StereoPair
from cuvslam_b200.types import level_sizes, make_tracks

DEV = "cuda"

# The mixed rig of the benchmark: 12 VGA, 12 HD and 8 1920x1200 cameras.
RIG_SHAPES = {
    "mixed32": [(640, 480)] * 12 + [(1280, 720)] * 12 + [(1920, 1200)] * 8,
    "hd4": [(1280, 720)] * 4,
}


def listed():
    return [
        # The smallest call a program makes: one VGA camera's pyramid, where launches count.
        {"name": "pyramid_vga", "kind": "pyramid", "w": 640, "h": 480, "input": "u8", "blur": False, "levels": 10},
        # A colour camera with the box prefilter, at an odd size (no 16-byte row alignment).
        {"name": "pyramid_rgb_odd", "kind": "pyramid", "w": 1921, "h": 1201, "input": "rgb", "blur": True, "levels": 10},
        # Topping up an HD camera's features under a mask, half of them still alive.
        {"name": "select_hd", "kind": "select", "w": 1280, "h": 720, "alive": 600, "want": 1000, "mask": True},
        # One odometry frame of a KITTI-shaped camera (1241x376, 5 levels, 1000 features), plain calls.
        {"name": "frame_1241x376", "kind": "frame", "w": 1241, "h": 376, "n": 1000, "levels": 5},
        # Tracking a full-HD-plus camera with as many features as a dense front-end keeps.
        {"name": "lk_fhd_8k", "kind": "lk", "w": 1920, "h": 1200, "n": 8191, "call": "mono", "sampling": "hardware",
         "predicted": False},
        # The FP32 restatement of the texture filter (the mode that equals the CPU oracle), HD camera.
        {"name": "lk_texture_hd", "kind": "lk", "w": 1280, "h": 720, "n": 3000, "call": "track", "sampling": "texture",
         "predicted": True},
        # A four-camera robot: the batched frame with retrack and the finish filters.
        {"name": "rig_hd4_finish", "kind": "rig", "rig": "hd4", "cams": 4, "w": 1280, "h": 720, "nmin": 500,
         "nmax": 1500, "finish": True},
        # The 32-camera mixed-resolution rig of the benchmark.
        {"name": "rig_mixed32", "kind": "rig", "rig": "mixed32", "cams": 32, "w": 1920, "h": 1200, "nmin": 300,
         "nmax": 3000, "finish": False},
        # Affine tracking of every feature of a 1920x1200 camera, 20 full-map steps.
        {"name": "affine_fhd_8k", "kind": "affine", "w": 1920, "h": 1200, "n": 8191, "cached": False},
        # Left-to-right matching of an eight-pair rig.
        {"name": "l2r_8pairs", "kind": "l2r", "w": 752, "h": 480, "n": 512, "pairs": 8, "levels": 4},
        # Training through the tracker: implicit adjoint, eight HD cameras.
        {"name": "diff_implicit_hd8", "kind": "diff", "mode": "implicit", "b": 8, "w": 1280, "h": 720, "n": 4096},
        # Training through the tracker: unrolled steps, eight HD cameras.
        {"name": "diff_unrolled_hd8", "kind": "diff", "mode": "unrolled", "b": 8, "w": 1280, "h": 720, "n": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pyramid", "pyramid", "select", "lk", "lk", "frame", "rig", "rig", "affine", "l2r", "diff", "diff"])
    w = _log(rng, 320, 1930)
    h = max(120, int(w * rng.uniform(0.3, 0.75)))
    c = {"kind": kind, "w": w, "h": h}
    if kind == "pyramid":
        c |= {"input": rng.choice(["u8", "u8", "rgb", "f32"]), "levels": rng.choice([4, 5, 10])}
        c["blur"] = c["input"] != "f32" and rng.random() < 0.4
    elif kind == "select":
        c |= {"alive": rng.randrange(0, 1200), "want": _log(rng, 50, 4000), "mask": rng.random() < 0.5}
    elif kind == "lk":
        c |= {"n": _log(rng, 30, 8191), "call": rng.choice(["track", "track", "mono", "horizontal"]),
              "sampling": rng.choice(["hardware", "hardware", "texture", "wide", "exact"]),
              "predicted": rng.random() < 0.5}
    elif kind == "frame":
        c |= {"n": _log(rng, 100, 2000), "levels": rng.choice([4, 5, 10])}
    elif kind == "rig":
        c |= {"rig": "uniform", "cams": rng.randint(1, 12), "nmin": 50, "nmax": _log(rng, 200, 3000),
              "finish": rng.random() < 0.5}
    elif kind == "affine":
        c |= {"n": _log(rng, 30, 8191), "cached": rng.random() < 0.5}
    elif kind == "l2r":
        c |= {"w": rng.randint(400, 1000), "h": rng.randint(300, 600), "n": _log(rng, 50, 1000),
              "pairs": rng.randint(1, 8), "levels": rng.choice([4, 5])}
    else:
        c |= {"mode": rng.choice(["implicit", "unrolled"]), "b": rng.randint(1, 8), "w": min(w, 1280), "h": min(h, 720),
              "n": _log(rng, 64, 4096)}
    return c


# ---------------------------------------------------------------- scenes
def _gen(seed):
    return torch.Generator(DEV).manual_seed(int(seed))


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device=DEV) * (hi - lo) + lo


def _similarity(g, w, h):
    """(2, 3) matrix about the frame centre: t ~ N(0, 2) px, 1 degree, 1% scale."""
    u = torch.rand(2, generator=g, device=DEV)
    t = torch.randn(2, generator=g, device=DEV) * 2.0
    a, s = ((u[0] * 2 - 1) * math.pi / 180).item(), (0.99 + 0.02 * u[1]).item()
    m = np.array([[math.cos(a), -math.sin(a)], [math.sin(a), math.cos(a)]]) * s
    c = np.array([(w - 1) / 2, (h - 1) / 2])
    return m, c - m @ c + t.double().cpu().numpy()


def _apply(warp, xy):
    m, t = warp
    return xy @ torch.from_numpy(m.T).to(xy) + torch.from_numpy(t).to(xy)


def _frames(seed, w, h):
    """(base frame, its successor through a similarity warp): float intensities, and the warp."""
    g = _gen(seed)
    margin, nb = 96.0, 400
    bx, by = _uniform(g, (nb,), -margin, w + margin), _uniform(g, (nb,), -margin, h + margin)
    sigma, amp = _uniform(g, (nb,), 2, 20), _uniform(g, (nb,), -60, 60)
    lattices = []
    for o in range(4):
        cell = 64 / 2**o
        n = [int((d + 2 * margin) / cell) + 3 for d in (h, w)]
        lattices.append((cell, _uniform(g, n, -1, 1), 16.0 / 2**o))
    warp = _similarity(g, w, h)
    ys, xs = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32),
                            torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
    out = []
    for k in range(2):
        if k:
            m, t = warp
            inv = np.linalg.inv(m)
            off = -inv @ t
            px = xs * float(inv[0, 0]) + ys * float(inv[0, 1]) + float(off[0])
            py = xs * float(inv[1, 0]) + ys * float(inv[1, 1]) + float(off[1])
            cxy = _apply(warp, torch.stack([bx, by], 1))
            cx, cy, s = cxy[:, 0], cxy[:, 1], sigma * math.sqrt(abs(np.linalg.det(m)))
        else:
            px, py, cx, cy, s = xs, ys, bx, by, sigma
        ex = torch.exp(-((torch.arange(w, device=DEV) - cx[:, None]) / s[:, None]).square() / 2)
        ey = torch.exp(-((torch.arange(h, device=DEV) - cy[:, None]) / s[:, None]).square() / 2)
        img = 128.0 + (ey * amp[:, None]).T @ ex
        for cell, lat, a in lattices:
            u = ((px + margin) / cell).clamp(0, lat.shape[1] - 1.001)
            v = ((py + margin) / cell).clamp(0, lat.shape[0] - 1.001)
            i, j = u.floor(), v.floor()
            fu, fv = u - i, v - j
            fu, fv = fu * fu * (3 - 2 * fu), fv * fv * (3 - 2 * fv)
            o = j.long() * lat.shape[1] + i.long()
            flat = lat.reshape(-1)
            top = flat[o] * (1 - fu) + flat[o + 1] * fu
            bot = flat[o + lat.shape[1]] * (1 - fu) + flat[o + lat.shape[1] + 1] * fu
            img = img + a * (top * (1 - fv) + bot * fv)
        out.append(img)
    return out[0], out[1], warp


def _u8(img, g=None):
    if g is not None:
        img = img + 2.0 * torch.randn(img.shape, generator=g, device=DEV)
    return img.round().clamp(0, 255).to(torch.uint8)


def _pair(seed, w, h):
    """(previous u8 frame, next u8 frame with sensor noise, warp)."""
    a, b, warp = _frames(seed, w, h)
    return _u8(a), _u8(b, _gen(seed + 1)), warp


def _stereo_pair(seed, w, h):
    """(left u8, right u8, disparity of right pixels): the left view resampled at x + d, d 5-40 px."""
    a, _, _ = _frames(seed, w, h)
    g = _gen(seed + 2)
    d = F.interpolate(_uniform(g, (1, 1, h // 32 + 3, w // 32 + 3), 5, 40), size=(h, w), mode="bicubic",
                      align_corners=True)[0, 0].clamp(2, 45)
    xs = torch.arange(w, device=DEV) + d
    grid = torch.stack([xs / (w - 1) * 2 - 1,
                        (torch.arange(h, device=DEV) / (h - 1) * 2 - 1)[:, None].expand(h, w)], -1)[None]
    right = F.grid_sample(a[None, None], grid, padding_mode="border", align_corners=True)[0, 0]
    return _u8(a), _u8(right, g), d


def _corners(img, n, seed):
    """n corners (texture coordinates, at sub-pixel places): the best pixel of every cell by the
    smaller eigenvalue of the structure tensor, strongest cells first, repeated if there are too few."""
    h, w = img.shape
    f = F.pad(img.float()[None, None], (1, 1, 1, 1), mode="replicate")
    gx, gy = (f[..., 1:-1, 2:] - f[..., 1:-1, :-2]) / 2, (f[..., 2:, 1:-1] - f[..., :-2, 1:-1]) / 2
    xx, yy, xy = (F.avg_pool2d(p, 7, 1, 3) for p in (gx * gx, gy * gy, gx * gy))
    e = (xx + yy) / 2 - torch.sqrt((xx - yy).square() / 4 + xy * xy)
    e[..., :8, :] = e[..., -8:, :] = 0
    e[..., :, :8] = e[..., :, -8:] = 0
    cell = max(3, int(math.sqrt(w * h / (1.3 * max(n, 1)))))
    v, at = F.max_pool2d(e, cell, cell, return_indices=True)
    at = at.reshape(-1)[torch.argsort(v.reshape(-1), descending=True, stable=True)][:n]
    p = torch.stack([at % w, at // w], 1).float() + 0.5
    p = p + _uniform(_gen(seed + 3), p.shape, -0.5, 0.5)
    return p.repeat(-(-n // max(len(p), 1)), 1)[:n].contiguous()


def _records(xy, off, radius, ncc=0.8):
    return make_tracks(xy.cpu().numpy(), None if off is None else off.cpu().numpy(), float(radius), ncc)


SAMPLINGS = {"hardware": _lib.FE_SAMPLE_HARDWARE, "texture": _lib.FE_SAMPLE_TEXTURE,
             "wide": _lib.FE_SAMPLE_TEXTURE_WIDE, "exact": _lib.FE_SAMPLE_EXACT}


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    s = types.SimpleNamespace(case=case, ctx=Context(0))
    _PREPARE[case["kind"]](s, case, seed * 1009)
    return s


def _planes(p):
    """Views of every level's image and gradients: what a pyramid's user reads."""
    return [[p.image(l), p.grad_x(l), p.grad_y(l)] for l in range(p.levels)]


def _fields(tracks):
    """A record buffer's results: positions, the 2x2 information and the status."""
    f = tracks.view(torch.float32)
    return {"xy": f[:, 0:2], "info": f[:, 4:8], "status": tracks[:, 32]}


def _pyramid_input(c, seed):
    a, _, _ = _pair(seed, c["w"], c["h"])
    if c["input"] == "rgb":
        g = _gen(seed + 5)
        return torch.stack([_u8(a.float() + o, g) for o in (-6.0, 0.0, 9.0)], -1).contiguous()
    return a.float() / 255.0 if c["input"] == "f32" else a


def _prepare_pyramid(s, c, seed):
    s.image = _pyramid_input(c, seed)
    s.pyr = ImagePyramid(c["w"], c["h"], c["levels"])
    s.out = _planes(s.pyr)


def _prepare_select(s, c, seed):
    a, b, warp = _pair(seed, c["w"], c["h"])
    s.pyr = ImagePyramid(c["w"], c["h"]).build(s.ctx, b)
    s.sel = Selection(s.ctx)
    s.new = torch.zeros((c["want"], 2), device=DEV)
    s.alive = _apply(warp, _corners(a, c["alive"], seed)) if c["alive"] else None
    s.mask = None
    if c["mask"]:  # the robot's own body covers the lower corners of the view
        ys, xs = torch.meshgrid(torch.arange(c["h"], device=DEV), torch.arange(c["w"], device=DEV), indexing="ij")
        s.mask = ((ys > 0.8 * c["h"]) & ((xs - c["w"] / 2).abs() > 0.3 * c["w"])).to(torch.uint8)


def _lk_inputs(c, seed):
    w, h = c["w"], c["h"]
    g = _gen(seed + 7)
    if c["call"] == "horizontal":
        a, b, d = _stereo_pair(seed, w, h)
        xy = _corners(a, c["n"], seed)
        near = d[xy[:, 1].long().clamp(0, h - 1), xy[:, 0].long().clamp(0, w - 1)]
        off = torch.stack([-near + torch.randn(len(near), generator=g, device=DEV), torch.zeros_like(near)], 1)
    else:
        a, b, warp = _pair(seed, w, h)
        xy = _corners(a, c["n"], seed)
        off = None
        if c["predicted"]:
            off = _apply(warp, xy) - xy + torch.randn(xy.shape, generator=g, device=DEV)
    return a, b, xy, off


def _prepare_lk(s, c, seed):
    a, b, xy, off = _lk_inputs(c, seed)
    s.prev, s.cur = ImagePyramid(c["w"], c["h"]).build(s.ctx, a), ImagePyramid(c["w"], c["h"]).build(s.ctx, b)
    s.records = tracks_to_device(_records(xy, off, c["w"]))
    s.tracks = s.records.clone()
    s.out = _fields(s.tracks)
    s.lk = LKFeatureTracker(s.ctx, c["call"] == "horizontal", SAMPLINGS[c["sampling"]])


def _prepare_frame(s, c, seed):
    a, s.image, _ = _pair(seed, c["w"], c["h"])
    s.prev = ImagePyramid(c["w"], c["h"], c["levels"]).build(s.ctx, a)
    s.cur = ImagePyramid(c["w"], c["h"], c["levels"])
    s.records = _records(_corners(a, c["n"], seed), None, c["w"])
    s.planes = _planes(s.cur)
    s.new = torch.zeros((c["n"], 2), device=DEV)
    s.lk, s.sel = LKFeatureTracker(s.ctx), Selection(s.ctx)


def _rig_cameras(c, seed):
    """[(w, h, features, seed)] of a rig."""
    shapes = RIG_SHAPES.get(c["rig"]) or [(c["w"], c["h"])] * c["cams"]
    n = torch.randint(c["nmin"], c["nmax"] + 1, (len(shapes),), generator=torch.Generator().manual_seed(77)).tolist()
    return [(w, h, k, seed + 31 * i) for i, ((w, h), k) in enumerate(zip(shapes, n))]


def _prepare_rig(s, c, seed):
    cams = _rig_cameras(c, seed)
    recs, views = [], []
    for w, h, n, sd in cams:
        a, b, _ = _pair(sd, w, h)
        recs.append(tracks_to_device(_records(_corners(a, n, sd), None, w)))
        views.append((b, ImagePyramid(w, h), ImagePyramid(w, h).build(s.ctx, a)))
    at = np.cumsum([0] + [k for _, _, k, _ in cams])
    # one buffer for every camera's tracks, new features, counts and ages, as a capture loop keeps them
    s.records = torch.cat(recs)
    s.tracks = s.records.clone()
    s.new_xy = torch.zeros((int(at[-1]), 2), device=DEV)
    s.new_count = torch.zeros(len(cams), dtype=torch.int32, device=DEV)
    s.age0 = torch.randint(1, 30, (int(at[-1]),), generator=_gen(seed + 9), device=DEV, dtype=torch.int32)
    s.age = s.age0.clone()
    s.frames = []
    for i, (img, cur, prev) in enumerate(views):
        lo, hi = int(at[i]), int(at[i + 1])
        fin = TrackFinish(s.age[lo:hi]) if c["finish"] else None
        f = CameraFrame(img, cur, prev, s.tracks[lo:hi], hi - lo, (0, 0, 0, 0), finish=fin)
        f.new_xy, f.new_count = s.new_xy[lo:hi], s.new_count[i:i + 1]
        s.frames.append(f)
    s.batch = Batch(s.ctx, s.frames)
    s.batch.autotune()
    s.new_xy.zero_()
    s.out = {**_fields(s.tracks), "new": s.new_xy, "count": s.new_count, "age": s.age,
             "top": [f.cur.image(f.cur.levels - 1) for f in s.frames]}


def _prepare_affine(s, c, seed):
    a, b, warp = _pair(seed, c["w"], c["h"])
    s.prev, s.cur = ImagePyramid(c["w"], c["h"]).build(s.ctx, a), ImagePyramid(c["w"], c["h"]).build(s.ctx, b)
    xy = _corners(a, c["n"], seed)
    off = _apply(warp, xy) - xy + 0.5
    s.records = tracks_to_device(_records(xy, off, 64.0))
    s.tracks = s.records.clone()
    s.out = _fields(s.tracks)
    s.st = (STFeatureTrackerWithCache if c["cached"] else STFeatureTracker)(s.ctx)


@functools.lru_cache(maxsize=None)
def _epipolar_table(w, h, lv):
    """The rig's calibration, which a program reads once: focal 458 px at 752 px width, 11 cm baseline."""
    sizes = level_sizes(w, h, lv)
    top = len(sizes) - 1
    k = (458.0 * w / 752, 458.0 * w / 752, w / 2 - 9, h / 2 + 8)
    return EpipolarCurves.pinhole(k, k, (np.eye(3), (-0.11, 0.0, 0.0)), top, *sizes[top])


def _prepare_l2r(s, c, seed):
    w, h, lv = c["w"], c["h"], c["levels"]
    s.curves = _epipolar_table(w, h, lv)
    s.pairs = []
    for i in range(c["pairs"]):
        a, b, _ = _stereo_pair(seed + 31 * i, w, h)
        s.pairs.append(StereoPair(ImagePyramid(w, h, lv).build(s.ctx, a), ImagePyramid(w, h, lv).build(s.ctx, b),
                                  _corners(a, c["n"], seed + 31 * i), curves=s.curves))
    s.matcher = StereoMatcher(s.ctx)


def _diff_inputs(c, seed):
    prev, cur, xy = [], [], []
    for i in range(c["b"]):
        a, b, _ = _pair(seed + 31 * i, c["w"], c["h"])
        prev.append(a.float() / 255)
        cur.append(b.float() / 255)
        xy.append(_corners(a, c["n"], seed + 31 * i))
    xy = torch.stack(xy)
    g = _gen(seed + 11)
    off = 0.5 * torch.randn(xy.shape, generator=g, device=DEV)
    return torch.stack(prev), torch.stack(cur), xy, off, torch.randn(xy.shape, generator=g, device=DEV) / xy.shape[1]


def _prepare_diff(s, c, seed):
    *leaves, s.grad = _diff_inputs(c, seed)
    s.leaves = [v.requires_grad_() for v in leaves]
    s.tracker = DiffTracker(s.ctx, c["b"], c["h"], c["w"], c["n"], mode=c["mode"])


_PREPARE = {"pyramid": _prepare_pyramid, "select": _prepare_select, "lk": _prepare_lk, "frame": _prepare_frame,
            "rig": _prepare_rig, "affine": _prepare_affine, "l2r": _prepare_l2r, "diff": _prepare_diff}


# ---------------------------------------------------------------- run
def run(state):
    return _RUN[state.case["kind"]](state)


def _run_pyramid(s):
    if s.case["input"] == "f32":
        s.pyr.build_f32(s.ctx, s.image)
    else:
        s.pyr.build(s.ctx, s.image, blur_filter=s.case["blur"])
    return s.out


def _run_select(s):
    new = s.sel.compute_gftt_and_select_features(s.pyr, 4, 4, 4, 4, s.mask, s.alive, s.case["want"])
    s.new[: len(new)] = new
    return [s.new, len(new)]


def _run_lk(s):
    s.tracks.copy_(s.records)
    if s.case["call"] == "mono":
        track_mono(s.ctx, s.prev, s.cur, s.tracks, sampling=SAMPLINGS[s.case["sampling"]])
    else:
        s.lk.track_points(s.prev, s.cur, s.tracks)
    return s.out


def _run_frame(s):
    s.cur.build(s.ctx, s.image)
    tracks = tracks_to_device(s.records)
    s.lk.track_points(s.prev, s.cur, tracks)
    out = tracks_from_device(tracks)
    ok = out["track_status"] == 1
    new = s.sel.compute_gftt_and_select_features(s.cur, 0, 0, 0, 0, None, out["track"][ok],
                                                 max(0, s.case["n"] - int(ok.sum())))
    s.new[: len(new)] = new
    return {"xy": out["track"], "status": out["track_status"], "new": s.new, "count": len(new), "cur": s.planes}


def _run_rig(s):
    s.tracks.copy_(s.records)
    if s.case["finish"]:
        s.age.copy_(s.age0)
    s.batch.run()
    return s.out


def _run_affine(s):
    s.tracks.copy_(s.records)
    if s.case["cached"]:
        s.st.track_points(s.cur, s.st.build_points_cache(s.prev, s.tracks), s.tracks)
    else:
        s.st.track_points(s.prev, s.cur, s.tracks)
    return s.out


def _run_l2r(s):
    out = s.matcher.track_primary_to_secondary(s.pairs)
    return [{"xy": t.view(torch.float32)[:, 0:2], "status": t[:, 32], "winner": w} for t, w, _ in out]


def _run_diff(s):
    pos, status = s.tracker(*s.leaves)
    return [pos.detach(), status, *torch.autograd.grad(pos, s.leaves, s.grad)]


_RUN = {"pyramid": _run_pyramid, "select": _run_select, "lk": _run_lk, "frame": _run_frame, "rig": _run_rig,
        "affine": _run_affine, "l2r": _run_l2r, "diff": _run_diff}


# ---------------------------------------------------------------- work
def _pyr_px(w, h, levels=10):
    return sum(a * b for a, b in level_sizes(w, h, levels))


def _lk_work(w, h, n, levels=10, planes=4):
    """Bytes and operations of tracking n points: per level the 10x10 texels under the patch from
    every plane that is read (or the whole plane where the patches overlap that much), 81 taps of
    each plane (7 operations a sample), the template's moments, and about two steps."""
    sizes = level_sizes(w, h, levels)
    b = sum(min(400.0 * n, 4.0 * a * d) * planes for a, d in sizes)
    return b + 160.0 * n, float(n) * len(sizes) * 81 * (3 * 7 + 15 + 2 * (7 + 10))


def work(case):
    c = case
    w, h, k = c["w"], c["h"], c["kind"]
    if k == "pyramid":
        px = _pyr_px(w, h, c["levels"])
        b = w * h * {"u8": 1, "rgb": 3, "f32": 4}[c["input"]] + 12 * px
        f = 36 * px
    elif k == "select":
        b, f = 8 * w * h + 8 * (c["alive"] + c["want"]), 80 * w * h
    elif k == "lk":
        b, f = _lk_work(w, h, c["n"], planes=3 if c["call"] == "horizontal" else 4)
    elif k == "frame":
        px = _pyr_px(w, h, c["levels"])
        b, f = _lk_work(w, h, c["n"], c["levels"])
        b, f = w * h + 12 * px + b, 36 * px + f + 80 * w * h
    elif k == "rig":
        b = f = 0.0
        for cw, ch, n, _ in _rig_cameras(c, 0):
            px = _pyr_px(cw, ch)
            lb, lf = _lk_work(cw, ch, n)
            b += cw * ch + 12 * px + lb
            f += 36 * px + lf + 80 * cw * ch
    elif k == "affine":
        b, f = _lk_work(w, h, c["n"])
        f = float(c["n"]) * 4 * 81 * 10 * (3 * 7 + 60)
    elif k == "l2r":
        b, f = _lk_work(w, h, c["n"], c["levels"], 3)
        b, f = c["pairs"] * b, c["pairs"] * 3 * f
    else:
        px = _pyr_px(w, h)
        lb, lf = _lk_work(w, h, c["n"])
        steps = 1 if c["mode"] == "implicit" else 5
        # two frames in, their pyramids out and read by both passes, two image gradients out
        b = c["b"] * (2 * 4 * w * h + 2 * 12 * px + 2 * lb + 2 * 4 * w * h)
        f = c["b"] * (2 * 36 * px + 3 * steps * lf)
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------- the same in 64 bits
# Selection picks pixels, the matcher candidates and the affine tracker's pivoted solve branches on its
# last bits: their outputs have no value in 64 bits that a 32-bit run approaches.  Images and
# tracked positions have one.
D64 = torch.float64


def _mirrored(n, r):
    i = torch.arange(-r, n + r, device=DEV)
    i = torch.where(i < 0, -i - 1, i)
    return torch.where(i >= n, 2 * n - i - 1, i).clamp(0, n - 1)


def _down64(img):
    """5x5 binomial at even pixels, mirrored edges; taps outside on both axes are left out."""
    h, w = img.shape
    k = torch.tensor([1.0, 4, 6, 4, 1], dtype=D64, device=DEV) / 16
    iy, ix = _mirrored(h, 2), _mirrored(w, 2)
    p = img[iy][:, ix]
    oy = torch.ones(h + 4, 1, dtype=D64, device=DEV)
    ox = torch.ones(1, w + 4, dtype=D64, device=DEV)
    oy[:2] = oy[-2:] = 0
    ox[:, :2] = ox[:, -2:] = 0
    p = p * torch.maximum(oy, ox)
    return F.conv2d(p[None, None], torch.outer(k, k)[None, None], stride=2)[0, 0][:(h + 1) // 2, :(w + 1) // 2]


def _grads64(img):
    h, w = img.shape
    k = torch.tensor([112.0, 913, 3047, 0, -3047, -913, -112], dtype=D64, device=DEV) / 8418
    gx = F.pad(F.conv2d(img[None, None], k.view(1, 1, 1, 7)), (3, 3, 0, 0))[0, 0]
    gy = F.pad(F.conv2d(img[None, None], k.view(1, 1, 7, 1)), (0, 0, 3, 3))[0, 0]
    return gx, gy


def _pyramid64(img, levels=10):
    out = []
    for i, _ in enumerate(level_sizes(img.shape[1], img.shape[0], levels)):
        img = _down64(img) if i else img
        out.append([img, *_grads64(img)])
    return out


def _bilinear64(plane, x, y):
    """Texture-coordinate samples (texel i covers [i, i + 1)) with clamped edges, and the fractions."""
    h, w = plane.shape
    u, v = x - 0.5, y - 0.5
    i, j = u.floor(), v.floor()
    fu, fv = u - i, v - j
    i0, i1 = i.long().clamp(0, w - 1), (i.long() + 1).clamp(0, w - 1)
    j0, j1 = j.long().clamp(0, h - 1) * w, (j.long() + 1).clamp(0, h - 1) * w
    flat = plane.reshape(-1)

    def at(o):
        return torch.gather(flat, 0, o.reshape(-1)).view(o.shape)

    a, b, c, d = at(j0 + i0), at(j0 + i1), at(j1 + i0), at(j1 + i1)
    ax, bx = b - a, d - c
    top, bot = a + fu * ax, c + fu * bx
    return top + fv * (bot - top), ax + fv * (bx - ax), bot - top


_G9 = [0.0135196, 0.0476622, 0.11723, 0.201168, 0.240841, 0.201168, 0.11723, 0.0476622, 0.0135196]


def _lk64(prev, cur, xy, off, radius, ncc_thr, horizontal=False, mode="reference"):
    """Pyramidal Lucas-Kanade of all points at once; (positions, kept).  mode: the reference rule (at
    most 11 steps a level, until one is below 0.12 px), "implicit" (then Newton steps to the fixed
    point at level 0), "unrolled" (10 steps a level)."""
    G = torch.tensor(_G9, dtype=D64, device=DEV)
    wt = torch.outer(G, G).reshape(1, 81)
    dx = torch.arange(9, device=DEV, dtype=D64).repeat(9)[None] - 4
    dy = torch.arange(9, device=DEV, dtype=D64).repeat_interleave(9)[None] - 4
    inner = ((dx.abs() <= 2) & (dy.abs() <= 2)).reshape(-1)
    h0, w0 = prev[0][0].shape
    top = len(prev) - 1
    ok0 = (xy[:, 0] >= 0) & (xy[:, 0] < w0) & (xy[:, 1] >= 0) & (xy[:, 1] < h0)
    end = xy + off
    ok0 = ok0 & (end[:, 0] >= 0) & (end[:, 0] < w0) & (end[:, 1] >= 0) & (end[:, 1] < h0)
    s, c = (xy - 0.5) / 2**top + 0.5, (end - 0.5) / 2**top + 0.5

    def inside(p, w, h):
        return (p[:, 0] >= 4) & (p[:, 0] + 5 < w) & (p[:, 1] >= 4) & (p[:, 1] + 5 < h)

    def patch(plane, p):
        return _bilinear64(plane, p[:, :1] + dx, p[:, 1:] + dy)

    kept = torch.zeros(len(xy), dtype=torch.bool, device=DEV)
    for level in range(top, -1, -1):
        pi, pgx, pgy = prev[level]
        ci = cur[level][0]
        h, w = ci.shape
        good = ok0 & inside(s, w, h)
        p1, gx = patch(pi, s)[0], patch(pgx, s)[0]
        gx = gx - gx.mean(1, keepdim=True)
        gy = torch.zeros_like(gx)
        if not horizontal:
            gy = patch(pgy, s)[0]
            gy = gy - gy.mean(1, keepdim=True)
        a, b, d = 1 + (wt * gx * gx).sum(1), (wt * gx * gy).sum(1), 1 + (wt * gy * gy).sum(1)
        det = a if horizontal else a * d - b * b
        ok0 = ok0 & (~good | (det >= 1.1920928955078125e-07))
        good = good & ok0
        start, conv, live = c, torch.zeros_like(good), good.clone()
        p2 = torch.zeros_like(p1)
        for _ in range(10 if mode == "unrolled" else 11):
            live = live & inside(c, w, h)
            if mode == "unrolled":
                good = good & live
            q = patch(ci, torch.where(live[:, None], c, s))[0]
            p2 = torch.where(live[:, None], q, p2)
            r = wt * (q - p1 - (q - p1).mean(1, keepdim=True))
            ex, ey = (r * gx).sum(1), (r * gy).sum(1)
            v = torch.stack([ex / a, 0 * ex], 1) if horizontal else \
                torch.stack([(d * ex - b * ey) / det, (a * ey - b * ex) / det], 1)
            small = v.square().sum(1) < 0.12**2
            if mode == "unrolled":
                conv = small & good
            else:
                conv = conv | (live & small)
                live = live & ~small
            c = torch.where(live[:, None], c + v, c)
        conv = conv & good & ((c - start).square().sum(1) <= (radius / 2**level)**2)
        u1, u2 = p1[:, inner], p2[:, inner]
        m1, m2 = u1.mean(1), u2.mean(1)
        vv = ((u1 * u1).mean(1) - m1 * m1) * ((u2 * u2).mean(1) - m2 * m2)
        ncc = ((u1 * u2).mean(1) - m1 * m2) / vv.clamp_min(1e-30).sqrt()
        conv = conv & (vv >= 1.1920928955078125e-07) & (ncc > ncc_thr)
        if level:
            c = torch.where((good & ~conv)[:, None], start, c)
            s, c = s * 2 - 0.5, c * 2 - 0.5
        else:
            kept = conv
    if mode == "implicit":
        def newton(at):
            q, qx, qy = patch(cur[0][0], at)
            r = wt * (q - p1 - (q - p1).mean(1, keepdim=True))
            e = torch.stack([(r * gx).sum(1), (r * gy).sum(1)], 1)
            qx, qy = qx - qx.mean(1, keepdim=True), qy - qy.mean(1, keepdim=True)
            j = torch.stack([(wt * gx * qx).sum(1), (wt * gx * qy).sum(1), (wt * gy * qx).sum(1),
                             (wt * gy * qy).sum(1)], 1).view(-1, 2, 2)
            dj = torch.where(torch.linalg.det(j).abs() > 0, torch.linalg.det(j), torch.ones_like(j[:, 0, 0]))
            v = -torch.stack([j[:, 1, 1] * e[:, 0] - j[:, 0, 1] * e[:, 1],
                              j[:, 0, 0] * e[:, 1] - j[:, 1, 0] * e[:, 0]], 1) / dj[:, None]
            return v, j, dj

        first, live, settled = c.clone(), kept.clone(), torch.zeros_like(kept)
        for _ in range(20):
            live = live & inside(c, w, h)
            v, j, dj = newton(torch.where(live[:, None], c, s))
            n2 = v.square().sum(1)
            live = live & (n2 <= 4)
            c = torch.where(live[:, None], c + v, c)
            live = live & ((c - first).square().sum(1) <= 4)
            done = live & (n2 < 1e-8)
            settled = settled | (done & (dj.abs() >= 0.01 * j.square().sum((1, 2))))
            live = live & ~done
        kept = settled
    kept = kept & ok0
    return torch.where(kept[:, None], c, xy), kept


def _exact_pyramid(c, seed):
    img = _pyramid_input(c, seed).to(D64)
    if c["input"] == "rgb":
        img = img @ torch.tensor([0.299, 0.587, 0.114], dtype=D64, device=DEV)
        if c["blur"]:
            return None  # the prefilter truncates to whole numbers
    if c["blur"]:
        k = torch.tensor([1.0, 2, 1], dtype=D64, device=DEV) / 4
        out = img.clone()
        out[1:-1, 1:-1] = F.conv2d(img[None, None], torch.outer(k, k)[None, None])[0, 0].floor()
        img = out
    return _pyramid64(img, c["levels"])


def _exact_lk(c, seed):
    a, b, xy, off = _lk_inputs(c, seed)
    prev, cur, xy = _pyramid64(a.to(D64)), _pyramid64(b.to(D64)), xy.to(D64)
    off = torch.zeros_like(xy) if off is None else off.to(D64)
    pos, kept = _lk64(prev, cur, xy, off, float(c["w"]), 0.8, c["call"] == "horizontal")
    if c["call"] == "mono":
        again, also = _lk64(prev, cur, xy, off, float(c["w"]), 0.85)
        pos = torch.where((also & ~kept)[:, None], again, pos)
    return {"xy": pos, "info": None, "status": None}


def _exact_frame(c, seed):
    a, b, _ = _pair(seed, c["w"], c["h"])
    prev, cur = _pyramid64(a.to(D64), c["levels"]), _pyramid64(b.to(D64), c["levels"])
    xy = _corners(a, c["n"], seed).to(D64)
    pos = _lk64(prev, cur, xy, torch.zeros_like(xy), float(c["w"]), 0.8)[0]
    return {"xy": pos, "status": None, "new": None, "count": None, "cur": cur}


def _exact_rig(c, seed):
    xy_out, top = [], []
    for w, h, n, sd in _rig_cameras(c, seed):
        a, b, _ = _pair(sd, w, h)
        prev, cur, xy = _pyramid64(a.to(D64)), _pyramid64(b.to(D64)), _corners(a, n, sd).to(D64)
        pos, kept = _lk64(prev, cur, xy, torch.zeros_like(xy), float(w), 0.8)
        if c["finish"]:
            again, also = _lk64(prev, cur, xy, torch.zeros_like(xy), float(w), 0.85)
            pos = torch.where((also & ~kept)[:, None], again, pos)
        xy_out.append(pos)
        top.append(cur[-1][0])
    return {"xy": torch.cat(xy_out), "info": None, "status": None, "new": None, "count": None, "age": None, "top": top}


def _exact_diff(c, seed):
    # The gradients are dominated by the few tracks near a texel's edge or a gate's limit, where the last
    # bits of a position decide between two derivatives: only the positions are given.
    prev, cur, xy, off, _ = _diff_inputs(c, seed)
    pos = [_lk64(_pyramid64(prev[b].to(D64) * 255), _pyramid64(cur[b].to(D64) * 255), xy[b].to(D64), off[b].to(D64),
                 2048.0, 0.8, False, c["mode"])[0] for b in range(c["b"])]
    return [torch.stack(pos), None, None, None, None, None]


_EXACT = {"pyramid": _exact_pyramid, "lk": _exact_lk, "frame": _exact_frame, "rig": _exact_rig, "diff": _exact_diff}


def exact(case, seed):
    fn = _EXACT.get(case["kind"])
    return fn(case, seed * 1009) if fn else None
