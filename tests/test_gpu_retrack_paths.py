"""The retrack pass in every sampling, with forks of every kind shown to occur, and in a batch that mixes cameras
with and without one; the adjoint's tile sums with tracks shown to carry gradient."""

import numpy as np
import pytest
import torch

from conftest import assert_tracks_equal
from cuvslam_b200 import _lib, synthetic
from cuvslam_b200.diff import DiffTracker
from cuvslam_b200.frontend import (Batch, CameraFrame, ImagePyramid, LKFeatureTracker, TrackFinish, track_mono,
                                   tracks_from_device, tracks_to_device)
from cuvslam_b200.types import make_tracks

pytestmark = pytest.mark.gpu

SAMPLINGS = [_lib.FE_SAMPLE_HARDWARE, _lib.FE_SAMPLE_TEXTURE, _lib.FE_SAMPLE_TEXTURE_WIDE, _lib.FE_SAMPLE_EXACT]


def _tracked(ctx, pa, pb, recs, threshold, sampling):
    r = recs.copy()
    r["ncc_threshold"] = threshold
    t = tracks_to_device(r)
    LKFeatureTracker(ctx, False, sampling).track_points(pa, pb, t)
    torch.cuda.synchronize()
    return tracks_from_device(t)


def _two_passes(ctx, pa, pb, recs, first, second, sampling):
    """The definition: (records, tracks that the second pass kept, tracks that it lost too)."""
    want, again = _tracked(ctx, pa, pb, recs, first, sampling), _tracked(ctx, pa, pb, recs, second, sampling)
    lost = (want["track_status"] == 0) & (recs["search_radius_px"] >= 0)
    for name in want.dtype.names:
        if name != "ncc_threshold":
            want[name][lost] = again[name][lost]
    return want, int((lost & (again["track_status"] == 1)).sum()), int((lost & (again["track_status"] == 0)).sum())


# gained: whether tracks must come back through the second threshold
@pytest.mark.parametrize("sampling", SAMPLINGS)
@pytest.mark.parametrize("first,second,gained", [(0.95, 0.5, True), (0.8, 0.85, False), (0.999, 0.9, True), (0.5, 0.999, False),
                                                 (2.0, 0.7, True), (0.8, 0.8, False)])
def test_every_sampling(ctx, sampling, first, second, gained):
    a, b, _ = synthetic.frame_pair(35, 640, 480)
    pa = ImagePyramid(640, 480).build(ctx, torch.from_numpy(a).cuda())
    pb = ImagePyramid(640, 480).build(ctx, torch.from_numpy(b).cuda())
    rng = np.random.default_rng(8)
    xy = rng.uniform((-3, -3), (643, 483), (1500, 2)).astype(np.float32)
    recs = make_tracks(xy, rng.normal(0, 3, (1500, 2)), 60.0, first)
    recs["search_radius_px"][::97] = -1.0
    got = tracks_to_device(recs)
    track_mono(ctx, pa, pb, got, retrack_ncc=second, sampling=sampling)
    torch.cuda.synchronize()
    want, back, gone = _two_passes(ctx, pa, pb, recs, first, second, sampling)
    assert gone > 0 and (back > 20 if gained else True)
    assert_tracks_equal(tracks_from_device(got), want)


@pytest.mark.parametrize("sampling", SAMPLINGS)
def test_batch_with_and_without_a_second_pass(ctx, sampling):
    """Cameras with another threshold each, one without finish filters (no second pass), one whose second pass has no
    threshold (0): each equals its two passes, or its one."""
    seconds = [0.5, None, 0.0, 0.9]
    frames, hosts, pyrs = [], [], []
    for i, second in enumerate(seconds):
        a, b, _ = synthetic.frame_pair(60 + i, 320, 240)
        pa = ImagePyramid(320, 240).build(ctx, torch.from_numpy(a).cuda())
        rng = np.random.default_rng(i)
        xy = rng.uniform((4, 4), (316, 236), (300, 2)).astype(np.float32)
        recs = make_tracks(xy, rng.normal(0, 2, (300, 2)), 60.0, 0.95)
        fin = None
        if second is not None:
            fin = TrackFinish(torch.ones(300, dtype=torch.int32, device="cuda"), retrack_ncc=second, collapse=False)
        frames.append(CameraFrame(torch.from_numpy(b).cuda(), ImagePyramid(320, 240), pa, tracks_to_device(recs), 0,
                                  finish=fin))
        hosts.append(recs)
        pyrs.append((pa, ImagePyramid(320, 240).build(ctx, torch.from_numpy(b).cuda())))
    batch = Batch(ctx, frames, sampling)
    backs = []
    for f, recs in zip(frames, hosts):  # the LK part alone, before the filters
        f.tracks.copy_(tracks_to_device(recs))
    batch.run_part(0)
    batch.run_part(1)
    torch.cuda.synchronize()
    for f, recs, (pa, pb), second in zip(frames, hosts, pyrs, seconds):
        if second:
            want, back, _ = _two_passes(ctx, pa, pb, recs, 0.95, second, sampling)
            backs.append(back)
        else:
            want = _tracked(ctx, pa, pb, recs, 0.95, sampling)
        assert_tracks_equal(tracks_from_device(f.tracks), want)
    assert max(backs) > 5
    batch.close()


@pytest.mark.parametrize("mode", ["implicit", "unrolled"])
def test_repeated_tracks_carry_gradient(ctx, mode):
    """Forty copies of each track: forty times the images' gradient within 64 roundings of the largest, with every
    kind of track (its patch over a power of two among them) shown to be tracked and to have one."""
    w, h = 161, 129
    prev, cur, _ = synthetic.frame_pair(51, w, h)
    rng = np.random.default_rng(1)
    grid = rng.uniform((8, 8), (w - 8, h - 8), (40, 2)).astype(np.float32)
    grid[:6] = [(32.3, 31.6), (63.7, 16.2), (16.1, 33.4), (64.2, 64.3), (33.1, 64.7), (128.2, 32.1)]
    g1 = rng.normal(size=(1, 40, 2)).astype(np.float32)

    def run(xy, g):
        t = DiffTracker(ctx, 1, h, w, len(xy), mode=mode)
        p, c = (torch.from_numpy(v.astype(np.float32) / 255)[None].cuda().requires_grad_() for v in (prev, cur))
        q = torch.from_numpy(xy)[None].cuda().requires_grad_()
        pos, st = t(p, c, q)
        grads = torch.autograd.grad(pos, (p, c, q), torch.from_numpy(g).cuda())
        out = st.cpu().numpy()[0], [v.cpu().numpy()[0] for v in grads]
        t.close()
        return out

    st1, one = run(grid, g1)
    st40, many = run(np.repeat(grid, 40, 0), np.repeat(g1, 40, 1))
    assert st1[:6].any() and st1[6:].any() and np.array_equal(np.repeat(st1, 40), st40)
    for a, b in zip(one[:2], many[:2]):
        scale = np.abs(a).max()
        assert scale > 0
        assert np.abs(b / 40 - a).max() <= 64 * 2.0**-23 * scale * len(grid)
    assert np.abs(one[2][st1]).max() > 0 and np.array_equal(np.repeat(one[2], 40, 0), many[2])
