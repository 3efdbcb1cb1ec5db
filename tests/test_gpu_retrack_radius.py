"""The retrack pass and search radii: a track runs again when its radius is a number that is not negative;
one without a radius (NaN, which no distance exceeds) keeps what the first pass gave it, in every sampling."""

import numpy as np
import pytest
import torch

from conftest import assert_tracks_equal
from cuvslam_b200 import _lib, synthetic
from cuvslam_b200.frontend import ImagePyramid, LKFeatureTracker, track_mono, tracks_from_device, tracks_to_device
from cuvslam_b200.types import make_tracks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampling", [_lib.FE_SAMPLE_HARDWARE, _lib.FE_SAMPLE_TEXTURE, _lib.FE_SAMPLE_TEXTURE_WIDE,
                                      _lib.FE_SAMPLE_EXACT])
@pytest.mark.parametrize("radius", [np.nan, -np.nan, -0.0, np.inf, -1.0])
def test_unusual_radii(ctx, sampling, radius):
    first, second = 0.97, 0.3  # most tracks are lost by the first threshold, most of them kept by the second
    a, b, _ = synthetic.frame_pair(34, 640, 480)
    pa = ImagePyramid(640, 480).build(ctx, torch.from_numpy(a).cuda())
    pb = ImagePyramid(640, 480).build(ctx, torch.from_numpy(b).cuda())
    rng = np.random.default_rng(9)
    xy = rng.uniform((5, 5), (635, 475), (600, 2)).astype(np.float32)
    recs = make_tracks(xy, rng.normal(0, 2, (600, 2)), 60.0, first)
    recs["search_radius_px"][::2] = np.float32(radius)

    def tracked(threshold):
        lk, r = LKFeatureTracker(ctx, False, sampling), recs.copy()
        r["ncc_threshold"] = threshold
        t = tracks_to_device(r)
        lk.track_points(pa, pb, t)
        torch.cuda.synchronize()
        return tracks_from_device(t)

    want, again = tracked(first), tracked(second)
    lost = (want["track_status"] == 0) & (recs["search_radius_px"] >= 0)
    gained = (want["track_status"] == 0) & (again["track_status"] == 1)
    assert gained[1::2].any() and (radius < 0 or radius == 0 or gained[::2].any())
    for name in want.dtype.names:
        if name != "ncc_threshold":
            want[name][lost] = again[name][lost]
    got = tracks_to_device(recs)
    track_mono(ctx, pa, pb, got, retrack_ncc=second, sampling=sampling)
    torch.cuda.synchronize()
    assert_tracks_equal(tracks_from_device(got), want)
