"""The retrack pass against its definition: every track through the first pass, the lost ones through a
second whole pass with the retrack threshold.  Thresholds on both sides of the tracks' own, so that gates
fork at coarse levels and at the last one, either way round, or never."""

import numpy as np
import pytest
import torch

from conftest import assert_tracks_equal
from cuvslam_b200 import _lib, synthetic
from cuvslam_b200.frontend import ImagePyramid, LKFeatureTracker, track_mono, tracks_from_device, tracks_to_device
from cuvslam_b200.types import make_tracks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampling", [_lib.FE_SAMPLE_HARDWARE, _lib.FE_SAMPLE_TEXTURE])
@pytest.mark.parametrize("first,second", [(0.8, 0.85), (0.8, 0.8), (0.95, 0.5), (0.999, 0.9), (0.5, 0.999), (2.0, 0.7),
                                          (-2.0, 0.9)])
def test_mono_equals_two_passes(ctx, sampling, first, second):
    a, b, _ = synthetic.frame_pair(33, 640, 480)
    pa = ImagePyramid(640, 480).build(ctx, torch.from_numpy(a).cuda())
    pb = ImagePyramid(640, 480).build(ctx, torch.from_numpy(b).cuda())
    rng = np.random.default_rng(8)
    xy = rng.uniform((-3, -3), (643, 483), (1500, 2)).astype(np.float32)
    recs = make_tracks(xy, rng.normal(0, 6, (1500, 2)), 60.0, first)
    recs["search_radius_px"][::97] = -1.0
    got = tracks_to_device(recs)
    track_mono(ctx, pa, pb, got, retrack_ncc=second, sampling=sampling)
    lk = LKFeatureTracker(ctx, False, sampling)
    one = tracks_to_device(recs)
    lk.track_points(pa, pb, one)
    again = recs.copy()
    again["ncc_threshold"] = second
    two = tracks_to_device(again)
    lk.track_points(pa, pb, two)
    torch.cuda.synchronize()
    want, second_pass = tracks_from_device(one), tracks_from_device(two)
    lost = (want["track_status"] == 0) & (recs["search_radius_px"] >= 0)
    for name in want.dtype.names:
        if name != "ncc_threshold":
            want[name][lost] = second_pass[name][lost]
    assert_tracks_equal(tracks_from_device(got), want)
