"""The affine tracker on both sides of its register budgets' dispatch: the same tracks one warp each, and
repeated until the launch has more tracks than resident warps, give the same records."""

import numpy as np
import pytest
import torch

from conftest import assert_tracks_equal
from cuvslam_b200 import _lib, synthetic
from cuvslam_b200.frontend import (ImagePyramid, STFeatureTracker, STFeatureTrackerWithCache, tracks_from_device,
                                   tracks_to_device)
from cuvslam_b200.types import make_tracks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampling", [_lib.FE_SAMPLE_TEXTURE, _lib.FE_SAMPLE_TEXTURE_WIDE, _lib.FE_SAMPLE_EXACT])
@pytest.mark.parametrize("shift,full", [(0, 20), (5, 5), (3, 0), (0, 0)])
def test_few_and_many_tracks(ctx, oracle, sampling, shift, full):
    a, b, warp = synthetic.frame_pair(12, 320, 240)
    pa = ImagePyramid(320, 240).build(ctx, torch.from_numpy(a).cuda())
    pb = ImagePyramid(320, 240).build(ctx, torch.from_numpy(b).cuda())
    rng = np.random.default_rng(4)
    xy = rng.uniform((-4, -4), (324, 244), (61, 2)).astype(np.float32)
    off = (synthetic.flow_texture(warp, xy.astype(np.float64)) - xy).astype(np.float32)
    one = make_tracks(xy, off, 16.0, 0.8)
    few = tracks_to_device(one)
    many = tracks_to_device(np.tile(one, 100))  # 6100 tracks: more than two blocks of eight warps on every SM
    st = STFeatureTracker(ctx, shift, full, sampling)
    st.track_points(pa, pb, few)
    st.track_points(pa, pb, many)
    torch.cuda.synchronize()
    got = tracks_from_device(few)
    want = oracle.st_track(oracle.pyramid(a), oracle.pyramid(b), one, shift, full, sampling)
    assert_tracks_equal(got, want)
    for part in tracks_from_device(many).reshape(100, 61):
        assert_tracks_equal(part, got)
    # and against the cache of the same patches
    cached = STFeatureTrackerWithCache(ctx, shift, full, sampling)
    few, many = tracks_to_device(one), tracks_to_device(np.tile(one, 100))
    cached.track_points(pb, cached.build_points_cache(pa, few), few)
    cached.track_points(pb, cached.build_points_cache(pa, many), many)
    torch.cuda.synchronize()
    got = tracks_from_device(few)
    for part in tracks_from_device(many).reshape(100, 61):
        part["cache_index"] = got["cache_index"]  # each copy has its own entry
        assert_tracks_equal(part, got)
