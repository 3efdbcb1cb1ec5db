"""FP32 pyramids whose deeper levels need several bands per block (rows too long for a block's share to be staged
at once), one row per band at the widest level 3 that the cluster takes, and the generic stages just past it;
and the FP32 first stage's bounded wait."""

import numpy as np
import pytest
import torch

from cuvslam_b200 import _lib
from cuvslam_b200.frontend import Context, ImagePyramid
from cuvslam_b200.types import level_sizes

pytestmark = pytest.mark.gpu

FLOATS = 12 * 1024  # the cluster's shared memory


def _equal(got, want):
    torch.cuda.synchronize()
    got = got.to_numpy()
    assert len(got) == len(want)
    for l, (g, w) in enumerate(zip(got, want)):
        for q in range(3):
            np.testing.assert_array_equal(g[q], w[q], err_msg=f"level {l} plane {q}")


# (w, h, rows of the next level that a band of level 3 can stage: fewer than a block's share; 0: generic stages)
@pytest.mark.parametrize("w,h,rows", [(4096, 4096, 9), (4100, 1100, 8), (12288, 240, 1), (12281, 232, 1), (12288, 130, None),
                                      (12289, 240, 0)])
def test_wide_frames(ctx, oracle, w, h, rows):
    sizes = level_sizes(w, h)
    ss = (sizes[3][0] + 3) & ~3
    if rows:
        assert (FLOATS // ss - 6) // 2 == rows and rows < -(-sizes[4][1] // 8)
    elif rows == 0:
        assert ss > FLOATS // 8
    else:  # level 3 is the last
        assert len(sizes) == 4 and FLOATS // ss - 6 < -(-sizes[3][1] // 8)
    rng = np.random.default_rng(w)
    img = (rng.random((h, w), dtype=np.float32) * 255).astype(np.float32)
    _equal(ImagePyramid(w, h).build_f32(ctx, torch.from_numpy(img).cuda()), oracle.pyramid_f32(img))


def test_first_stage_wait_that_runs_out(ctx, oracle):
    """A wait limit of 0: the tiles' staging copies give up at once and are drained, the launch ends, the context
    says so and builds correctly again."""
    w, h = 1280, 720
    img = (np.random.default_rng(2).random((h, w), dtype=np.float32) * 255).astype(np.float32)
    dimg = torch.from_numpy(img).cuda()
    c = Context(0)
    try:
        c.set_wait_limit(0)
        ImagePyramid(w, h).build_f32(c, dimg)
        with pytest.raises(_lib.FeError, match="device fault"):
            c.device_status()
        assert c.device_status() == 0
        c.set_wait_limit(_lib.FE_DEFAULT_WAIT_LIMIT)
        _equal(ImagePyramid(w, h).build_f32(c, dimg), oracle.pyramid_f32(img))
        assert c.device_status() == 0
    finally:
        c.close()
