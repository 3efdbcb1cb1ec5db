"""The final order of many kept keys, where chunks are sorted first: one camera with several chunks, and a batch
whose cameras lie on both sides of one, against the oracle and against the cameras one by one."""

import os

import numpy as np
import pytest
import torch

from conftest import gpu_pyramid
from cuvslam_b200.frontend import Batch, CameraFrame, Context, ImagePyramid, Selection

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dctx():
    os.environ["CUVSLAM_FE_DEBUG_MAPS"] = "1"
    c = Context(0)
    del os.environ["CUVSLAM_FE_DEBUG_MAPS"]
    yield c
    c.close()


# six chunks and a few keys, eight, and a frame with fewer cells than are asked for
@pytest.mark.parametrize("w,h,want", [(2048, 1152, 12250), (2048, 1152, 12289), (2048, 1152, 16320), (1000, 780, 14000)])
def test_one_camera(dctx, oracle, w, h, want):
    rng = np.random.default_rng(want)
    img = rng.integers(0, 256, (h, w), dtype=np.uint8)
    sel = Selection(dctx)
    got = sel.compute_gftt_and_select_features(gpu_pyramid(dctx, img), 0, 0, 0, 0, None, None, want).cpu().numpy()
    exp = oracle.select(sel.debug_maps(w, h)[0].cpu().numpy(), None, want, (0, 0, 0, 0), None)["sel"]
    assert got.shape == exp.shape
    # positions: the refinement's fast division against the oracle's (the tolerance of test_gpu_select.py)
    np.testing.assert_allclose(got, exp, rtol=0, atol=2e-4)


def test_equal_strengths_over_chunks(dctx, oracle):
    """A periodic pattern: thousands of cells of one strength, ordered by cell across the chunks."""
    w, h, want = 1600, 1200, 16000
    y, x = np.mgrid[0:h, 0:w]
    img = (((x // 4) + (y // 4)) % 2 * 200 + 20).astype(np.uint8)
    sel = Selection(dctx)
    got = sel.compute_gftt_and_select_features(gpu_pyramid(dctx, img), 0, 0, 0, 0, None, None, want).cpu().numpy()
    exp = oracle.select(sel.debug_maps(w, h)[0].cpu().numpy(), None, want, (0, 0, 0, 0), None)["sel"]
    assert got.shape == exp.shape and len(got) > 4096
    np.testing.assert_allclose(got, exp, rtol=0, atol=2e-4)


@pytest.mark.parametrize("overlap", ["after LK", "after LK and the burn"])
def test_batch_on_both_sides_of_a_chunk(ctx, overlap):
    w, h = 480, 400  # 3000 cells
    wants = [0, 1, 500] + [2030 + k for k in range(33)] + [2990, 2999, 3000, 3100]
    rng = np.random.default_rng(6)
    imgs = [torch.from_numpy(rng.integers(0, 256, (h, w), dtype=np.uint8)).cuda() for _ in range(4)]
    frames = [CameraFrame(imgs[i % 4], ImagePyramid(w, h), None, None, n) for i, n in enumerate(wants)]
    batch = Batch(ctx, frames)
    batch.set_tuning(response_overlap=overlap)
    batch.run()
    torch.cuda.synchronize()
    pyrs = [ImagePyramid(w, h).build(ctx, im) for im in imgs]
    for i, (f, n) in enumerate(zip(frames, wants)):
        one = Selection(ctx).compute_gftt_and_select_features(pyrs[i % 4], 0, 0, 0, 0, None, None, n)
        k = int(f.new_count.item())
        assert k == len(one), (n, k, len(one))
        assert torch.equal(f.new_xy[:k], one), n
    assert max(int(f.new_count.item()) for f in frames) > 2048
    batch.close()
