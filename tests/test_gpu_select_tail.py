"""The selection's alive features, quotas and final ranks where their blocks and dispatches change:
feature counts around a block, more features than cells (ranked burn), kept counts around a rank block
and past its key chunk, and equal strengths, against the oracle's selection on the same response map."""

import os

import numpy as np
import pytest
import torch

from conftest import gpu_pyramid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dctx():
    os.environ["CUVSLAM_FE_DEBUG_MAPS"] = "1"
    from cuvslam_b200.frontend import Context

    c = Context(0)
    del os.environ["CUVSLAM_FE_DEBUG_MAPS"]
    yield c
    c.close()


def _check(dctx, oracle, img, alive, want, borders=(0, 0, 0, 0), mask=None):
    from cuvslam_b200.frontend import Selection

    h, w = img.shape
    pyr = gpu_pyramid(dctx, img)
    sel = Selection(dctx)
    got = sel.compute_gftt_and_select_features(pyr, *borders, mask, alive, want).cpu().numpy()
    resp = sel.debug_maps(w, h)[0].cpu().numpy()
    exp = oracle.select(resp, alive, want, borders, mask)["sel"]
    assert got.shape == exp.shape
    # positions: the refinement's fast division against the oracle's (the tolerance of test_gpu_select.py)
    np.testing.assert_allclose(got, exp, rtol=0, atol=2e-4)


@pytest.mark.parametrize("n", [0, 1, 31, 32, 33, 63, 64, 65, 607])
def test_alive_counts(dctx, oracle, n):
    """A 200x150 frame has 25 x 18 = 450 cells: 607 features take the ranked burn, the others the spread one.
    Some lie outside the frame and on its edges."""
    rng = np.random.default_rng(n)
    img = rng.integers(0, 256, (150, 200), dtype=np.uint8)
    alive = rng.uniform((-6, -6), (206, 156), (n, 2)).astype(np.float32)
    alive[: n // 8] = np.round(alive[: n // 8])
    _check(dctx, oracle, img, alive if n else None, 120)


@pytest.mark.parametrize("want", [1, 31, 32, 33, 2047, 2048, 2049, 4000])
def test_kept_counts(dctx, oracle, want):
    rng = np.random.default_rng(want)
    img = rng.integers(0, 256, (480, 640), dtype=np.uint8)
    _check(dctx, oracle, img, None, want, (3, 5, 7, 2))


@pytest.mark.parametrize("shape", [(64, 64), (65, 71), (7, 90), (120, 9)])
def test_equal_strengths(dctx, oracle, shape):
    """A periodic pattern: every cell's strength occurs many times, ordered by cell; frames of few or no
    cells."""
    h, w = shape
    y, x = np.mgrid[0:h, 0:w]
    img = (((x // 4) + (y // 4)) % 2 * 200 + 20).astype(np.uint8)
    _check(dctx, oracle, img, np.array([[w / 2, h / 2]], np.float32), 300)
