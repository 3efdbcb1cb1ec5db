"""The adjoint's tile sums and pyramid adjoint at plane sizes and record counts where their paths change:
planes that end inside a 32x32 tile, odd and even levels, gradient planes whose rows are not 16-byte aligned,
tiles with no record, with many (tracks on one spot) and with patches over a power of two (taps with
their own fractions).  test_gpu_adjoint.py holds the same paths to the FP64 adjoint."""

import numpy as np
import pytest
import torch

from cuvslam_b200 import synthetic
from cuvslam_b200.diff import DiffTracker

pytestmark = pytest.mark.gpu


def _run(ctx, w, h, mode, xy, prev, cur, g):
    t = DiffTracker(ctx, 1, h, w, len(xy), mode=mode)
    p, c = (torch.from_numpy(a.astype(np.float32) / 255)[None].cuda().requires_grad_() for a in (prev, cur))
    q = torch.from_numpy(xy)[None].cuda().requires_grad_()
    pos, st = t(p, c, q)
    grads = torch.autograd.grad(pos, (p, c, q), g)
    torch.cuda.synchronize()
    out = pos.detach().cpu().numpy()[0], st.cpu().numpy()[0], [v.cpu().numpy()[0] for v in grads]
    t.close()
    return out


@pytest.mark.parametrize("shape", [(96, 64), (97, 65), (130, 95), (161, 129)])
@pytest.mark.parametrize("mode", ["implicit", "unrolled"])
def test_sums_of_repeated_tracks(ctx, shape, mode):
    """Forty copies of a track add up to forty times its gradient (long tiles), in any order of copies: the
    sums run in track order, so the relative difference stays within 40 roundings of FP32."""
    w, h = shape
    prev, cur, _ = synthetic.frame_pair(51, w, h)
    rng = np.random.default_rng(w)
    base = rng.uniform((6, 6), (w - 6, h - 6), (12, 2)).astype(np.float32)
    base[:3] = [(32.3, 31.6), (63.7, 16.2), (16.1, 33.4)]  # patches across powers of two
    g1 = rng.normal(size=(1, 12, 2)).astype(np.float32)
    _, st1, one = _run(ctx, w, h, mode, base, prev, cur, torch.from_numpy(g1).cuda())
    _, st40, many = _run(ctx, w, h, mode, np.repeat(base, 40, 0), prev, cur, torch.from_numpy(np.repeat(g1, 40, 1)).cuda())
    assert np.array_equal(np.repeat(st1, 40), st40)
    for a, b in zip(one[:2], many[:2]):
        scale = np.abs(a).max()
        if scale > 0:
            assert np.abs(b / 40 - a).max() <= 64 * 2.0**-23 * np.abs(a).sum() / np.count_nonzero(a) + 64 * 2.0**-23 * scale
    assert np.array_equal(np.repeat(one[2], 40, 0), many[2])
