"""Pyramids without grad_y planes (a secondary or current camera's, which the trackers read only for its
image): the FP32 and RGB builds and the adjoint's own build leave the missing planes out and write the
others as a full build does."""

import ctypes

import numpy as np
import pytest
import torch

from cuvslam_b200 import _lib, synthetic
from cuvslam_b200.diff import DiffTracker
from cuvslam_b200.frontend import ImagePyramid

pytestmark = pytest.mark.gpu

MARK = 0x5A  # a byte no build leaves in place over a whole plane


def _planes(p, without):
    """{(level, plane): array}; the planes left out must still hold the mark."""
    torch.cuda.synchronize()
    out = {}
    for l in range(p.levels):
        for q, plane in enumerate((p.image(l), p.grad_x(l), p.grad_y(l))):
            a = plane.cpu().numpy()
            if q == 2 and l in without:
                assert (np.ascontiguousarray(a).view(np.uint8) == MARK).all(), f"level {l}: grad_y was written"
            else:
                out[l, q] = a
    return out


def _compare(build, w, h, levels, without):
    full, part = ImagePyramid(w, h, levels), ImagePyramid(w, h, levels)
    part.storage.fill_(MARK)
    without = [l for l in without if l < part.levels]
    kept = {l: part.desc.grad_y[l] for l in without}
    for l in without:
        part.desc.grad_y[l] = None
    build(full)
    build(part)
    for l, ptr in kept.items():
        part.desc.grad_y[l] = ptr
    got, want = _planes(part, without), _planes(full, ())
    for key, a in got.items():
        np.testing.assert_array_equal(a, want[key], err_msg=f"(level, plane) {key}")


# the levels 0-2 tile with whole and ragged groups of four columns, with and without deeper levels, and the
# generic stages (fewer than three levels)
@pytest.mark.parametrize("w,h,levels", [(640, 480, 10), (1241, 377, 10), (131, 97, 3), (61, 60, 3), (333, 200, 2)])
@pytest.mark.parametrize("without", [range(10), [1], [2], [0, 3, 4]])
def test_f32_build(ctx, w, h, levels, without):
    rng = np.random.default_rng(w + h)
    img = torch.from_numpy((rng.random((h, w), dtype=np.float32) * 255).astype(np.float32)).cuda()
    _compare(lambda p: p.build_f32(ctx, img), w, h, levels, list(without))


@pytest.mark.parametrize("w,h", [(640, 480), (131, 97)])
@pytest.mark.parametrize("without", [range(1, 10), [1], [2]])
def test_rgb_and_u8_builds(ctx, w, h, without):
    """These entries ask for level 0's grad_y only."""
    rng = np.random.default_rng(w)
    rgb = torch.from_numpy(rng.integers(0, 256, (h, w, 3), dtype=np.uint8)).cuda()
    _compare(lambda p: p.build(ctx, rgb), w, h, 10, list(without))
    _compare(lambda p: p.build(ctx, rgb[..., 1].contiguous()), w, h, 10, list(without))


@pytest.mark.parametrize("mode", ["implicit", "unrolled"])
def test_adjoint_with_a_current_pyramid_without_grad_y(ctx, mode):
    """The adjoint asks for grad_y of the previous frame only: same tracks and gradients."""
    w, h, n = 320, 240, 40
    prev, cur, _ = synthetic.frame_pair(5, w, h)
    rng = np.random.default_rng(3)
    xy = torch.from_numpy(rng.uniform((20, 20), (w - 20, h - 20), (1, n, 2)).astype(np.float32)).cuda()
    g = torch.from_numpy(rng.normal(size=(1, n, 2)).astype(np.float32)).cuda()
    frames = [torch.from_numpy(a.astype(np.float32) / 255)[None].cuda() for a in (prev, cur)]

    def run(without):
        t = DiffTracker(ctx, 1, h, w, n, mode=mode)
        if without:  # the same jobs planned again over a current pyramid without the planes
            _lib.check(ctx.lib.fe_adjoint_destroy(t.handle), "fe_adjoint_destroy")
            t.handle = None
            for l in range(t.cur_pyr[0].levels):
                t.cur_pyr[0].desc.grad_y[l] = None
            handle = ctypes.c_void_p()
            _lib.check(ctx.lib.fe_adjoint_create(ctx.handle, t._jobs, 1, t.mode, t.iterations,
                                                 ctypes.c_float(t.tolerance), ctypes.byref(handle)), "fe_adjoint_create")
            t.handle = handle
        t.set_inputs(*frames, xy)
        t.build_pyramids()
        t.forward_step()
        t.grad_xy.copy_(g)
        t.backward_step()
        torch.cuda.synchronize()
        pos, status = t.outputs()
        out = [v.cpu().numpy() for v in (pos, status, t.grad_prev, t.grad_cur, t.grad_track, t.grad_offset)]
        t.close()
        return out

    want, got = run(False), run(True)
    assert want[1].any() and np.abs(want[2]).max() > 0
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
