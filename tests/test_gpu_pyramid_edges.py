"""The FP32 first stage, the uint8 tile's word loads and the RGB input kernel at the sizes where their
tiles, strips and aligned words end: every level equal to the oracle, bit for bit."""

import numpy as np
import pytest
import torch

from cuvslam_b200.frontend import ImagePyramid

pytestmark = pytest.mark.gpu


def _check(pyr, want):
    torch.cuda.synchronize()
    got = pyr.to_numpy()
    assert len(got) == len(want)
    for l, (g, w) in enumerate(zip(got, want)):
        for q in range(3):
            np.testing.assert_array_equal(g[q], w[q], err_msg=f"level {l} plane {q}")


# one tile less, exactly one, one more; 100 x 97 is the staged region (smaller frames use plain copies);
# three levels only; a level 3 wide enough for several bands per CTA of the deeper levels
@pytest.mark.parametrize("shape", [(60, 60), (63, 64), (64, 65), (96, 99), (97, 100), (98, 104), (129, 128), (191, 257),
                                   (333, 1000), (1080, 64), (2049, 2050)])
@pytest.mark.parametrize("aligned", [True, False])
def test_f32_frames(ctx, oracle, shape, aligned):
    """FP32 frames from an aligned buffer (TMA) and from a view one float into a wider one (plain copies)."""
    h, w = shape
    rng = np.random.default_rng(h * 4099 + w)
    img = (rng.random(shape, dtype=np.float32) * 255).astype(np.float32)
    if aligned:
        pitch = (w + 3) // 4 * 4
        buf = torch.zeros((h, pitch), dtype=torch.float32, device="cuda")
        src = buf[:, :w]
    else:
        buf = torch.full((h, w + 3), float("nan"), dtype=torch.float32, device="cuda")
        src = buf[:, 1:w + 1]
    src.copy_(torch.from_numpy(img))
    _check(ImagePyramid(w, h).build_f32(ctx, src), oracle.pyramid_f32(img))


@pytest.mark.parametrize("levels", [3, 4, 10])
def test_f32_level_counts(ctx, oracle, levels):
    """No deeper level, one (gradients only in the second launch), and all of them."""
    rng = np.random.default_rng(levels)
    img = rng.standard_normal((200, 330)).astype(np.float32)
    _check(ImagePyramid(330, 200, levels).build_f32(ctx, torch.from_numpy(img).cuda()), oracle.pyramid_f32(img)[:levels])


@pytest.mark.parametrize("shape", [(60, 61), (131, 130), (163, 177), (164, 353), (376, 1241)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("blur", [False, True])
def test_u8_unaligned_frames(ctx, oracle, shape, offset, blur):
    """uint8 frames at every byte alignment: the tile's words are shifted together from aligned ones."""
    h, w = shape
    rng = np.random.default_rng(h * 31 + w + offset)
    img = rng.integers(0, 256, shape, dtype=np.uint8)
    flat = torch.zeros(h * (w + 2) + offset, dtype=torch.uint8, device="cuda")
    src = flat[offset:].view(h, w + 2)[:, :w]
    src.copy_(torch.from_numpy(img))
    _check(ImagePyramid(w, h).build(ctx, src, blur_filter=blur), oracle.pyramid_f32(oracle.level0(img, box=blur)))


@pytest.mark.parametrize("shape", [(60, 61), (61, 128), (65, 129), (95, 131)])
@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("blur", [False, True])
def test_rgb_unaligned_frames(ctx, shape, offset, blur):
    """RGB frames at several byte alignments equal the same frame from an aligned buffer of another
    pitch, whose level 0 equals the conversion's own expression."""
    h, w = shape
    rng = np.random.default_rng(h * 17 + w + offset)
    img = rng.integers(0, 256, shape + (3,), dtype=np.uint8)
    flat = torch.zeros(h * (3 * w + 5) + offset, dtype=torch.uint8, device="cuda")
    src = torch.as_strided(flat, (h, w, 3), (3 * w + 5, 3, 1), offset)
    src.copy_(torch.from_numpy(img))
    a = ImagePyramid(w, h).build(ctx, src, blur_filter=blur)
    b = ImagePyramid(w, h).build(ctx, torch.from_numpy(img).cuda(), blur_filter=blur)
    torch.cuda.synchronize()
    for x, y in zip(a.to_numpy(), b.to_numpy()):
        for q in range(3):
            np.testing.assert_array_equal(x[q], y[q])
    if not blur:
        f = img.astype(np.float64)
        gray = 0.299 * f[..., 0] + 0.587 * f[..., 1] + 0.114 * f[..., 2]
        # three roundings of at most half an ulp of 255, and the coefficients' own (2^-25 relative)
        assert np.abs(a.to_numpy()[0][0] - gray).max() <= 4 * 2.0**-17
