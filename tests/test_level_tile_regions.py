"""Shared-memory regions of the kernels that build levels 0-2 from a tile (pyramid.cu: the uint8 kernel, namespace
l012, and the FP32 first stage, namespace lead), restated on the CPU with their present passes: the staged
region, the mirrored cells put in place around the image, the column pairs of levels 1 and 2, the corner pixels
redone, level 3's core, the outputs.  Every read lies in its region; every value that reaches an output of the
image comes from a pixel of the frame or from a cell that an earlier pass computed from such; the mirrored
cells are read inside the image and written outside it, so that no thread reads what another one writes.  Bounds,
not values: the GPU tests compare those with the oracle.

The deeper levels' bands of both (shared by a queue of items, or by a cluster of eight blocks) are restated below:
rows of every level covered once, every tap of a band among its staged rows, the staged rows inside the memory."""

import numpy as np
import pytest

from cuvslam_b200.types import level_sizes


class Kernel:
    def __init__(self, t2, w, h, ox, oy):
        self.t2, self.w, self.h, self.ox, self.oy = t2, w, h, ox, oy
        self.s1, self.s1s, self.s2, self.s2s = 2 * t2 + 15, 2 * t2 + 16, t2 + 6, t2 + 8


U8 = Kernel(32, 176, 163, 32, 19)
F32 = Kernel(16, 100, 97, 20, 18)


def mirror(i, n):
    i = i if i >= 0 else -i - 1
    return i if i < n else 2 * n - i - 1


def mirror_rings(good, rw, rh, ax, ay, w, h):
    """good: cells that hold what the mirror addressing reads there; `good[:rh, :rw]` is the region."""
    src = good.copy()
    for i in range(4 * (rw + rh)):
        col = i < 4 * rh
        k = i if col else i - 4 * rh
        m, p = k & 3, k >> 2
        x = (m - 2 if m < 2 else w + m - 2) if col else ax + p
        y = ay + p if col else (m - 2 if m < 2 else h + m - 2)
        cx, cy = x - ax, y - ay
        if not (0 <= cx < rw and 0 <= cy < rh) or y < -2 or y > h + 1 or (not col and not 0 <= x < w):
            continue
        sx, sy = mirror(x, w) - ax, mirror(y, h) - ay
        if not (0 <= sx < rw and 0 <= sy < rh):
            continue
        assert not (0 <= x < w and 0 <= y < h), "a mirrored cell inside the image"
        assert 0 <= sx + ax < w and 0 <= sy + ay < h, "a source outside the image"
        good[cy, cx] = src[sy, sx]


def corner(good, ax, ay, sw, sh, x, y):
    """Cells that the 25-tap rule reads at a corner pixel: all in the region, the ones that count good."""
    for k in range(5):
        for l in range(5):
            xc, yc = 2 * x - 2 + l, 2 * y - 2 + k
            r, c = mirror(yc, sh) - ay, mirror(xc, sw) - ax
            assert 0 <= r < good.shape[0] and 0 <= c < good.shape[1]
            if not ((xc < 0 or xc >= sw) and (yc < 0 or yc >= sh)):
                assert good[r, c]


def down(good, rows, cols, r0, c0):
    """Whether the 5x5 windows at rows r0 + 2 r, columns c0 + 2 c hold only good cells (rows x cols of them)."""
    out = np.ones((rows, cols), bool)
    for k in range(5):
        for l in range(5):
            out &= good[r0 + k:r0 + k + 2 * rows - 1:2, c0 + l:c0 + l + 2 * cols - 1:2]
    return out


def in_image(rows, cols, ax, ay, w, h):
    y, x = ay + np.arange(rows)[:, None], ax + np.arange(cols)[None, :]
    return (x >= 0) & (x < w) & (y >= 0) & (y < h)


def corners(w, h):
    return {(x, y) for x in (0, w - 1) for y in (0, h - 1)}


def check_tile(K, sizes, X2, Y2):
    (w0, h0), (w1, h1), (w2, h2) = sizes[:3]
    a0x, a0y, a1x, a1y, a2x, a2y = 4 * X2 - K.ox, 4 * Y2 - K.oy, 2 * X2 - 8, 2 * Y2 - 8, X2 - 4, Y2 - 3
    b0 = in_image(K.h, K.w, a0x, a0y, w0, h0)
    edge = a0x < 0 or a0y < 0 or a0x + K.w > w0 or a0y + K.h > h0
    if edge:
        mirror_rings(b0, K.w, K.h, a0x, a0y, w0, h0)

    # level 1: cell (r, c) reads the staged rows 2 r + dr .. + 4 and columns 2 c + dc .. + 4
    dr, dc = 2 * a1y - 2 - a0y, 2 * a1x - 2 - a0x
    assert (dr, dc) == ((1, 14) if K is U8 else (0, 2))
    assert dr + 2 * (K.s1 - 1) + 4 < K.h and dc + 2 * (K.s1 - 1) + 4 < K.w
    v1 = down(b0, K.s1, K.s1, dr, dc)
    img1 = in_image(K.s1, K.s1, a1x, a1y, w1, h1)
    fixed = {(x, y) for x, y in corners(w1, h1) if a1x <= x < a1x + K.s1 and a1y <= y < a1y + K.s1}
    if edge:
        for x, y in fixed:
            corner(b0, a0x, a0y, w0, h0, x, y)
            v1[y - a1y, x - a1x] = True
    assert v1[img1].all(), "level 1"
    b1 = np.zeros((K.s1, K.s1s), bool)
    b1[:, :K.s1] = img1
    if edge:
        mirror_rings(b1, K.s1, K.s1, a1x, a1y, w1, h1)

    # level 2, stored from column X2 - 4: cell (r, c + 1) reads level 1's rows 2 r .. and columns 2 c ..
    assert 2 * a2y - 2 - a1y == 0 and 2 * (a2x + 1) - 2 - a1x == 0
    assert 2 * (K.s2 - 1) + 4 < K.s1 and 2 * (K.s2 - 1) + 4 < K.s1s
    v2 = down(b1, K.s2, K.s2, 0, 0)
    img2 = in_image(K.s2, K.s2, a2x + 1, a2y, w2, h2)
    if edge:
        for x, y in corners(w2, h2):
            if a2x < x <= a2x + K.s2 and a2y <= y < a2y + K.s2:
                corner(b1, a1x, a1y, w1, h1, x, y)
                v2[y - a2y, x - a2x - 1] = True
    assert v2[img2].all(), "level 2"
    b2 = np.zeros((K.s2, K.s2s), bool)
    b2[:, 1:1 + K.s2] = img2
    if edge:
        mirror_rings(b2, K.s2s, K.s2, a2x, a2y, w2, h2)

    # level 3's core
    if len(sizes) > 3:
        w3, h3 = sizes[3]
        t3 = K.t2 // 2
        dr, dc = Y2 - 2 - a2y, X2 - 2 - a2x
        assert dr + 2 * (t3 - 1) + 4 < K.s2 and dc + 2 * (t3 - 1) + 4 < K.s2s
        v3 = down(b2, t3, t3, dr, dc)
        for y in range(t3):
            for x in range(t3):
                gx, gy = X2 // 2 + x, Y2 // 2 + y
                if gx < w3 and gy < h3:
                    if (gx, gy) in corners(w3, h3):
                        corner(b2, a2x, a2y, w2, h2, gx, gy)
                    else:
                        assert v3[y, x], (gx, gy)

    # outputs: the core's pixels and their seven taps along each axis, whose loads reach four columns and
    # three rows past the core whether used or not
    for lev, (good, ax, ay) in enumerate(((b0, a0x, a0y), (b1, a1x, a1y), (b2, a2x, a2y))):
        w, h = sizes[lev]
        n = K.t2 << (2 - lev)
        cx, cy = (X2 << (2 - lev)) - ax, (Y2 << (2 - lev)) - ay
        assert cx >= 4 and cy >= 3 and cx + n + 4 <= good.shape[1] and cy + n + 3 <= good.shape[0], lev
        assert cx % 4 == 0 and good.shape[1] % 4 == 0  # aligned 16-byte (uint8: word) loads
        y, x = ay + cy + np.arange(n)[:, None], ax + cx + np.arange(n)[None, :]
        inside = (x < w) & (y < h)
        for j in range(-3, 4):
            row = good[cy:cy + n, cx + j:cx + j + n]
            assert row[inside & (x > 2) & (x < w - 3)].all() and (j or row[inside].all()), (lev, "x", j)
            assert good[cy + j:cy + j + n, cx:cx + n][inside & (y > 2) & (y < h - 3)].all(), (lev, "y", j)


SIZES = [(57, 57), (58, 61), (63, 120), (64, 64), (97, 61), (100, 97), (130, 57), (640, 480), (1241, 376), (1920, 1200),
         (2047, 1535), (12289, 240)]


@pytest.mark.parametrize("K", [U8, F32], ids=["u8", "f32"])
@pytest.mark.parametrize("w,h", SIZES)
def test_regions(K, w, h):
    sizes = level_sizes(w, h)
    (w2, h2) = sizes[2]
    tx, ty = -(-w2 // K.t2), -(-h2 // K.t2)
    for Y in sorted({0, 1, ty // 2, ty - 2, ty - 1} & set(range(ty))):
        for X in sorted({0, 1, tx // 2, tx - 2, tx - 1} & set(range(tx))):
            check_tile(K, sizes, X * K.t2, Y * K.t2)


def test_items_cover_the_regions():
    """The passes' work items: the uint8 kernel's column pairs x bands, the FP32 kernel's pairs x strips (the last
    strip overlaps the one before), as loads of whole words inside a row of the region."""
    # uint8, level 1: 40 pairs x 12 bands of 7 rows; three words from column 4 pp + 12 (two in the last pair)
    rows = {b * 7 + r for b in range(12) for r in range(min(7, U8.s1 - 7 * b))}
    assert rows == set(range(U8.s1)) and 40 * 12 <= 512
    for pp in range(40):
        two = 2 * pp + 1 < U8.s1
        assert 4 * pp + 12 + (12 if two else 8) <= U8.w and 2 * pp + 1 < U8.s1s
        assert 4 * pp + 14 + (6 if two else 4) < 4 * pp + 12 + (12 if two else 8)  # the taps are among the bytes
    # level 2: 19 pairs x 13 bands of 3 rows, two 16-byte loads from column 4 pp
    assert {b * 3 + r for b in range(13) for r in range(min(3, U8.s2 - 3 * b))} == set(range(U8.s2))
    assert 19 * 13 <= 512 and all(4 * pp + 8 <= U8.s1s and 2 * pp + 2 < U8.s2s for pp in range(19))
    # FP32, level 1: 24 pairs x 10 strips of 5 rows; columns 4 pp + 2 .. 4 pp + 7, and + 8 for a second column
    assert {min(5 * s, F32.s1 - 5) + r for s in range(10) for r in range(5)} == set(range(F32.s1)) and 24 * 10 <= 256
    for pp in range(24):
        last = 4 * pp + (8 if 2 * pp + 1 < F32.s1 else 7)
        assert last < F32.w and (4 * pp + 2) % 2 == 0 and (4 * pp + 4) % 4 == 0 and 2 * pp + 1 < F32.s1s
    assert 2 * (F32.s1 - 5) + 2 * 5 + 3 <= F32.h and F32.w % 4 == 0
    # level 2: a pair of one row per thread
    assert 11 * F32.s2 <= 256 and all(4 * pp + 8 <= F32.s1s and 2 * pp + 2 < F32.s2s for pp in range(11))
    # level 0: 16 column groups x 16 strips of four rows
    assert 16 * 16 == 256 and F32.oy + 60 + 3 + 3 < F32.h and F32.ox + 60 + 8 <= F32.w


def test_tma_boxes():
    """The copies' innermost coordinate and row are multiples of 16 bytes, the boxes fill their regions."""
    for X2 in range(0, 4096, 32):
        assert (4 * X2 - U8.ox) % 16 == 0
    for X2 in range(0, 4096, 16):
        assert (4 * X2 - F32.ox) * 4 % 16 == 0
    assert U8.w % 16 == 0 and F32.w * 4 % 16 == 0 and max(U8.w, U8.h, F32.w, F32.h) <= 256


# ---------------------------------------------------------------- deeper levels
def pad4(w):
    return (w + 3) & ~3


def u8_cap():
    b1 = -(-U8.w * U8.h // 128) * 128
    return ((b1 + 4 * (U8.s1 * U8.s1s + U8.s2 * U8.s2s)) // 4) & ~3


def check_band(s_h, n_h, r0, rows):
    """Band [r0, r0 + rows) of the next level: the staged rows hold its taps and its gradients'; returns them."""
    r1 = min(n_h, r0 + rows)
    lo, hi = max(0, 2 * r0 - 3), min(s_h - 1, 2 * r1 + 2)
    for y in range(r0, r1):
        for k in range(5):
            assert lo <= mirror(2 * y - 2 + k, s_h) <= hi
    for y in range(min(s_h, 2 * r0), min(s_h, 2 * r1)):
        assert lo <= y <= hi and (not 2 < y < s_h - 3 or lo <= y - 3 and y + 3 <= hi)
    return hi - lo + 1


DEEP = SIZES + [(4096, 4096), (12288, 240), (12288, 130), (240, 12288), (3000, 4000), (8192, 8192), (120, 4000)]


@pytest.mark.parametrize("w,h", DEEP)
def test_bands_of_the_queue(w, h):
    """plan_deep_items: levels 3 .. of a uint8 build as up to two banded phases and a rest item."""
    lv, cap = level_sizes(w, h)[3:], u8_cap()
    n = len(lv)
    need = [sum(pad4(a) * b for a, b in lv[k:]) for k in range(n)]
    r = next((k for k in range(min(n, 3)) if need[k] <= cap), None)
    if r is None:
        return  # generic stages
    while r < 2 and r + 1 < n and lv[r][0] * lv[r][1] > 2048:
        r += 1
    assert need[r] <= cap
    for p in range(r):
        rows = (cap // pad4(lv[p][0]) - 6) // 2
        if rows < 1:
            return  # generic stages
        rows = min(rows, max(4, -(-256 // lv[p + 1][0])))
        bands = -(-lv[p + 1][1] // rows)
        covered = []
        for b in range(bands):
            staged = check_band(lv[p][1], lv[p + 1][1], b * rows, rows)
            assert staged * pad4(lv[p][0]) <= cap
            covered += range(2 * b * rows, min(lv[p][1], 2 * min(lv[p + 1][1], (b + 1) * rows)))
        assert covered == list(range(lv[p][1])), "a row of the source level without gradients"


@pytest.mark.parametrize("w,h", DEEP)
def test_bands_of_the_cluster(w, h):
    """pyramid_deep_kernel: each level's rows in eight bands, a band in steps that fit its shared memory."""
    floats, lv = 12 * 1024, level_sizes(w, h)[3:]
    if not lv or pad4(lv[0][0]) > floats // 8:
        return  # generic stages
    for t, (sw, sh) in enumerate(lv):
        ss, covered = pad4(sw), []
        if t + 1 < len(lv):
            nh = lv[t + 1][1]
            per = -(-nh // 8)
            step = min(per, (floats // ss - 6) // 2)
            assert step >= 1
            for rank in range(8):
                end = min(nh, (rank + 1) * per)
                for r0 in range(rank * per, end, step):
                    rows = min(step, end - r0)
                    assert check_band(sh, nh, r0, rows) * ss <= floats
                    covered += range(2 * r0, min(sh, 2 * min(nh, r0 + rows)))
        else:
            per = -(-sh // 8)
            step = min(per, floats // ss - 6)
            assert step >= 1
            for rank in range(8):
                end = min(sh, (rank + 1) * per)
                for y0 in range(rank * per, end, step):
                    y1, lo = min(y0 + step, end), max(0, y0 - 3)
                    rows = min(sh, y1 + 3) - lo
                    assert rows * ss <= floats
                    assert all(lo <= y - 3 and y + 3 < lo + rows for y in range(y0, y1) if 2 < y < sh - 3)
                    covered += range(y0, y1)
        assert covered == list(range(sh))
