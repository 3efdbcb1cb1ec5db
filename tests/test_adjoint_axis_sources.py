"""adjoint_pixel's straight-line lists of sources (axis_sources, lk_adjoint.cu) restated on the CPU: along an axis of
n they name exactly the next level's coordinates whose 5 taps read each coordinate, directly or through the
mirror, with the taps' weights and in the order of the loops they stand for; in two dimensions, with the rule
for corners, they are the transpose of the filter-and-decimate."""

import numpy as np
import pytest

BINOM = (1.0, 4.0, 6.0, 4.0, 1.0)


def binom5(k):
    return BINOM[k] / 16.0 if 0 <= k <= 4 else BINOM[0] / 16.0


def axis_sources(c, n, m):
    X, w = [-1] * 5, [0.0] * 5
    for j in range(3):
        k = (c & 1) + 2 * j
        p = (c + 2 - k) >> 1
        X[j] = p if k < 5 and 0 <= p < m else -1
        w[j] = binom5(k)
    X[3] = 0 if c <= 1 else -1
    w[3] = binom5(1) if c == 0 else binom5(0)
    odd = n & 1
    X[4] = m - 1 if c == n - 1 or (odd and c == n - 2) else -1
    w[4] = binom5(3) if c == n - 1 and odd else binom5(4)
    return X, w


def loops(c, n, m):
    """[(source, weight, through the mirror)] by loops over the virtual coordinates and taps."""
    out = []
    for a, v in enumerate((c, -c - 1 if c <= 1 else None, 2 * n - c - 1 if c >= n - 2 else None)):
        if v is None:
            continue
        for k in range(5):
            if (v + 2 - k) & 1:
                continue
            X = (v + 2 - k) // 2
            if 0 <= X < m:
                out.append((X, binom5(k), a > 0))
    return out


@pytest.mark.parametrize("n", list(range(15, 70)) + [127, 128, 1023, 1024])
def test_axis(n):
    m = (n + 1) // 2
    for c in range(n):
        X, w = axis_sources(c, n, m)
        got = [(X[j], w[j], j >= 3) for j in range(5) if X[j] >= 0]
        assert got == loops(c, n, m), c


def _mirror(i, n):
    i = i if i >= 0 else -i - 1
    return i if i < n else 2 * n - i - 1


@pytest.mark.parametrize("w,h", [(15, 15), (16, 17), (17, 16), (30, 21), (33, 40)])
def test_transpose(w, h):
    uw, uh = (w + 1) // 2, (h + 1) // 2
    D = np.zeros((uh, uw, h, w))
    for Y in range(uh):
        for X in range(uw):
            for k in range(5):
                for l in range(5):
                    y, x = 2 * Y - 2 + k, 2 * X - 2 + l
                    if not ((x < 0 or x >= w) and (y < 0 or y >= h)):
                        D[Y, X, _mirror(y, h), _mirror(x, w)] += binom5(k) * binom5(l)
    T = np.zeros_like(D)
    for y in range(h):
        Ys, wy = axis_sources(y, h, uh)
        for x in range(w):
            Xs, wx = axis_sources(x, w, uw)
            for a in range(5):
                for b in range(5):
                    if Ys[a] >= 0 and Xs[b] >= 0 and (a < 3 or b < 3):
                        T[Ys[a], Xs[b], y, x] += wy[a] * wx[b]
    np.testing.assert_array_equal(T, D)


@pytest.mark.parametrize("w,h", [(64, 40), (61, 33), (130, 31)])
def test_fast_path_loads(w, h):
    """The four-pixel path: two aligned floats at x / 2 and one on either side hold every source of its pixels."""
    uw, uh = (w + 1) // 2, (h + 1) // 2
    taken = 0
    for y in range(h):
        for x in range(0, w, 4):
            ub = ((x >> 1) - 1) & ~3 if (x >> 1) - 1 >= 0 else 0
            if not (x >= 8 and x + 10 <= w and y >= 6 and y + 7 <= h and ub + 8 <= uw and ((y + 2) >> 1) < uh):
                continue
            taken += 1
            cols = range((x >> 1) - 1, (x >> 1) + 3)
            assert cols[0] >= 0 and cols[-1] < uw and (x >> 1) % 2 == 0
            rows = [(y + 2 - ky) >> 1 for ky in range(y & 1, 5, 2)]
            assert min(rows) >= 0 and max(rows) < uh
            for i in range(4):
                got = [(cols[((i + 2 - kx) >> 1) + 1], binom5(kx), False) for kx in range(i & 1, 5, 2)]
                assert got == loops(x + i, w, uw)
    assert taken
