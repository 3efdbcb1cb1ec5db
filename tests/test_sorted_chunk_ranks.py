"""The selection's ranks from sorted chunks (final_kernel, select.cu), restated on the CPU: the branch-free binary
searches of a key in every chunk of 2048 read inside the keys and add up to its rank, as counting does."""

import numpy as np
import pytest

CHUNK, MAX_KEYS = 2048, 16384


@pytest.mark.parametrize("n", [2049, 2050, 4095, 4096, 4097, 6000, 12289, 16383, 16384])
@pytest.mark.parametrize("spread", [1 << 60, 1 << 14])
def test_ranks(n, spread):
    rng = np.random.default_rng(n)
    keys = rng.choice(spread, n, replace=False) if spread < 1 << 20 else np.unique(rng.integers(0, spread, 2 * n))
    keys = rng.permutation(keys)[:n].astype(np.int64)
    order = np.argsort(np.argsort(keys))
    for at in range(0, n, CHUNK):
        part = slice(at, min(n, at + CHUNK))
        o = np.argsort(keys[part])
        keys[part], order[part] = keys[part][o], order[part][o]
    rank = np.zeros(n, np.int64)
    for q in range(MAX_KEYS // CHUNK):
        less, step = np.zeros(n, np.int64), CHUNK
        while step:
            at = q * CHUNK + less + step
            ok = at <= min(n, (q + 1) * CHUNK)
            assert (at[ok] >= 1).all() and (at[ok] <= n).all()
            ok[ok] = keys[at[ok] - 1] < keys[ok]
            less[ok] += step
            step >>= 1
        rank += less
    assert np.array_equal(rank, order) and len(set(rank)) == n
