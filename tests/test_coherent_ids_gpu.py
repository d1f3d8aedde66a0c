"""Sorted slices whose ids are not spread over [0, n): runs of consecutive
ids, clumps far apart, strided ids -- at the edges of the one-warp, one-CTA
and window sorts.  Every query is an interval of a 1-D set whose objects are
given chosen ids, so the expected slice is known; equality is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 21
SIZES = [2, 31, 33, 257, 1023, 1024, 1025, 4097, 8191, 8192, 8193, 9000]


def pick(pattern, size, rng):
    """`size` distinct ids of [0, N)."""
    if pattern == "run":
        return np.arange(size) + rng.integers(0, N - size)
    if pattern == "strided":
        return np.arange(size) * 64 + rng.integers(0, N - 64 * size)
    if pattern == "clumps":  # four dense runs far apart: crowded buckets
        at = np.sort(rng.choice(N >> 15, 4, replace=False)) << 15
        return np.unique(np.concatenate([a + np.arange(-(-size // 4)) for a in at]))[:size]
    if pattern == "tails":  # most ids in one region, dense runs of 40 elsewhere
        k = min(size, 40)
        tail = np.concatenate([(w << 17) + 7 + np.arange(k) for w in (3, 9, 15)])[:size // 2]
        body = rng.choice(1 << 16, size - len(tail), replace=False) + (5 << 17)
        return np.concatenate([body, tail])
    return rng.choice(N, size, replace=False)


@pytest.mark.parametrize("pattern", ["run", "strided", "clumps", "tails", "random"])
def test_slices_of_coherent_ids(qcp, pattern):
    rng = np.random.default_rng(11)
    for size in SIZES:
        want = np.unique(pick(pattern, size, rng))
        x = np.full((N, 1), 0.75, np.float32)
        x[want, 0] = 0.25
        with qcp.Index.build(x) as ix:
            res = ix.search(np.array([[0.2, 0.3], [0.8, 0.9]], np.float32))
        assert np.array_equal(res.hits(0), want), (pattern, size)
        assert len(res.hits(1)) == 0
