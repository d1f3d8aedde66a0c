"""The build's sort where the keys' top bits do not tell objects apart: few
distinct points (long runs of equal keys), tight clusters (long runs of equal
top bits), runs around the length that is ordered in place, keys with few
effective bits, tile edges.  Keys and order equal a stable sort of the
oracle's keys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(kind, n, dims, rng):
    if kind == "one":
        return np.full((n, dims), 0.3, np.float32)
    if kind == "few":
        return rng.random((7, dims), dtype=np.float32)[rng.integers(0, 7, n)]
    if kind == "tight":  # a cube of side 2^-13 around each of three centres
        return (rng.random((3, dims), dtype=np.float32)[rng.integers(0, 3, n)] * np.float32(0.9)
                + rng.random((n, dims), dtype=np.float32) * np.float32(2.0 ** -13)).astype(np.float32)
    if kind == "corner":  # most objects clamped to one corner, the rest close to it
        p = np.maximum(rng.normal(0.0, 2.0 ** -13, (n, dims)), 0).astype(np.float32)
        p[rng.random(n) < 0.9] = 0
        return p
    if kind == "runs":  # groups of 1..40 objects within 2^-20 of each other
        c = rng.random((n // 20 + 1, dims), dtype=np.float32) * np.float32(0.9)
        return (c[rng.integers(0, len(c), n)] + rng.random((n, dims), dtype=np.float32) * np.float32(2.0 ** -20)
                ).astype(np.float32)
    return rng.random((n, dims), dtype=np.float32)


def test_longest_runs(qcp, oracle):
    """Runs about and beyond the longest that is ordered in place."""
    rng = np.random.default_rng(3)
    for n, dups in ((300_000, 262_100), (300_000, 262_200), (700_000, 600_000)):
        objs = (rng.random((n, 2), dtype=np.float32) * np.float32(2.0 ** -18)).astype(np.float32)
        objs[rng.permutation(n)[:dups]] = np.float32(2.0 ** -19)
        objs[:40] = 0.9  # the highest bits are used
        want = oracle.hilbert_keys(objs, 2, False, 32, 1)
        order = np.argsort(want, kind="stable")
        with qcp.Index.build(objs) as ix:
            keys, perm, _ = ix.export()
        assert np.array_equal(keys, want[order]) and np.array_equal(perm, order.astype(np.int32)), (n, dups)


@pytest.mark.parametrize("dims,bits,mode", [(3, 21, 0), (2, 32, 0), (2, 31, 1), (1, 32, 0), (4, 16, 0), (3, 11, 0),
                                            (5, 12, 0), (8, 8, 0), (6, 10, 0), (7, 9, 0), (3, 20, 1), (2, 17, 0),
                                            (4, 7, 0)])
@pytest.mark.parametrize("kind", ["one", "few", "tight", "corner", "runs", "uniform"])
def test_order(qcp, oracle, dims, bits, mode, kind):
    rng = np.random.default_rng(dims * 100 + bits)
    for n in (2, 3583, 3585, 20_001, 60_001):
        objs = points(kind, n, dims, rng)
        want = oracle.hilbert_keys(objs, dims, False, bits, 1 - mode)
        order = np.argsort(want, kind="stable")
        with qcp.Index.build(objs, key_mode=mode, key_bits=bits) as ix:
            keys, perm, _ = ix.export()
        assert np.array_equal(keys, want[order]), (kind, n)
        assert np.array_equal(perm, order.astype(np.int32)), (kind, n)
