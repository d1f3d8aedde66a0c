"""Batches that are not in node order and have more 32-leaf groups than the
grid's warps take in four rounds: items of few leaves, of many, and around the
line between them, trees of one level up, ragged last leaves, inverted and
infinite boxes -- ids and counts equal the oracle's, with and without recorded
hit bits and in a captured plan."""
import numpy as np
import pytest

from conftest import assert_same_hits

pytestmark = pytest.mark.gpu

WARPS = 148 * 8 * 8  # of the default grid


# (every batch has at least 8 WARPS / (fanout / 32) boxes, an item or more each: twice that)
@pytest.mark.parametrize("dims,rect,fanout,n,q,side", [
    (3, False, 256, 255, 10_000, 0.2), (2, False, 256, 60_001, 10_000, 0.1),  # one and two levels
    (3, False, 256, 150_001, 9_700, 0.01), (3, False, 256, 70_001, 12_000, 0.3), (3, False, 256, 70_001, 12_000, 0.15),
    (1, False, 224, 200_003, 12_000, 0.02), (4, True, 256, 100_001, 10_000, 0.3), (8, True, 128, 40_001, 20_000, 0.5),
    (5, False, 96, 50_001, 27_000, 0.4), (2, True, 32, 30_011, 78_000, 0.05), (6, True, 192, 30_001, 13_000, 0.5),
    (7, False, 160, 30_001, 16_000, 0.5)])
def test_counts_and_ids(qcp, oracle, dims, rect, fanout, n, q, side):
    rng = np.random.default_rng(n + q)
    lo = rng.random((n, dims), dtype=np.float32)
    objs = np.concatenate([lo, lo + rng.exponential(0.01, lo.shape).astype(np.float32)], 1) if rect else lo
    c = rng.random((q, dims), dtype=np.float32)
    half = (np.float32(side / 2) * rng.uniform(0.5, 1.5, (q, dims))).astype(np.float32)
    boxes = np.concatenate([c - half, c + half], 1)
    boxes[0, :dims], boxes[0, dims:] = -np.inf, np.inf
    boxes[1, :dims], boxes[1, dims:] = np.inf, -np.inf
    boxes[2, 0] = np.nan
    swapped = boxes[3:6].copy()
    boxes[3:6, :dims], boxes[3:6, dims:] = swapped[:, dims:], swapped[:, :dims]
    # the oracle on a part: rows of all kinds
    some = np.concatenate([np.arange(6), np.sort(rng.choice(np.arange(6, q), 150, replace=False))])
    offs, ids = oracle.ids(objs, dims, rect, boxes[some])
    want = np.diff(offs).astype(np.int64)

    def check(o, i):
        assert np.array_equal(np.diff(o.astype(np.int64))[some], want)
        got = np.concatenate([i[int(o[k]):int(o[k + 1])] for k in some])
        assert np.array_equal(got, ids)

    with qcp.Index.build(objs, is_rect=rect, fanout=fanout) as ix:
        all_counts = ix.counts(boxes, algo="plain").astype(np.int64)  # for the other rows
        assert np.array_equal(all_counts[some], want)
        assert np.array_equal(ix.counts(boxes).astype(np.int64), all_counts)
        for hit_cache in (0, 1):
            res = ix.search(boxes, hit_cache=hit_cache, timing=True)
            items = qcp.last_stats()["leaf_items"]
            check(res.offsets, res.ids)
            assert np.array_equal(np.diff(res.offsets.astype(np.int64)), all_counts)
        assert items * (fanout // 32) >= 8 * WARPS
        if len(res.ids) < 5e7:
            with qcp.Plan(ix, q, len(res.ids) + 1) as plan:
                got = plan.run(boxes)
                assert np.array_equal(got[0], res.offsets.astype(got[0].dtype)) and np.array_equal(got[1], res.ids)
