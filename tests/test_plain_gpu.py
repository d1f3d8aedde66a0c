"""The plain traversal at its edges: fan-outs from one warp's to one CTA's,
one to four levels, ragged last leaves, lists of leaves that fill up more than
once, boxes over everything and nothing, rectangles with lo > hi -- ids, their
key order without the sort, and counts."""
import numpy as np
import pytest

from conftest import assert_same_hits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,rect,fanout,n,q", [
    (3, False, 32, 31, 9), (3, False, 32, 33, 9), (2, False, 32, 40_001, 60), (2, True, 96, 70_001, 60),
    (3, False, 128, 200_003, 80), (1, False, 160, 30_001, 40), (2, False, 256, 300_007, 40),
    (4, True, 128, 20_001, 50), (8, False, 224, 30_001, 40), (6, True, 32, 9_001, 40)])
def test_plain(qcp, oracle, dims, rect, fanout, n, q):
    rng = np.random.default_rng(n)
    objs = rng.random((n, dims), dtype=np.float32)
    if rect:
        objs = np.concatenate([objs, objs + rng.normal(0.02, 0.02, objs.shape).astype(np.float32)], 1)
    half = rng.uniform(0, 0.5, (q, dims)).astype(np.float32) ** np.float32(2.0 if dims < 4 else 0.5)
    c = rng.random((q, dims), dtype=np.float32)
    boxes = np.concatenate([c - half, c + half], 1)
    boxes[0, :dims], boxes[0, dims:] = -np.inf, np.inf
    boxes[1, :dims], boxes[1, dims:] = 1.0, 0.0
    boxes[2, 0] = np.nan
    offs, ids = oracle.ids(objs, dims, rect, boxes)
    with qcp.Index.build(objs, is_rect=rect, fanout=fanout) as ix:
        res = ix.search(boxes, algo="plain")
        assert_same_hits(res.offsets, res.ids, offs, ids)
        assert np.array_equal(ix.counts(boxes, algo="plain"), np.diff(offs))
        place = np.empty(n, np.int64)
        place[ix.export()[1]] = np.arange(n)
        res = ix.search(boxes, algo="plain", sort=False)
        assert np.array_equal(res.offsets, offs)
        for k in range(q):
            got = res.ids[int(offs[k]):int(offs[k + 1])]
            assert np.all(np.diff(place[got]) > 0)
            assert np.array_equal(np.sort(got), ids[int(offs[k]):int(offs[k + 1])])
