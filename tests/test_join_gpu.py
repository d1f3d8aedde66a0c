"""The count and write passes at their edges: fan-outs with 1 to 8 leaf groups
and with half-filled warps, ragged last leaves, batches with and without node
order, hit bits that find no room, calls without them, and the captured
pipeline -- ids and counts equal the oracle's."""
import numpy as np
import pytest

from conftest import assert_same_hits

pytestmark = pytest.mark.gpu


def make(dims, rect, n, q, seed):
    rng = np.random.default_rng(seed)
    lo = (rng.random((n, dims), dtype=np.float32) ** 2).astype(np.float32)
    objs = lo
    if rect:
        objs = np.concatenate([lo, lo + rng.exponential(0.02, (n, dims)).astype(np.float32)], 1)
    c = lo[rng.integers(0, n, q)]
    # about as many ids in all for the larger sets
    side = 0.5 * min(1.0, (1e8 / (n * q)) ** (1.0 / dims))
    h = (rng.uniform(0.0, side, (q, 1)) * rng.uniform(0.5, 1.0, (q, dims))).astype(np.float32)
    if dims > 1:  # long boxes: many partially covered leaves for their ids
        h[:, 0] *= 12
        h[:, 1:] /= np.float32(12 ** (1 / (dims - 1)))
    boxes = np.concatenate([c - h, c + h], 1)
    boxes[0, :dims], boxes[0, dims:] = -np.inf, np.inf  # everything
    boxes[1, :dims], boxes[1, dims:] = 1.0, 0.0         # nothing
    boxes[2, 0] = np.nan                                # passes every test of that side
    boxes[3, 0], boxes[4, dims] = 0.0, -0.0             # zero bounds of either sign ...
    lo[:40, 0], lo[40:80, 0] = 0.0, -0.0                # ... against zero coordinates
    objs[:80, 0] = lo[:80, 0]
    return np.ascontiguousarray(objs, np.float32), np.ascontiguousarray(boxes, np.float32)


@pytest.mark.parametrize("dims,rect,fanout,n,q", [
    (3, False, 32, 33_001, 300), (2, True, 96, 50_001, 210), (4, False, 128, 70_001, 400), (1, False, 224, 20_001, 90),
    (5, True, 128, 35_001, 2047), (6, False, 192, 40_001, 70), (7, False, 32, 9_001, 2200), (3, False, 128, 127, 5),
    (8, True, 256, 70_003, 300),
    # at least 16,384 leaves and 2,048 boxes: node order
    (3, False, 32, 524_289, 2049), (2, False, 64, 1_048_600, 2048), (2, True, 96, 1_600_001, 2100),
    (8, True, 128, 2_097_200, 2700), (2, False, 160, 2_700_001, 3700)])
def test_counts_and_ids(qcp, oracle, dims, rect, fanout, n, q):
    objs, boxes = make(dims, rect, n, q, n)
    offs, ids = oracle.ids(objs, dims, rect, boxes)
    with qcp.Index.build(objs, is_rect=rect, fanout=fanout) as ix:
        assert np.array_equal(ix.counts(boxes), np.diff(offs))
        for hit_cache in (0, 1, 0):
            for lanes in (32, 16, 8):
                res = ix.search(boxes, hit_cache=hit_cache, lanes_per_item=lanes)
                assert_same_hits(res.offsets, res.ids, offs, ids)
        if n >= 500_000:
            ix.search(boxes, timing=True).release()
            st = qcp.last_stats()
            assert st["leaf_items"] >= max(24576, 12 * ix.info()["level_nodes"][1])
            assert st["hits"] == len(ids) and 0 < st["objects_covered"] < len(ids)
        with qcp.Plan(ix, q, len(ids) + 1) as plan:
            got = plan.run(boxes)
            assert_same_hits(got[0], got[1], offs, ids)
            got = plan.run(boxes[:3])
            assert_same_hits(got[0], got[1], offs[:4], ids[:int(offs[3])])


def test_hit_bits_without_room(qcp, oracle):
    # more partially covered leaves than the first call's hit bits hold
    # (2^21 words, 8 per leaf): the write pass tests the rest
    objs, boxes = make(2, False, 524_301, 3000, 5)
    boxes[3:, 1] = -1.0
    boxes[3:, 3] = 2.0
    boxes[3:, 0] = np.random.default_rng(6).random(len(boxes) - 3, dtype=np.float32) ** 2
    boxes[3:, 2] = boxes[3:, 0] + np.float32(2e-3)
    offs, ids = oracle.ids(objs, 2, False, boxes)
    with qcp.Index.build(objs, fanout=32) as ix:
        for q in (2000, 3000, 3000):  # not in node order, in node order, with room
            res = ix.search(boxes[:q], timing=True)
            assert_same_hits(res.offsets, res.ids, offs[:q + 1], ids[:int(offs[q])])
            assert qcp.last_stats()["leaves_partial"] * 8 > 1 << 21
