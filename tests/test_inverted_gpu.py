"""Rectangles with lo > hi in some dimension, which can miss a box that covers
their leaf's MBR: every traversal, batch size and kind of index tests them one
by one, and an index rebuilt without them counts whole leaves again -- ids and
counts equal the oracle's."""
import ctypes

import numpy as np
import pytest

from conftest import assert_same_hits

pytestmark = pytest.mark.gpu


def make(dims, n, q, share, seed):
    rng = np.random.default_rng(seed)
    lo = rng.random((n, dims), dtype=np.float32)
    hi = lo + rng.exponential(0.01, (n, dims)).astype(np.float32)
    inv = rng.random((n, dims)) < share
    lo, hi = np.where(inv, hi, lo), np.where(inv, lo, hi)
    c = rng.random((q, dims), dtype=np.float32)
    half = rng.uniform(0, 0.3, (q, dims)).astype(np.float32) * np.float32(min(1.0, (3e8 / n / q) ** (1 / dims)))
    boxes = np.concatenate([c - half, c + half], 1)
    boxes[0, :dims], boxes[0, dims:] = -1, 2  # covers everything
    return np.concatenate([lo, hi], 1), boxes


@pytest.mark.parametrize("dims,fanout,n,q,share", [
    (1, 32, 31, 20, 0.5), (1, 64, 40_001, 200, 0.3), (2, 96, 60_001, 300, 0.001), (3, 128, 50_001, 200, 1.0),
    (8, 256, 20_001, 60, 0.1),
    (2, 32, 600_001, 2100, 1e-5)])  # node order
def test_inverted(qcp, oracle, tmp_path, dims, fanout, n, q, share):
    import torch
    objs, boxes = make(dims, n, q, share, n)
    offs, ids = oracle.ids(objs, dims, True, boxes)
    with qcp.Index.build(objs, is_rect=True, fanout=fanout) as built:
        built.save(str(tmp_path / "ix"))
        with qcp.Index.load(str(tmp_path / "ix")) as loaded:
            for ix in (built, loaded):
                for algo in ("batched", "plain", "hybrid"):
                    res = ix.search(boxes, algo=algo)
                    assert_same_hits(res.offsets, res.ids, offs, ids)
                    assert np.array_equal(ix.counts(boxes, algo=algo), np.diff(offs))
                res = ix.search(boxes, hit_cache=1)
                assert_same_hits(res.offsets, res.ids, offs, ids)
                d_boxes = torch.from_numpy(boxes).cuda()
                d_counts = torch.zeros(q, dtype=torch.int64, device="cuda")
                torch.cuda.synchronize()
                lib = qcp.load_library()
                assert lib.qcp_query_counts_noalloc(ix._h, ctypes.c_void_p(d_boxes.data_ptr()), q,
                                                    ctypes.c_void_p(d_counts.data_ptr()), None) == 0
                assert np.array_equal(d_counts.cpu().numpy(), np.diff(offs))
                with qcp.Plan(ix, q, len(ids) + 1) as plan:
                    got = plan.run(boxes)
                    assert_same_hits(got[0], got[1], offs, ids)


def test_rebuilt(qcp, oracle):
    plan = qcp.BuildPlan(30_001, 2, is_rect=True)
    for share in (0.0, 0.2, 0.0):
        objs, boxes = make(2, 30_001, 100, share, 7)
        offs, ids = oracle.ids(objs, 2, True, boxes)
        ix = plan.run(objs)
        res = ix.search(boxes, timing=True)
        covered = qcp.last_stats()["leaves_covered"]
        assert (covered == 0) if share else (covered > 0)
        assert_same_hits(res.offsets, res.ids, offs, ids)
    plan.close()
