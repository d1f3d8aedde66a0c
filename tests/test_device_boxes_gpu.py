"""Boxes on the device: read in place (16-byte aligned) or from a copy, by
every traversal, with result slices of all sort classes in one batch -- ids
and counts equal the oracle's."""
import numpy as np
import pytest

from conftest import assert_same_hits

pytestmark = pytest.mark.gpu


def make(dims, n, q):
    rng = np.random.default_rng(n + dims)
    objs = rng.random((n, dims), dtype=np.float32)
    # from empty slices to all n ids: one warp's, one CTA's and the windows'
    side = np.float32(0.5) * np.geomspace(1e-5, 2.2, q).astype(np.float32) ** np.float32(1.0 / dims)
    c = rng.random((q, dims), dtype=np.float32)
    boxes = np.concatenate([c - side[:, None], c + side[:, None]], 1)
    return objs, np.ascontiguousarray(boxes[rng.permutation(q)])


@pytest.mark.parametrize("dims,n,q", [(1, 40_003, 1), (2, 120_001, 257), (3, 90_001, 300), (3, 127, 5),
                                      (8, 30_001, 64)])
def test_boxes_in_place_and_copied(qcp, oracle, dims, n, q):
    import torch
    objs, boxes = make(dims, n, q)
    offs, ids = oracle.ids(objs, dims, False, boxes)
    flat = torch.zeros(boxes.size + 8, dtype=torch.float32, device="cuda")
    with qcp.Index.build(objs) as ix:
        for shift in (0, 4, 1, 2):  # floats past a 256-byte boundary
            d = flat[shift:shift + boxes.size]
            d.copy_(torch.from_numpy(boxes.ravel()))
            torch.cuda.synchronize()
            for algo in ("batched", "plain", "hybrid"):
                for timing in (False, True):
                    res = ix.search(d, q=q, algo=algo, timing=timing)
                    assert_same_hits(res.offsets, res.ids, offs, ids)
                assert np.array_equal(ix.counts(d, q=q, algo=algo), np.diff(offs))
            res = ix.search(d, q=q, sort=False)
            assert np.array_equal(res.offsets, offs)
            for k in range(q):
                assert np.array_equal(np.sort(res.ids[int(offs[k]):int(offs[k + 1])]), ids[int(offs[k]):int(offs[k + 1])])
            assert np.array_equal(d.cpu().numpy(), boxes.ravel())
