"""The work counters of a timed plain traversal: its own, whatever ran on the
workspace before -- nothing (its memory is new), a batched call, itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_counters(qcp):
    rng = np.random.default_rng(4)
    objs = rng.random((400_001, 2), dtype=np.float32)
    whole = np.tile(np.float32([-1, -1, 2, 2]), (3, 1))  # slices sorted through windows
    some = np.float32([[0.1, 0.1, 0.2, 0.2]])
    qcp.Index.build(objs).search(whole, timing=True)  # leaves used memory behind
    for first in (None, "batched", "plain"):
        with qcp.Index.build(objs) as ix:
            if first:
                ix.search(whole, algo=first, timing=True)
            for boxes, windows in ((whole, 3 * len(objs)), (some, 0)):
                res = ix.search(boxes, algo="plain", timing=True)
                st = qcp.last_stats()
                assert st["hits"] == res.total_hits
                assert st["sort_window_ids"] == windows
                # the plain traversal counts no leaves and no frontier
                assert st["leaves_covered"] == st["leaves_partial"] == st["objects_covered"] == 0
                assert not any(st["frontier_items"]) and st["leaf_items"] == 0
