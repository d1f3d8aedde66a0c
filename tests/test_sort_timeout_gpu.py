"""A wait of the build's sort that runs out, by a limit of no polls at all: the
build and the captured build return the timeout status, nothing is read or
written through the incomplete pairs, and the same objects build again."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = 4


@pytest.fixture
def polls(qcp):
    lib = qcp.load_library()
    yield lambda n: lib.qcp_test_sort_polls(ctypes.c_int(n))
    lib.qcp_test_sort_polls(ctypes.c_int(-1))


@pytest.mark.parametrize("dims,bits,rect", [(3, 0, False), (3, 10, False), (2, 0, True)])
def test_expired_wait(qcp, oracle, polls, dims, bits, rect):
    n = 3_000_001  # a thousand tiles: far more than run at once
    rng = np.random.default_rng(n + dims + bits)
    objs = rng.random((n, dims), dtype=np.float32)
    if rect:
        objs = np.concatenate([objs, objs + np.float32(0.001)], 1)
    polls(0)
    for _ in range(3):
        with pytest.raises(qcp.QcpError) as err:
            qcp.Index.build(objs, is_rect=rect, key_bits=bits)
        assert err.value.status == TIMEOUT
    polls(-1)
    want = oracle.hilbert_keys(objs, dims, rect, bits or (21 if dims == 3 else 32), 1)
    order = np.argsort(want, kind="stable")
    with qcp.Index.build(objs, is_rect=rect, key_bits=bits) as ix:
        keys, perm, _ = ix.export()
    assert np.array_equal(keys, want[order]) and np.array_equal(perm, order.astype(np.int32))


def test_expired_wait_in_a_captured_build(qcp, oracle, polls):
    n = 3_000_001
    objs = np.random.default_rng(9).random((n, 3), dtype=np.float32)
    boxes = np.array([[0.2] * 3 + [0.21] * 3, [0.5] * 3 + [0.6] * 3], np.float32)
    offs, ids = oracle.ids(objs, 3, False, boxes)
    polls(0)
    plan = qcp.BuildPlan(n, 3)  # the limit is recorded with the launches
    polls(-1)
    for _ in range(2):
        with pytest.raises(qcp.QcpError) as err:
            plan.run(objs)
        assert err.value.status == TIMEOUT
    plan.close()
    plan = qcp.BuildPlan(n, 3)
    res = plan.run(objs).search(boxes)
    assert np.array_equal(res.offsets, offs) and np.array_equal(res.ids, ids)
    plan.close()


@pytest.mark.parametrize("n", [3071, 3072, 3073, 6143, 6144, 6145])
@pytest.mark.parametrize("dims,bits", [(1, 32), (3, 21), (2, 32)])
def test_tile_edges(qcp, oracle, n, dims, bits):
    """Tiles exactly full, one pair over and one short, with most of the last
    digits 255: those share a counter with the slots past a short tile's end."""
    rng = np.random.default_rng(n + dims)
    for share in (0.0, 0.7, 1.0):
        objs = rng.random((n, dims), dtype=np.float32)
        objs[rng.random(n) < share] = 1.0
        want = oracle.hilbert_keys(objs, dims, False, bits, 1)
        order = np.argsort(want, kind="stable")
        with qcp.Index.build(objs, key_bits=bits) as ix:
            keys, perm, _ = ix.export()
        assert np.array_equal(keys, want[order]), share
        assert np.array_equal(perm, order.astype(np.int32)), share
