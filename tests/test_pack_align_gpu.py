"""Device objects at addresses that are only float-aligned, every row width, and
fan-outs that leave threads of a block without a leaf: keys, order and leaf
MBRs equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,rect,fanout", [(1, False, 32), (2, False, 96), (3, False, 160), (4, False, 128),
                                              (2, True, 224), (4, True, 64), (8, True, 256), (5, False, 192),
                                              (7, True, 32), (6, False, 128)])
@pytest.mark.parametrize("skip", [0, 1, 2])
def test_rows_at_any_float_address(qcp, oracle, dims, rect, fanout, skip):
    import torch
    rng = np.random.default_rng(dims + fanout)
    n = 5 * fanout + 7
    lo = rng.normal(0.5, 0.4, (n, dims)).astype(np.float32)  # some below 0 and above 1
    objs = np.concatenate([lo, lo + rng.random((n, dims), dtype=np.float32)], 1) if rect else lo
    objs = np.ascontiguousarray(objs, np.float32)
    buf = torch.zeros(objs.size + skip, device="cuda")
    buf[skip:] = torch.from_numpy(objs).cuda().reshape(-1)
    bits = min(21, 64 // dims)
    want = oracle.hilbert_keys(objs, dims, rect, bits, 1)
    order = np.argsort(want, kind="stable")
    with qcp.Index.build(buf[skip:], dims=dims, n=n, is_rect=rect, fanout=fanout, key_bits=bits) as ix:
        keys, perm, mbr = ix.export(level=0)
    assert np.array_equal(keys, want[order])
    assert np.array_equal(perm, order.astype(np.int32))
    assert np.array_equal(mbr, oracle.node_mbrs(objs[order], dims, rect, fanout)[0])
