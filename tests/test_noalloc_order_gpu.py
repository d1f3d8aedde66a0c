"""The allocation-free counts of large batches over many leaves, which go in
node order as the other counts do: equal to the oracle's, nothing allocated, and
about as quick as the others."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def noalloc(qcp, ix, d_boxes, d_counts):
    lib = qcp.load_library()
    assert lib.qcp_query_counts_noalloc(ix._h, ctypes.c_void_p(d_boxes.data_ptr()), d_boxes.shape[0],
                                        ctypes.c_void_p(d_counts.data_ptr()), None) == 0, lib.qcp_last_error()


@pytest.mark.parametrize("dims,fanout,n,q", [(2, 32, 530_001, 1024), (2, 32, 530_001, 4000), (3, 64, 1_100_003, 2500)])
def test_counts(qcp, oracle, dims, fanout, n, q):
    import torch
    rng = np.random.default_rng(q)
    objs = rng.random((n, dims), dtype=np.float32)
    c = rng.random((q, dims), dtype=np.float32)
    half = np.float32(0.5 * 0.002 ** (1 / dims))
    boxes = np.concatenate([c - half, c + half], 1)
    want = np.diff(oracle.ids(objs, dims, False, boxes)[0]).astype(np.int64)
    d_boxes = torch.from_numpy(boxes).cuda()
    with qcp.Index.build(objs, fanout=fanout) as ix:
        for k in range(3):
            m = q if k < 2 else 900  # too few boxes for it
            d_counts = torch.full((m,), -1, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            noalloc(qcp, ix, d_boxes[:m].contiguous(), d_counts)
            torch.cuda.synchronize()
            assert k == 0 or torch.cuda.mem_get_info()[0] == free
            assert np.array_equal(d_counts.cpu().numpy(), want[:m])


def test_as_quick_as_the_other_counts(qcp):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    n, q = 8_000_000, 20_000
    which = torch.randint(0, 64, (n,), generator=g, device="cuda")
    objs = (torch.randn((n, 3), generator=g, device="cuda") * 0.02
            + torch.rand((64, 3), generator=g, device="cuda")[which]).clamp_(0, 0.999999).contiguous()
    c = objs[torch.randint(0, n, (q,), generator=g, device="cuda")]
    boxes = torch.cat([c - 0.012, c + 0.012], 1).contiguous()
    counts = torch.zeros(q, dtype=torch.int64, device="cuda")
    with qcp.Index.build(objs, dims=3, n=n) as ix:
        def ms(call):
            runs = []
            for _ in range(9):
                torch.cuda.synchronize()
                t = time.perf_counter()
                call()
                runs.append((time.perf_counter() - t) * 1e3)
            return sorted(runs)[4]
        free = ms(lambda: noalloc(qcp, ix, boxes, counts))
        other = ms(lambda: ix.counts(boxes, q=q))
        assert np.array_equal(counts.cpu().numpy(), ix.counts(boxes, q=q).astype(np.int64))
    assert free < 1.2 * other, (free, other)
