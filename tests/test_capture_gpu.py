"""Calls on a stream that is being captured: they allocate and wait, so they
are refused, leave the capture as it was, and the index answers the next
ordinary call -- with workspaces that are new and that have been used."""
import numpy as np
import pytest

from conftest import assert_same_hits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("used", [False, True])
def test_refused_while_capturing(qcp, oracle, used):
    import torch
    rng = np.random.default_rng(5)
    objs = rng.random((200_003, 3), dtype=np.float32)
    c = rng.random((300, 3), dtype=np.float32)
    boxes = np.concatenate([c - np.float32(0.1), c + np.float32(0.1)], 1)
    offs, ids = oracle.ids(objs, 3, False, boxes)
    d_objs, d_boxes = torch.from_numpy(objs).cuda(), torch.from_numpy(boxes).cuda()
    x = torch.zeros(8, device="cuda")
    st = torch.cuda.Stream()
    with qcp.Index.build(objs) as ix:
        if used:
            ix.search(boxes, stream=st.cuda_stream)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(st):
            graph.capture_begin(capture_error_mode="relaxed")
            x.add_(1)
            calls = [lambda: ix.search(boxes, stream=st.cuda_stream),
                     lambda: ix.search(d_boxes, q=300, stream=st.cuda_stream, result_mem=qcp.MEM_DEVICE),
                     lambda: ix.search(boxes, algo="plain", stream=st.cuda_stream),
                     lambda: ix.counts(boxes, stream=st.cuda_stream),
                     lambda: qcp.Index.build(d_objs, dims=3, n=len(objs), stream=st.cuda_stream)]
            for call in calls:
                with pytest.raises(qcp.QcpError) as err:
                    call()
                assert err.value.status == 5  # QCP_ERR_CUDA
            graph.capture_end()
        torch.cuda.synchronize()
        for stream in (0, st.cuda_stream):
            res = ix.search(boxes, stream=stream)
            assert_same_hits(res.offsets, res.ids, offs, ids)
            assert np.array_equal(ix.counts(boxes, stream=stream), np.diff(offs))
        # the capture holds its own work and nothing of the calls
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, torch.ones_like(x))
