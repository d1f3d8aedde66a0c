"""Device memory that a caller gets from the library -- results, a plan's
outputs, a build plan's input -- is what cudaMalloc gives: an interprocess
handle can be taken, and other GPUs can map it, whatever its size."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ipc_status(ptr):
    import torch
    torch.cuda.init()
    rt = ctypes.CDLL(None)
    if not hasattr(rt, "cudaIpcGetMemHandle"):
        for line in open("/proc/self/maps"):
            if "libcudart" in line:
                rt = ctypes.CDLL(line.split()[-1])
                break
    handle = (ctypes.c_char * 64)()
    status = rt.cudaIpcGetMemHandle(ctypes.byref(handle), ctypes.c_void_p(int(ptr)))
    rt.cudaGetLastError()
    return status


@pytest.mark.parametrize("n,q,half", [(2000, 3, 0.05), (300_001, 40, 0.2), (4_000_000, 30, 0.5)])
def test_results(qcp, n, q, half):
    rng = np.random.default_rng(n)
    objs = rng.random((n, 3), dtype=np.float32)
    c = rng.random((q, 3), dtype=np.float32)
    boxes = np.concatenate([c - np.float32(half), c + np.float32(half)], 1)
    for _ in range(2):  # and buffers that an earlier index left
        with qcp.Index.build(objs) as ix:
            for algo in ("batched", "plain"):
                for _ in range(2):
                    res = ix.search(boxes, algo=algo, result_mem=qcp.MEM_DEVICE)
                    assert res.total_hits
                    assert ipc_status(res.offsets) == 0 and ipc_status(res.ids) == 0
                    res.release()
            plan = qcp.Plan(ix, q, 100_000)
            _, _, offs, ids = plan.run_device(np.ascontiguousarray(boxes[:1] * 0), q=1)
            assert ipc_status(offs) == 0 and ipc_status(ids) == 0
            plan.close()
    for m in (100, 200_000):
        plan = qcp.BuildPlan(m, 3)
        assert ipc_status(plan.input_ptr()) == 0
        plan.close()
