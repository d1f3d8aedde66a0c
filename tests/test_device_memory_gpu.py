"""Device memory that an index leaves behind: no more than 2 GiB of what its
results and workspaces took, once they are freed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_memory_is_given_back(qcp):
    import torch
    rng = np.random.default_rng(2)
    objs = rng.random((5_000_000, 3), dtype=np.float32)
    whole = np.tile(np.float32([-1, -1, -1, 2, 2, 2]), (10, 1))
    torch.cuda.synchronize()
    qcp.Index.build(objs[:1000]).close()  # the library's own start
    before = torch.cuda.mem_get_info()[0]
    ix = qcp.Index.build(objs)
    held = [ix.search(whole, result_mem=qcp.MEM_DEVICE) for _ in range(16)]  # 200 MB of ids each
    assert all(r.total_hits == 50_000_000 for r in held)
    assert before - torch.cuda.mem_get_info()[0] > 16 * 200e6
    for r in held:
        r.release()
    ix.close()
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < (2 << 30) + (64 << 20)
