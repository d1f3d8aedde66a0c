"""Sorts of enough objects that the keys are sampled first: objects that share
their keys' top bits never, now and then, mostly and always, and many equal
keys (which do not count as sharing) -- order and keys equal a stable sort of
the oracle's.  And close objects cost about what the sweeps they need cost."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (1 << 19) + 4097


def points(kind, dims, rng):
    x = rng.random((N, dims), dtype=np.float32)
    if kind == "spread":
        return x
    if kind.startswith("cube"):  # a small cube, a few objects elsewhere
        x[40:] = x[40:] * np.float32(2.0 ** -int(kind[4:])) + np.float32(0.3)
        return x
    if kind == "few":
        return x[:900][rng.integers(0, 900, N)]
    if kind == "origin":  # nine in ten have the key 0
        x[rng.random(N) < 0.9] = 0
        return x
    half = rng.random(N) < 0.5  # half of them close together
    x[half] = x[half] * np.float32(2.0 ** -12) + np.float32(0.7)
    return x


@pytest.mark.parametrize("dims,bits", [(3, 21), (2, 32), (8, 8), (5, 7)])
@pytest.mark.parametrize("kind", ["spread", "cube3", "cube5", "cube7", "cube11", "few", "origin", "half"])
def test_order(qcp, oracle, dims, bits, kind):
    objs = np.ascontiguousarray(points(kind, dims, np.random.default_rng(dims)))
    want = oracle.hilbert_keys(objs, dims, False, bits, 1)
    order = np.argsort(want, kind="stable")
    with qcp.Index.build(objs, key_bits=bits) as ix:
        keys, perm, _ = ix.export()
    assert np.array_equal(keys, want[order])
    assert np.array_equal(perm, order.astype(np.int32))


def test_close_objects_cost_little_more(qcp):
    """12 M objects in 64 clusters, spread or close: eight sweeps instead of
    four are less than 1.7 times the rebuild (four, then eight, were twice)."""
    import torch
    n = 12_000_000
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    which = torch.randint(0, 64, (n,), generator=g, device="cuda")
    centres = torch.rand((64, 3), generator=g, device="cuda")
    noise = torch.randn((n, 3), generator=g, device="cuda")
    plan = qcp.BuildPlan(n, 3)
    ms = []
    for sigma in (0.03, 0.0005):
        objs = (noise * sigma + centres[which]).clamp_(0, 0.999999).contiguous()
        runs = []
        for _ in range(9):
            torch.cuda.synchronize()
            t = time.perf_counter()
            plan.run(objs)
            runs.append(time.perf_counter() - t)
        ms.append(sorted(runs)[len(runs) // 2] * 1e3)
    plan.close()
    assert ms[1] < 1.7 * ms[0], ms
