"""k-means-clustered keys at the edges of the assignment kernel's centre
groups and tiles (8 and 1,024 centres), of its object blocks, with ties and
with coinciding centres, for every dimension count: keys and order equal the
oracle's restatement bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n,K", [(1, 5000, 1), (2, 257, 7), (3, 1000, 9), (4, 2049, 1023), (5, 1500, 1025),
                                      (6, 700, 16), (7, 900, 700), (8, 600, 24), (3, 640_001, 40), (6, 330_003, 33)])
def test_assignment_edges(qcp, oracle, dims, n, K):
    rng = np.random.default_rng(n + K)
    # a coarse grid: many objects coincide and many distances tie
    objs = (rng.integers(0, 12, (n, dims)) / 16).astype(np.float32)
    bits = min(21, 64 // dims)
    want = oracle.kmeans_keys(objs, dims, False, bits, K, 4)
    order = oracle.sort_perm(want)
    with qcp.Index.build(objs, key_mode=qcp.KEY_KMEANS, key_bits=bits, kmeans_clusters=K, kmeans_iters=4) as ix:
        keys, perm, _ = ix.export()
    assert np.array_equal(keys, want[order])
    assert np.array_equal(perm, order.astype(np.int32))
