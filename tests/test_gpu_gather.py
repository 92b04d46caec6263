"""Results to the host at the sizes where the way changes: one pinned chunk
(straight from the kernel), several, and more than the ring holds."""
import numpy as np
import pytest

import dycgraph_b200 as dg

pytestmark = pytest.mark.gpu
INF = 0xFFFFFFFF


def star(n):
    off = np.full(n + 1, n - 1, np.uint64)
    off[0] = 0
    return off, np.arange(1, n, dtype=np.uint32)


@pytest.mark.parametrize("n", [2, 131_072, 131_073, 262_145, 1_300_001])
@pytest.mark.parametrize("queries", [0, 3])
def test_values_and_parents(n, queries):
    e = dg.Engine("bfs")
    e.load_csr(n, *star(n))
    if queries:
        e.set_queries([0, 1, n - 1][:queries], "batched")
    e.start()
    gone = np.unique([1, n // 2, n - 1])
    gone = gone[gone > 0]
    e.apply_batch([(0, int(v)) for v in gone], [])
    want = np.ones(n, np.uint32)
    want[0] = 0
    want[gone] = INF
    parents = np.where(want == 1, 0, INF).astype(np.uint32)
    v, p = e.gather()
    assert (v == want).all() and (p == parents).all()
    if queries:
        v, p = e.gather_query(2)
        assert v[n - 1] == 0 and int((v == INF).sum()) == n - 1 and (p == INF).all()


@pytest.mark.parametrize("n", [2, 262_144, 1_300_001])
def test_ranks(n):
    e = dg.Engine("pr", epsilon=1e-9)
    e.load_csr(n, *star(n))
    e.start()
    x, r = e.gather_ranks()
    want = np.full(n, 0.15 + 0.85 * 0.15 / (n - 1))
    want[0] = 0.15
    # two FP32 roundings of values below 1, and what stays below epsilon
    assert np.abs(x - want).max() <= 2 * 2.0 ** -24 + 1e-9
    assert np.abs(r).max() <= 1e-9
