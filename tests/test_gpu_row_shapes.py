"""Row lengths and wave sizes at the edges of the repair kernels' work
distribution, against the oracle: rows around an 8-lane group's, a warp's and a
CTA tile's slots, waves around the launch's warp count (one, two and four rows
per warp), ordered and unordered closures."""
import numpy as np
import pytest

import dycgraph_b200 as dg
import oracle
from tests import cases

pytestmark = pytest.mark.gpu

ALGO = {"sssp": oracle.SSSP, "bfs": oracle.BFS, "cc": oracle.CC}
LENGTHS = [0, 1, 7, 8, 9, 31, 32, 33, 63, 64, 65]
LONG = [127, 128, 129, 255, 256, 257, 4095, 4096, 4097, 9000]


def fan(width, seed):
    """0 -> 1..width, whose rows cycle through LENGTHS (the first ones through
    LONG), into n - width targets; the last vertex has an in-edge from every row."""
    rng = np.random.default_rng(seed)
    n = width + 20_000
    u, v = [np.zeros(width, np.int64)], [np.arange(1, width + 1)]
    for i in range(1, width + 1):
        k = LONG[i - 1] if i <= len(LONG) else LENGTHS[i % len(LENGTHS)]
        u.append(np.full(k, i))
        t = rng.choice(n - width - 1, size=k, replace=False) + width + 1 if k else np.zeros(0, np.int64)
        if k:
            t[0] = n - 1
        v.append(t)
    key = np.unique(np.concatenate(u) * n + np.concatenate(v))
    uu, vv = key // n, key % n
    off = np.zeros(n + 1, np.uint64)
    np.add.at(off, uu + 1, 1)
    return n, np.cumsum(off).astype(np.uint64), vv.astype(np.uint32), cases.hw(uu, vv)


@pytest.mark.parametrize("algo,stored,delta", [("sssp", True, 0), ("sssp", True, 40),
                                               ("sssp", False, 0), ("bfs", False, 1),
                                               ("cc", False, 0), ("cc", False, 1)])
@pytest.mark.parametrize("width", [31, 4736, 4737, 9473])
def test_row_lengths_and_wave_sizes(width, algo, stored, delta):
    n, off, dst, w = fan(width, width)
    e = dg.Engine(algo, weight_mode="stored" if stored else "hash128", ordered_delta=delta)
    e.load_csr(n, off, dst, w if stored else None)
    e.start()
    orc = oracle.Oracle(ALGO[algo], n, off, dst, w if stored else None,
                        weight_mode=oracle.WEIGHT_STORED if stored else oracle.WEIGHT_HASH128)
    orc.init()
    assert (e.gather()[0] == orc.values()[0]).all()
    rng = np.random.default_rng(width + 1)
    hit = rng.permutation(width)[:max(20, width * 3 // 4)] + 1
    hit = np.unique(np.concatenate([hit[hit <= width], np.arange(1, min(width, 10) + 1)]))
    gone = [(0, int(x), int(w[x - 1]) if stored else 1) for x in hit]
    back = [(0, int(x), 3) for x in hit[::2]]
    for dels, adds in ((gone, []), ([], back), (back, gone)):
        e.apply_batch(dels, adds)
        orc.apply_batch(dels, adds)
        assert (e.gather()[0] == orc.values()[0]).all()
