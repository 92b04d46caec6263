"""Ingest and mutation at the edges of their forms, slot order included: batch
sizes around the block sorts' capacities and above them (the device-wide sort),
unequal numbers of deletions and insertions, repeated, missing and out-of-range
records, and rows whose unsorted suffix is matched by chunks (duplicates of one
neighbour on both sides of what a deletion asks for). The model is the
occurrence semantics themselves: a deletion removes the first live occurrences
in slot order, insertions append sorted by neighbour, equal ones in arrival
order; in-rows the same with the roles exchanged."""
import numpy as np
import pytest

import dycgraph_b200 as dg
from tests import cases

pytestmark = pytest.mark.gpu
N = 3000


class Rows:
    def __init__(self, src, dst, w):
        self.rows = [[] for _ in range(N)]
        self.add(src, dst, w)

    def remove(self, src, dst):
        missing = 0
        for u, v in zip(src.tolist(), dst.tolist()):
            row = self.rows[u]
            at = next((i for i, x in enumerate(row) if x[0] == v), None)
            if at is None:
                missing += 1
            else:
                del row[at]
        return missing

    def add(self, src, dst, w):
        order = np.lexsort((np.arange(len(src)), dst, src))
        for i in order.tolist():
            self.rows[src[i]].append((int(dst[i]), int(w[i])))

    def flat(self):
        return [x for r in self.rows for x in r]


def batch(rng, out, nd, na, hub):
    u, v = rng.integers(0, N, na), rng.integers(0, N, na)
    u[: na // 3] = hub                      # a long suffix ...
    v[: na // 3] = rng.integers(0, 40, na // 3)  # ... with many occurrences of few neighbours
    v[na // 3: na // 2] = hub + 1           # and the same for an in-row
    a = np.stack([u, v, rng.integers(1, 65, na)], 1)
    live = [(s, x[0]) for s in rng.permutation(N)[:400].tolist() for x in out.rows[s][:6]]
    live += [(hub, x[0]) for x in out.rows[hub][:nd // 2]]
    pick = rng.integers(0, max(1, len(live)), nd)
    d = np.array([live[i] + (1,) for i in pick.tolist()] if live else np.zeros((nd, 3)), np.int64)
    d = d.reshape(-1, 3)
    gone = rng.random(nd) < 0.1
    d[gone, 1] = rng.integers(0, N, int(gone.sum()))  # mostly missing
    for r in (d, a):                                 # records without such a vertex
        bad = rng.random(len(r)) < 0.02
        r[bad, rng.integers(0, 2)] = N + rng.integers(0, 9)
    return d.astype(np.uint32), a.astype(np.uint32)


def valid(r):
    return r[(r[:, 0] < N) & (r[:, 1] < N)].astype(np.int64)


@pytest.mark.parametrize("replay", [False, True])
@pytest.mark.parametrize("nd,na", [(1, 0), (0, 1), (128, 128), (129, 60), (1024, 1025),
                                   (300, 4097), (4096, 700), (8192, 8192), (8193, 8192),
                                   (100, 30_000)])
def test_batches_leave_the_rows_the_model_has(nd, na, replay):
    rng = np.random.default_rng(nd * 31 + na)
    n, m = N, 20_000
    key = np.unique(rng.integers(0, N, m) * N + rng.integers(0, N, m))
    src, dst = key // N, key % N
    w = rng.integers(1, 65, len(key))
    off = np.concatenate([[0], np.bincount(src, minlength=N).cumsum()]).astype(np.uint64)
    e = dg.Engine("sssp", weight_mode="stored", page_shift=8, hbm_graph_budget_bytes=4 << 20)
    e.load_csr(n, off, dst.astype(np.uint32), w.astype(np.uint32))
    if replay:
        e.set_queries([0], "batched")
    e.start()
    out, inc = Rows(src, dst, w), Rows(dst, src, w)
    for step in range(4):
        d, a = batch(rng, out, nd, na, hub=7)
        st = e.apply_batches([(d, a)])[0] if replay else e.apply_batch(d, a)
        vd, va = valid(d), valid(a)
        missing = out.remove(vd[:, 0], vd[:, 1])
        inc.remove(vd[:, 1], vd[:, 0])
        out.add(va[:, 0], va[:, 1], va[:, 2])
        inc.add(va[:, 1], va[:, 0], va[:, 2])
        assert st["missing_deletes"] == missing
        assert st["invalid_updates"] == len(d) + len(a) - len(vd) - len(va)
        o, gd, gw = e.csr()
        want = out.flat()
        assert [int(x) for x in np.diff(o.astype(np.int64))] == [len(r) for r in out.rows]
        assert (gd == [x[0] for x in want]).all(), step
        assert (gw == [x[1] for x in want]).all(), step
        for v in (0, 7, 8, 9, 39):
            gd, gw = e.row(v, incoming=True)
            assert gd.tolist() == [x[0] for x in inc.rows[v]], (step, v)
            assert gw.tolist() == [x[1] for x in inc.rows[v]], (step, v)
