"""Deletions of edges that occur many times in a long unsorted suffix, fewer of them than
there are: the earliest occurrences go, whatever the multiplicities, and the suffix is
read a bounded number of times for all records together (a walk of it per record read
gigabytes for a snapshot of Zipf-distributed updates). Weights name the occurrences:
each has its own."""
import numpy as np
import pytest

import dycgraph_b200 as dg

pytestmark = pytest.mark.gpu


def first_ones_gone(row, gone):
    """Indices of `row` that stay when each neighbour of `gone` loses an occurrence per
    mention, earliest first; and the mentions that found none."""
    order = np.argsort(row, kind="stable")
    ids, start, count = np.unique(row[order], return_index=True, return_counts=True)
    rank = np.empty(len(row), np.int64)
    rank[order] = np.arange(len(row)) - np.repeat(start, count)
    size = int(max(row.max(initial=0), gone.max(initial=0))) + 1
    want = np.bincount(gone, minlength=size)
    have = np.bincount(row, minlength=size)
    return np.flatnonzero(rank >= want[row]), int(np.maximum(want - have, 0).sum())


class Star:
    """Vertex 0 and its outgoing row, with the incoming rows on the other side."""

    def __init__(self, n, initial, **options):
        self.n, self.next = n, 1
        self.nb = np.sort(np.asarray(initial, np.int64))
        self.w = self.fresh(len(initial))
        off = np.full(n + 1, len(initial), np.uint64)
        off[0] = 0
        self.e = dg.Engine("sssp", weight_mode="stored", source=1, **options)
        self.e.load_csr(n, off, self.nb.astype(np.uint32), self.w.astype(np.uint32))
        self.e.start()

    def fresh(self, count):
        self.next += count
        return np.arange(self.next - count, self.next)

    def step(self, gone, new):
        w = self.fresh(len(new))
        zero = lambda x: np.zeros(len(x), np.int64)  # noqa: E731
        st = self.e.apply_batch(
            np.stack([zero(gone), gone, zero(gone)], 1).astype(np.uint32),
            np.stack([zero(new), new, w], 1).astype(np.uint32))
        stay, missing = first_ones_gone(self.nb, np.asarray(gone, np.int64))
        order = np.argsort(new, kind="stable")
        self.nb = np.concatenate([self.nb[stay], np.asarray(new, np.int64)[order]])
        self.w = np.concatenate([self.w[stay], w[order]])
        assert st["missing_deletes"] == missing
        dst, ww = self.e.row(0)
        assert np.array_equal(dst, self.nb) and np.array_equal(ww, self.w)
        for v in np.unique(np.concatenate([gone[:3], new[:3], [2]]).astype(np.int64)):
            dst, ww = self.e.row(int(v), incoming=True)
            assert (dst == 0).all() and np.array_equal(ww, self.w[self.nb == v])
        return st


@pytest.mark.parametrize("budget", [0, 8 << 20])
def test_zipf_updates_of_one_row(budget):
    n, rng = 30_000, np.random.default_rng(3)
    s = Star(n, rng.permutation(n - 2)[:20_000] + 2, hbm_graph_budget_bytes=budget, page_shift=8,
             cache_policy="hotness" if budget else "none")
    zipf = lambda k: (rng.zipf(1.1, 4 * k)[:4 * k] % (n - 2))[:k] + 2  # noqa: E731
    s.step(np.zeros(0, np.int64), zipf(150_000))
    for nd, na in ((20_000, 15_000), (3, 40_000), (40_000, 10), (1, 0), (5000, 0)):
        length = len(s.nb)
        gone = rng.choice(s.nb, nd, replace=False)     # most want fewer than there are
        gone[:nd // 100] = 2                           # and some more than there are
        st = s.step(gone, zipf(na))
        # the suffixes once in both directions (4 bytes a slot), two 128-byte lines per
        # record and direction, 16 bytes per slot of what is appended or moves
        assert st["mutate_link_bytes"] + st["mutate_hbm_bytes"] <= (
            2 * 4 * length + 2 * 256 * nd + 2 * 16 * (length + na) + 16 * na + (1 << 20))


def test_more_such_records_than_are_counted_at_a_time():
    # 150,000 neighbours twice each in the suffix, a few of them three times; one
    # occurrence of each goes, two of some: three rounds of 65,536 records
    pairs, n = 150_000, 160_000
    s = Star(n, [2, 3])
    nb = np.arange(5, 5 + pairs)
    s.step(np.zeros(0, np.int64), np.concatenate([nb, nb[::7]]))
    s.step(np.zeros(0, np.int64), nb)
    s.step(np.concatenate([nb, nb[::7], nb[::21]]), [2, 2])
    s.step(nb[::5], nb[::3])
