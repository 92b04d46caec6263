"""Rows whose block is full: compacted in place, moved, or refused, in slot order.
The model is the occurrence semantics on one hub row with distinct neighbours: a
deletion takes the neighbour out, insertions follow in ascending order. relocated_rows
and arena_used tell which way a row went."""
import numpy as np
import pytest

import dycgraph_b200 as dg

pytestmark = pytest.mark.gpu
HUB = 0


class Hub:
    """An engine with one long row (outgoing or incoming) of `degree` distinct
    neighbours 1.. and a model of it."""

    def __init__(self, degree, n, incoming, stored, **options):
        self.n, self.incoming = n, incoming
        self.row = np.arange(1, degree + 1, dtype=np.int64)
        if incoming:
            off = np.minimum(np.maximum(np.arange(n + 1) - 1, 0), degree).astype(np.uint64)
            dst = np.full(degree, HUB, np.uint32)
        else:
            off = np.full(n + 1, degree, np.uint64)
            off[0] = 0
            dst = self.row.astype(np.uint32)
        self.e = dg.Engine("sssp", weight_mode="stored" if stored else "hash128", **options)
        self.stored = stored
        self.e.load_csr(n, off, dst, self.weight(self.row) if stored else None)
        self.e.start()

    @staticmethod
    def weight(nb):
        return (np.asarray(nb) % 60 + 1).astype(np.uint32)

    def records(self, nb):
        nb = np.asarray(nb, np.int64)
        u, v = (nb, np.full(len(nb), HUB)) if self.incoming else (np.full(len(nb), HUB), nb)
        return np.stack([u, v, self.weight(nb)], 1).astype(np.uint32)

    def apply(self, gone, new):
        st = self.e.apply_batch(self.records(gone), self.records(new))
        assert st["missing_deletes"] == 0
        self.row = np.concatenate([self.row[~np.isin(self.row, gone)], np.sort(new)])
        return st

    def check(self):
        dst, w = self.e.row(HUB, incoming=self.incoming)
        assert np.array_equal(dst, self.row)
        if self.stored:
            assert np.array_equal(w, self.weight(self.row))
        assert self.e.info()["live_edges"] == len(self.row)


def capacity(degree):
    """Slots of the block that the loader gives a row."""
    return 1 << int(degree + degree // 16).bit_length()


@pytest.mark.parametrize("incoming,stored", [(False, True), (True, False)])
def test_hub_larger_than_the_headroom(incoming, stored):
    # the row's own block is as large as the whole headroom (2^20 slots): asking for
    # the next larger one would overrun the arena, and is never needed
    degree, n, step = 800_000, 900_000, 50_000
    h = Hub(degree, n, incoming, stored)
    assert capacity(degree) == 1 << 20
    rng = np.random.default_rng(4)
    spare = np.arange(degree + 1, degree + 1 + step)
    for _ in range(14):  # some 2.8 blocks' worth of appended slots
        gone = rng.choice(h.row, step, replace=False)
        assert h.apply(gone, spare)["insertions"] == step
        spare = gone
    h.check()


def test_rows_past_half_of_the_headroom_stay_when_they_fit():
    # 60,000 rows alike, so one row is the model of all of them. Their first growth, to
    # blocks of 16, takes 960,000 of the 2^20 spare slots; from then on a full row whose
    # live occurrences and a reserve fit stays, more than half full or not
    rows, n = 60_000, 60_040
    row = list(range(rows, rows + 7))
    off = np.minimum(np.arange(n + 1), rows).astype(np.uint64) * 7
    e = dg.Engine("pr", epsilon=1.0)  # (no incoming rows, nothing to repair)
    e.load_csr(n, off, np.tile(np.array(row, np.uint32), rows))
    e.start()
    first = e.info()

    def records(targets):
        u = np.repeat(np.arange(rows), len(targets))
        return np.stack([u, np.tile(targets, rows), np.ones(len(u))], 1).astype(np.uint32)

    def step(gone, new):
        st = e.apply_batch(records(gone), records(new))
        assert st["missing_deletes"] == 0
        for v in gone:
            row.remove(v)
        row.extend(sorted(new))
        o, dst, _ = e.csr()
        assert (np.diff(o.astype(np.int64))[:rows] == len(row)).all()
        assert (dst.reshape(rows, -1) == np.array(row, np.uint32)).all()
        return st["relocated_rows"], e.info()["arena_used"] - first["arena_used"]

    assert step([], [rows + 30, rows + 9]) == (rows, 16 * rows)
    gone = row[1:8:2]
    assert step(gone, [rows + 20 + i for i in range(6)]) == (0, 16 * rows)  # 9 + 6 slots
    for _ in range(6):  # 11 of 16 slots live, three deleted and three inserted each time
        moved = step(row[::3][:3], [v for v in range(rows, rows + 40) if v not in row][:3])
        assert moved == (0, 16 * rows)
