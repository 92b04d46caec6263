"""Rows of every length class that fill their block and are copied, in their own
block or to a new one: by a warp, by a CTA, by the whole grid in one or several
steps. Outgoing and incoming rows, one and two words per slot, with and without
resident pages. The model is the occurrence semantics on one hub row with distinct
neighbours (a deletion takes the neighbour out, insertions follow in ascending
order); relocated_rows and arena_used tell which way the row went."""
import numpy as np
import pytest

import dycgraph_b200 as dg

pytestmark = pytest.mark.gpu
ROOT, HUB, FIRST = 0, 1, 2  # the hub's row starts two slots into its arena


def weight(nb):
    return (np.asarray(nb) % 60 + 1).astype(np.uint32)


class Hub:
    def __init__(self, degree, incoming, stored, **options):
        self.n, self.incoming, self.stored = degree + FIRST, incoming, stored
        self.row = np.arange(FIRST, self.n, dtype=np.int64)
        u, v = np.full(degree, HUB), self.row
        if incoming:
            u, v = v, u
        # an edge from the root to the hub, or back: two slots ahead of the hub's row
        u, v = np.append(u, HUB if incoming else ROOT), np.append(v, ROOT if incoming else HUB)
        order = np.lexsort((v, u))
        u, v = u[order], v[order]
        off = np.concatenate([[0], np.bincount(u, minlength=self.n).cumsum()]).astype(np.uint64)
        self.e = dg.Engine("sssp", weight_mode="stored" if stored else "hash128", source=ROOT,
                           **options)
        self.e.load_csr(self.n, off, v.astype(np.uint32),
                        weight(np.maximum(u, v)) if stored else None)
        self.e.start()

    def records(self, nb):
        nb = np.asarray(nb, np.int64)
        u, v = np.full(len(nb), HUB), nb
        if self.incoming:
            u, v = v, u
        return np.stack([u, v, weight(nb)], 1).astype(np.uint32)

    def apply(self, gone, new):
        st = self.e.apply_batch(self.records(gone), self.records(new))
        assert st["missing_deletes"] == 0
        self.row = np.concatenate([self.row[~np.isin(self.row, gone)], np.sort(np.asarray(new, np.int64))])
        return st

    def check(self):
        dst, w = self.e.row(HUB, incoming=self.incoming)
        assert np.array_equal(dst, self.row)
        if self.stored:
            assert np.array_equal(w, weight(self.row))
        assert self.e.info()["live_edges"] == len(self.row) + 1
        if self.incoming:
            return
        # the hub's vertex invalidated and expanded again: the repair reads the row
        # where its pages are, in HBM or on the host
        self.e.apply_batch([(ROOT, HUB, 7)], [(ROOT, HUB, 7)])
        want = np.full(self.n, 0xFFFFFFFF, np.int64)
        at = 7 if self.stored else (ROOT + HUB) % 128 + 1
        want[ROOT], want[HUB] = 0, at
        step = weight(self.row) if self.stored else (HUB + self.row) % 128 + 1
        want[self.row] = at + step
        assert np.array_equal(self.e.gather()[0], want)


def filled(degree, short, rng, **options):
    """A hub whose row uses all but `short` slots of its block, with as many live
    ones as it was loaded with."""
    h = Hub(degree, **options)
    cap = 1 << int(degree + degree // 16).bit_length()
    back = rng.choice(h.row, cap - degree - short, replace=False)
    h.apply(back, [])
    assert h.apply([], back)["relocated_rows"] == 0
    return h, cap


FORMS = [dict(incoming=False, stored=True), dict(incoming=True, stored=False),
         dict(incoming=False, stored=False, hbm_graph_budget_bytes=64 << 20, page_shift=8),
         dict(incoming=True, stored=True, hbm_graph_budget_bytes=64 << 20, page_shift=8)]
# (blocks of 2^10 .. 2^21 slots; the last takes two steps of the grid)
DEGREES = [700, 1500, 3000, 12_000, 20_000, 100_000, 200_000, 1_300_000]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("degree", DEGREES)
@pytest.mark.parametrize("short", [0, 2])
def test_half_dead_row_is_compacted_in_its_block(degree, short, form):
    if degree > 1_000_000 and short:
        pytest.skip("one size of the longest is enough")
    rng = np.random.default_rng(degree + short)
    h, cap = filled(degree, short, rng, **form)
    gone = rng.choice(h.row, degree * 6 // 10, replace=False)
    h.apply(gone, [])
    used = h.e.info()["arena_used"]
    st = h.apply([], gone[:short + 1])  # one more than the block holds
    assert st["relocated_rows"] == 0 and h.e.info()["arena_used"] == used
    h.check()
    # its order, its index and its room are as they should be: deletions find
    # everything, and what is left of the block fills without a move
    again = rng.choice(h.row, len(h.row) // 3, replace=False)
    h.apply(again, [])
    h.check()
    st = h.apply([], gone[short + 1:short + 1 + cap // 8])
    assert st["relocated_rows"] == 0
    h.check()


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("degree", DEGREES[:-1])
def test_live_row_moves_without_its_deleted_slots(degree, form):
    rng = np.random.default_rng(degree)
    h, cap = filled(degree, 2, rng, arena_headroom_permille=8000, **form)
    gone = rng.choice(h.row, degree // 10, replace=False)
    h.apply(gone, [])
    used = h.e.info()["arena_used"]
    st = h.apply([], gone[:3])
    assert st["relocated_rows"] == 1
    assert h.e.info()["arena_used"] == used + 2 * cap
    h.check()
    h.apply(rng.choice(h.row, len(h.row) // 3, replace=False), gone[3:])
    h.check()


@pytest.mark.parametrize("half_dead", [True, False])
def test_a_long_row_is_copied_at_a_fair_part_of_the_link_rate(half_dead):
    # 2^20 slots in over the host link and at most as many out, for three records: the
    # time that the bytes take one after the other, times eight for a small launch
    _, read_gbs = dg.measure_host_link(0, 256 << 20)
    bound = 8 * 2 * 4 * (1 << 20) / (read_gbs * 1e6)
    ms = []
    for seed in range(3):
        rng = np.random.default_rng(seed)
        h, _ = filled(900_000, 2, rng, incoming=False, stored=False, arena_headroom_permille=8000)
        gone = rng.choice(h.row, 540_000 if half_dead else 1000, replace=False)
        h.apply(gone, [])
        st = h.apply([], gone[:3])
        assert st["relocated_rows"] == (0 if half_dead else 1)
        ms.append(st["ms_mutate"])
        h.e.close()
    assert min(ms) < bound, (ms, bound)
