"""Deletions in a row whose unsorted suffix is longer than what the matching keeps in
HBM between its two passes (16384 chunks of 256 slots): records on both sides of that
line, in the prefix, repeated ones that want fewer occurrences than there are, and
missing ones. The model is the occurrence semantics: the first live occurrences in
slot order go."""
import numpy as np
import pytest

import dycgraph_b200 as dg

pytestmark = pytest.mark.gpu
KEPT = 16384 * 256


def test_suffix_longer_than_the_kept_part():
    degree, extra = 4_000_000, 4_300_000
    n = degree + extra + 1000
    off = np.full(n + 1, degree, np.uint64)
    off[0] = 0
    e = dg.Engine("pr", epsilon=1.0)  # (no incoming rows, nothing to repair)
    e.load_csr(n, off, np.arange(1, degree + 1, dtype=np.uint32))
    e.start()
    new = np.arange(degree + 1, degree + 1 + extra, dtype=np.int64)
    new[10:13] = new[10]  # three occurrences each, early and late
    new[-20:-17] = new[-20]
    record = lambda v: np.stack([np.zeros(len(v)), v, np.ones(len(v))], 1).astype(np.uint32)  # noqa: E731
    st = e.apply_batch([], record(new))
    assert st["relocated_rows"] == 0 and extra > KEPT
    row = np.concatenate([np.arange(1, degree + 1), new])
    rng = np.random.default_rng(0)
    for early, late in ((2, 1), (2, 2), (1, 3)):  # of the repeated ones
        live = {k: np.count_nonzero(row == k) for k in (new[10], new[-20])}
        gone = [rng.choice(row[:degree // 2], 5, replace=False),
                rng.choice(row[degree:degree + KEPT // 2], 7, replace=False),
                rng.choice(row[degree + KEPT + 1000:-100], 9, replace=False),
                np.full(early, new[10]), np.full(late, new[-20]), [n - 1, n - 2, n - 2]]
        gone = np.unique(np.concatenate(gone[:3])).tolist() + np.concatenate(gone[3:]).tolist()
        gone = [int(v) for v in gone]
        missing = 3 + max(0, early - live[new[10]]) + max(0, late - live[new[-20]])
        st = e.apply_batch(record(rng.permutation(gone)), [])
        for v in gone:
            at = np.flatnonzero(row == v)
            if len(at):
                row = np.delete(row, at[0])
        assert st["missing_deletes"] == missing
        dst, _ = e.row(0)
        assert np.array_equal(dst, row)
