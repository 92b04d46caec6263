"""PageRank one round per call, across the line between dense rounds (a scan finds the
next frontier) and sparse ones (pushes append to it), and the frontier that a launch
leaves behind when max_rounds ends it: the next round consumes exactly the vertices
whose residual is above epsilon, x takes that residual in one FP32 addition, and the
residuals keep x + r = 0.15 + 0.85 P^T x."""
import numpy as np
import pytest

import dycgraph_b200 as dg
from tests import cases

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -24  # one FP32 rounding, relative


def residual_gap(e, rounds):
    """How far r is from 0.15 + 0.85 P^T x - x, in multiples of what FP32 may lose: in
    every round a vertex's residual takes at most one addition per in-edge, of a term
    with two roundings, and x takes one, none of a sum above 1 + x + 0.85 P^T x."""
    off, dst, _ = e.csr()
    n = len(off) - 1
    deg = np.diff(off.astype(np.int64))
    src = np.repeat(np.arange(n), deg)
    x, r = (a.astype(np.float64) for a in e.gather_ranks())
    pulled = 0.85 * np.bincount(dst, weights=x[src] / deg[src], minlength=n)
    indeg = np.bincount(dst, minlength=n)
    allowed = rounds * (indeg + 3) * ULP * (1 + np.abs(x) + pulled)
    return np.max(np.abs(0.15 + pulled - x - r) / allowed)


def next_round(e, eps):
    """One empty call: the frontier rule, exactly. Returns the vertices consumed."""
    x, r = e.gather_ranks()
    st = e.apply_batch([], [])
    x2, _ = e.gather_ranks()
    due = np.abs(r) > np.float32(eps)
    assert np.array_equal(x2, np.where(due, x + r, x))
    assert st["waves"] == (1 if due.any() else 0) or not due.any()
    return int(due.sum())


@pytest.mark.parametrize("scale,budget", [(11, 0), (13, 1 << 20)])
def test_rounds_of_a_solve_one_call_each(scale, budget):
    n, off, dst, _ = cases.small_rmat(scale, 8, 4)
    eps = 1e-4
    e = dg.Engine("pr", epsilon=eps, max_rounds=1, page_shift=8, hbm_graph_budget_bytes=budget)
    e.load_csr(n, off, dst)
    e.start()  # (the first round: every vertex)
    dense = sparse = 0
    for rounds in range(2, 200):
        due = next_round(e, eps)
        assert residual_gap(e, rounds) <= 1
        dense += due * 16 >= n
        sparse += 0 < due * 16 < n
        if not due:
            break
    assert dense >= 3 and sparse >= 3 and not due
    assert np.max(np.abs(e.gather_ranks()[1])) <= np.float32(eps)


@pytest.mark.parametrize("frontier", [98, 99, 100, 101, 102])
def test_frontiers_around_the_dense_line(frontier):
    # vertex 0 gets as many new neighbours as makes a frontier of the wanted size out of
    # n = 1600; each of them points at two of the others
    n, eps = 1600, 1e-4
    src = np.concatenate([[0], np.repeat(np.arange(1, n), 2)])
    dst = np.concatenate([[1], (np.repeat(np.arange(1, n), 2) * 7 + np.tile([3, 11], n - 1)) % n])
    order = np.lexsort((dst, src))
    off = np.concatenate([[0], np.bincount(src, minlength=n).cumsum()]).astype(np.uint64)
    e = dg.Engine("pr", epsilon=eps, max_rounds=1)
    e.load_csr(n, off, dst[order].astype(np.uint32))
    e.start()
    rounds = 1
    while next_round(e, eps):
        rounds += 1
        assert rounds < 200
    x, r = (a.astype(np.float64) for a in e.gather_ranks())
    k = frontier - 1  # (the old neighbour's residual moves, too)
    new = np.arange(2, 2 + k)
    # what the amend adds: alpha x (1 / (k + 1) - 1) to the old one, alpha x / (k + 1) to
    # the new ones, which is far above epsilon and what is left of earlier rounds
    moved = r.copy()
    moved[1] += 0.85 * x[0] * (1 / (k + 1) - 1)
    moved[new] += 0.85 * x[0] / (k + 1)
    due = np.abs(moved) > eps
    changed = np.append(new, 1)
    assert due.sum() == frontier and np.abs(np.abs(moved[changed]) - eps).min() > 1e-6
    st = e.apply_batch([], [(0, int(v)) for v in new])
    assert st["waves"] == 1
    x2, _ = (a.astype(np.float64) for a in e.gather_ranks())
    # four roundings of terms below x[0], and one of the sum
    tol = 8 * ULP * (x[0] + np.abs(x) + 1)
    assert (np.abs(x2 - np.where(due, x + moved, x)) <= tol).all()
    for _ in range(200):
        rounds += 1
        left = next_round(e, eps)
        assert residual_gap(e, rounds + 1) <= 1
        if not left:
            break
    assert not left
