"""The learned policy on an engine whose HBM budget holds no page: features and
history are kept, nothing can be admitted, and every form of a snapshot call goes
through with the oracle's results."""
import ctypes

import numpy as np
import pytest

import dycgraph_b200 as dg
import oracle
from dycgraph_b200 import engine as eng
from tests import cases

pytestmark = pytest.mark.gpu


def apply(e, d, a, stats):
    d, a = eng.edges_array(d), eng.edges_array(a)
    p = ctypes.POINTER(eng.Edge)
    rc = dg.lib().dycg_apply_batch(e._h, d.ctypes.data_as(p), len(d), a.ctypes.data_as(p), len(a),
                                   ctypes.byref(stats) if stats is not None else None)
    assert rc == 0


@pytest.mark.parametrize("budget", [0, 1])
@pytest.mark.parametrize("stats", [True, False])
def test_learned_policy_without_cache_slots(stats, budget):
    n, off, dst, w = cases.small_rmat(11, 8, 3)
    e = dg.Engine("sssp", weight_mode="stored", page_shift=8, hbm_graph_budget_bytes=budget,
                  cache_policy="learned")
    e.load_csr(n, off, dst, w)
    e.start()
    assert e.info()["cache_slots"] == 0
    orc = oracle.Oracle(oracle.SSSP, n, off, dst, w, weight_mode=oracle.WEIGHT_STORED)
    orc.init()
    for step in range(4):
        o, dd, ww = orc.csr()
        d, a = cases.random_batch(n, o, dd, ww, 200, 200, step)
        st = eng.BatchStats() if stats else None
        apply(e, d, a, st)
        orc.apply_batch(d, a)
        assert np.array_equal(e.gather()[0], orc.values()[0]), step
        if stats:
            assert st.cache_pages_loaded == 0 and st.cache_pages_evicted == 0
    # the halves of a snapshot as calls of their own, then the maintenance
    d, a = cases.random_batch(n, *orc.csr(), 50, 50, 9)
    e.delete_edges(d)
    e.insert_edges(a)
    e.cache_maintenance()
    orc.apply_batch(d, a)
    assert np.array_equal(e.gather()[0], orc.values()[0])
