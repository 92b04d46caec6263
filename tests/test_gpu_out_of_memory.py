"""Device memory that runs out inside a call, made by holding nearly all of it in
another allocation: the call returns its error, and what follows is either refused
(the snapshot was under way) or right (it was not)."""
import gc

import numpy as np
import pytest
import torch

import dycgraph_b200 as dg
import oracle
from tests import cases

pytestmark = pytest.mark.gpu
ENOMEM, ESTATE = -3, -4
LEFT = 64 << 20


class Held:
    """All device memory but LEFT bytes."""

    def __enter__(self):
        gc.collect()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.block = torch.empty(free - LEFT, dtype=torch.uint8, device="cuda")

    def __exit__(self, *_):
        del self.block
        torch.cuda.empty_cache()


def graph():
    return cases.small_rmat(16, 4, 5)


def test_snapshot_that_runs_out_of_memory_under_way_fails_the_engine():
    n, off, dst, w = graph()
    e = dg.Engine("sssp", weight_mode="stored")
    e.load_csr(n, off, dst, w)
    e.set_queries(np.arange(256, dtype=np.uint32), "batched")  # 128 MB of keys to save
    e.start()
    d, a = cases.random_batch(n, off, dst, w, 300, 300, 1)
    e.apply_batch(d, a)
    with Held():
        # the graph is mutated when the tuner finds no room for the saved state
        with pytest.raises(dg.DycgError) as err:
            e.tune_query_mapping(a, d)
        assert err.value.code == ENOMEM
    for call in (lambda: e.apply_batch(a, d), lambda: e.apply_batches([(a, d)])):
        with pytest.raises(dg.DycgError) as err:
            call()
        assert err.value.code == ESTATE
    e.close()
    # another engine on the same context is not touched by any of it
    e = dg.Engine("sssp", weight_mode="stored")
    e.load_csr(n, off, dst, w)
    e.start()
    orc = oracle.Oracle(oracle.SSSP, n, off, dst, w, weight_mode=oracle.WEIGHT_STORED)
    orc.init()
    e.apply_batch(d, a)
    orc.apply_batch(d, a)
    assert np.array_equal(e.gather()[0], orc.values()[0])


def test_batch_buffers_that_do_not_fit_leave_the_engine_usable():
    n, off, dst, w = graph()
    e = dg.Engine("sssp", weight_mode="stored")
    e.load_csr(n, off, dst, w)
    e.start()
    orc = oracle.Oracle(oracle.SSSP, n, off, dst, w, weight_mode=oracle.WEIGHT_STORED)
    orc.init()
    for step in range(3):
        o, dd, ww = orc.csr()
        d, a = cases.random_batch(n, o, dd, ww, 300, 300, step)
        e.apply_batch(d, a)
        orc.apply_batch(d, a)
        assert np.array_equal(e.gather()[0], orc.values()[0]), step
        with Held():
            # (the first list alone, 16 bytes a record, is twice what is left)
            with pytest.raises(dg.DycgError) as err:
                e.reserve_batch(8 << 20)
            assert err.value.code == ENOMEM
    e.reserve_batch(2000)
    d, a = cases.random_batch(n, *orc.csr(), 2000, 2000, 9)
    e.apply_batch(d, a)
    orc.apply_batch(d, a)
    assert np.array_equal(e.gather()[0], orc.values()[0])
