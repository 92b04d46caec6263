"""dycg_graph_info.device_bytes counts every device buffer the engine holds, the row and
chunk lists of a batch included, as the device's own figure of free memory shows."""
import gc

import numpy as np
import pytest
import torch

import dycgraph_b200 as dg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("queries", [0, 33])
def test_device_bytes_is_what_the_device_gave(queries):
    n, m = 4_000_000, 8_000_000
    rng = np.random.default_rng(1)
    src = np.sort(rng.integers(0, n, m))
    off = np.concatenate([[0], np.bincount(src, minlength=n).cumsum()]).astype(np.uint64)
    dst = rng.integers(0, n, m).astype(np.uint32)

    def build():
        e = dg.Engine("sssp", hbm_graph_budget_bytes=64 << 20)
        e.load_csr(n, off, dst)
        if queries:
            e.set_queries(np.arange(queries, dtype=np.uint32), "batched")
        e.start()
        e.apply_batch([], [(0, 1)])
        return e

    build().close()  # (code, and what the runtime keeps for itself)
    gc.collect()     # (engines that earlier tests left open)
    free0, _ = torch.cuda.mem_get_info()
    e = build()
    free1, _ = torch.cuda.mem_get_info()
    held = e.info()["device_bytes"]
    # the runtime hands memory out in 2 MB pieces: at most one more per buffer, of
    # some eighty, and graphs and small buffers share a few
    assert held <= free0 - free1 + (8 << 20)
    assert held >= free0 - free1 - (176 << 20)
    e.reserve_batch(4 << 20)
    free2, _ = torch.cuda.mem_get_info()
    grown = e.info()["device_bytes"] - held
    assert grown > 500 << 20  # (two directions, 16-byte records, keys twice, ...)
    assert abs(grown - (free1 - free2)) <= 64 << 20
    e.close()
