"""The repair's phase times: every phase that a snapshot has is timed, one that it has
not is zero, and together they fit into the repair's own time."""
import numpy as np
import pytest

import dycgraph_b200 as dg
from tests import cases

pytestmark = pytest.mark.gpu
PHASES = ["ms_phase_invalidate", "ms_phase_seed", "ms_phase_pull", "ms_phase_closure"]


@pytest.mark.parametrize("form", ["single", "batched", "replayed"])
def test_every_phase_of_a_snapshot_is_timed(form):
    n, off, dst, w = cases.small_rmat(14, 8, 2)
    e = dg.Engine("sssp", weight_mode="stored")
    e.load_csr(n, off, dst, w)
    if form != "single":
        e.set_queries(np.arange(40, dtype=np.uint32), "batched")
    e.start()
    d, a = cases.random_batch(n, off, dst, w, 20_000, 20_000, 3)

    def times(dels, adds):
        st = e.apply_batches([(dels, adds)])[0] if form == "replayed" else e.apply_batch(dels, adds)
        t = {k: st[k] for k in PHASES}
        # (the repair's time is taken by events around the launch, or by the same timer)
        assert 0 < sum(t.values()) <= st["ms_repair"] + 0.002, (t, st["ms_repair"])
        return t

    t = times(d[:10_000], a[:10_000])
    assert all(t[k] > 0 for k in PHASES), t
    if form != "replayed":  # (a replayed graph has all phases, whatever its batch)
        t = times(d[10_000:], [])
        assert t["ms_phase_seed"] == 0 and t["ms_phase_pull"] > 0, t
        t = times([], a[10_000:])
        assert t["ms_phase_invalidate"] == 0 and t["ms_phase_seed"] > 0, t
