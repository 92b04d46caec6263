"""dycg_group_updates with few and many segments for its records: counted from the
segments' side or from the records', at the line between the two, against numpy; and
what a small batch pays for a long list of segments."""
import numpy as np
import pytest
import torch

import dycgraph_b200 as dg
from tests.test_gpu_group import group_ref, run_group

pytestmark = pytest.mark.gpu


def capacity(n):
    """Records that the form which serves n of them is made for."""
    return next((c for c in (256, 1024, 4096, 8192) if n <= c), n)


@pytest.mark.parametrize("n", [1, 256, 257, 4096, 4097, 8192, 8193, 30_000])
@pytest.mark.parametrize("kind", ["below", "at", "above", "many"])
@pytest.mark.parametrize("nv", [70_000, (1 << 32) - 1])
def test_segment_counts(n, kind, nv):
    c = capacity(n)
    nseg = {"below": 2 * c - 1, "at": 2 * c + 1, "above": 2 * c + 2, "many": 300_000}[kind]
    rng = np.random.default_rng(n + nseg)
    rec = rng.integers(0, nv, size=(n, 3), dtype=np.uint64)
    rec[rng.random(n) < 0.5] //= 1000           # several runs in a segment
    rec[n // 2:n // 2 + n // 8] = rec[0]        # and repeated records
    rec[rng.random(n) < 0.02, 1] = min(nv + 5, (1 << 32) - 1)
    ends = np.sort(rng.integers(0, nv, nseg, dtype=np.uint64))  # empty segments, short of nv
    ends[nseg // 3:nseg // 3 + 5] = ends[nseg // 3]             # and equal ends
    rec, ends = rec.astype(np.uint32), ends.astype(np.uint32)
    for fn in (dg.lib().dycg_group_updates, dg.lib().dycg_group_updates_noalloc):
        rc, keys, mult, bad, seg = run_group(fn, rec, nv, ends)
        assert rc == 0
        uk, cnt, rbad, rseg = group_ref(rec, nv, ends)
        assert (keys == uk).all() and (mult == cnt).all()
        assert bad == rbad and (seg == rseg).all()


@pytest.mark.parametrize("n", [10, 300, 8192])
def test_many_segments_cost_a_small_batch_little(n):
    nv, out = 1 << 24, {}
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    rec = torch.randint(0, nv, (n, 3), device="cuda", generator=g, dtype=torch.int32)
    uv, mult = (torch.empty(k * n, dtype=torch.int32, device="cuda") for k in (2, 1))
    counts = torch.empty(2, dtype=torch.int32, device="cuda")
    for nseg in (1, 1 << 20):
        ends = torch.arange(1, nseg + 1, dtype=torch.int32, device="cuda") * (nv // nseg)
        seg = torch.empty(nseg, dtype=torch.int32, device="cuda")
        best = float("inf")
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(10):
                rc = dg.lib().dycg_group_updates(
                    rec.data_ptr(), n, nv, ends.data_ptr(), nseg, uv.data_ptr(), mult.data_ptr(),
                    seg.data_ptr(), counts.data_ptr(), torch.cuda.current_stream().cuda_stream)
                assert rc == 0
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        out[nseg] = best
    # (4 MB of counts are cleared; from the segments' side it was 50 to 500 times)
    assert out[1 << 20] < 10 * out[1], out
