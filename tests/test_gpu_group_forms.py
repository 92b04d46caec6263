"""dycg_group_updates at the edges of its forms (one CTA of several sizes, the
device-wide sort) and of its keys (vertex counts around powers of two, up to the
largest), with empty, covering and short segment lists, against numpy."""
import numpy as np
import pytest

import dycgraph_b200 as dg
from tests.test_gpu_group import group_ref, run_group

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [1, 2, 255, 256, 257, 1 << 20, (1 << 31) - 1, (1 << 32) - 1])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1024, 1025, 4096, 4097, 8192, 8193, 20_000])
def test_forms(n, nv):
    rng = np.random.default_rng(n * 7 + nv % 1000)
    top = min(nv + 3, (1 << 32) - 1)
    rec = rng.integers(max(0, top - 40), top + 1, size=(n, 3)).astype(np.uint32)
    rec[rng.random(n) < 0.5] //= np.uint32(3)
    rec[n // 2:n // 2 + n // 8] = rec[0]
    ends = np.unique(rng.integers(0, nv + 1, 5)).astype(np.uint32)  # ascending, short of nv
    for fn in (dg.lib().dycg_group_updates, dg.lib().dycg_group_updates_noalloc):
        rc, keys, mult, bad, seg = run_group(fn, rec, nv, ends)
        assert rc == 0
        uk, cnt, rbad, rseg = group_ref(rec, nv, ends)
        assert (keys == uk).all() and (mult == cnt).all()
        assert bad == rbad and (seg == rseg).all()
