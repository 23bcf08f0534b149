"""velo_search_device_static at the borders between its CTA widths (1, 3 and 8
events per SM) and at its largest batch: the oracle's tracks for every event.
"""
import numpy as np
import pytest

from conftest import index_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm,more", [(1, 0), (1, 1), (3, 0), (3, 1), (8, 0), (8, 1), (0, 4096)])
def test_widths(gpu_ctx, oracle_lib, per_sm, more):
    from cl_forward_gb300 import generator, native
    from test_zz_no_alloc import _call_static, _hits, _lists
    n = per_sm * gpu_ctx.sm_count + more
    params = generator.GenParams(pv_mean=1.0, tracks_per_pv=3.0 if n > 1000 else 20.0)
    blobs = [oracle_lib.sort_by_x(b) for b in generator.generate(range(9300, 9400), params)[0]]
    few = [b for b in blobs if _hits(b) <= (50 if n > 1000 else 400)]
    want = [index_lists(t) for t in oracle_lib.search(few, 4)[0]]
    assert sum(len(t) for t in want) > 0
    st, got, status = _call_static(native.load(), [few[k % len(few)] for k in range(n)])
    assert st == native.OK and not np.any(status)
    for e in range(n):
        assert _lists(got[e]) == want[e % len(few)], f"event {e}"
