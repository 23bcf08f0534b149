"""Where the automatic launch of a batch of at most one event per SM keeps its
events: in shared memory up to 4,000 hits with the default tile (smem_hits =
50), and up to the caller's own tile with any other or with a register build of
the caller's choice.  Every event gives the oracle's tracks on either side.
"""
import numpy as np
import pytest

from conftest import index_lists

pytestmark = pytest.mark.gpu

TILE = 4000   # hits


def _blobs(oracle_lib):
    """Events of every size, a few hits to well above the tile, and at most one per SM."""
    from cl_forward_gb300 import generator
    small = generator.GenParams(pv_mean=0.5)
    blobs = generator.generate(range(8800, 8812), small)[0] + generator.generate(range(8820, 8832))[0]
    blobs += generator.generate(range(8840, 8858), generator.CONFIG_STRESS)[0]
    return [oracle_lib.sort_by_x(b) for b in blobs]


@pytest.mark.parametrize("options, threads, tile", [
    (dict(), 512, TILE), (dict(smem_hits=50), 512, TILE), (dict(smem_hits=49), 512, 49), (dict(smem_hits=51), 512, 51),
    (dict(smem_hits=1300), 512, 1300), (dict(register_ctas=4), 64, 50), (dict(ctas_per_sm=1), 64, 50),
    (dict(threads_per_event=512, register_ctas=5), 512, 50)])
def test_tile(gpu_ctx, oracle_lib, options, threads, tile):
    from cl_forward_gb300 import native
    blobs = _blobs(oracle_lib)
    hits = np.array([int(np.frombuffer(b[4:8], "<i4")[0]) for b in blobs])
    assert len(blobs) <= gpu_ctx.sm_count and np.sum(hits > TILE) >= 3 and np.sum((hits > 3000) & (hits <= TILE)) >= 3
    got, status = gpu_ctx.search(blobs, native.default_options(**options))
    want, ostatus = oracle_lib.search(blobs, 4)
    stats = gpu_ctx.stats()
    assert stats.block == threads
    assert stats.events_in_global == np.sum(hits > tile)
    for e in range(len(blobs)):
        if not ostatus[e] & oracle_lib.PARITY_EXCLUDING:
            assert status[e] == ostatus[e] and index_lists(got[e]) == index_lists(want[e]), f"event {e}"
    assert np.sum(np.asarray(ostatus) & oracle_lib.PARITY_EXCLUDING == 0) > len(blobs) // 2
