"""Unsorted events, whose seeding walks the candidate windows a few hits at a
time, and h1 windows over several z per module, at module sizes around that
number of hits: equality with the oracle.
"""
import numpy as np
import pytest

from conftest import index_lists

pytestmark = pytest.mark.gpu


def _unsorted(blob, seed):
    """The event with the hits of each module in another order."""
    from cl_forward_gb300.events import Event, pack_event, unpack_event
    e = unpack_event(blob)
    rng = np.random.Generator(np.random.PCG64(seed))
    at = np.concatenate([s + rng.permutation(n) for s, n in zip(e.hit_start, e.hit_num)]).astype(int)
    return pack_event(Event(e.sensor_z, e.hit_start, e.hit_num, e.hit_id[at], e.x[at], e.y[at], e.z[at]))


@pytest.mark.parametrize("threads", [32, 64, 512])
@pytest.mark.parametrize("z_style", ["one", "many"])
@pytest.mark.parametrize("per_module", [1, 3, 4, 5, 8, 9, 40])
def test_module_sizes(gpu_ctx, oracle_lib, per_module, z_style, threads):
    from cl_forward_gb300 import native
    from test_gpu_pair_seeding import _event
    blobs = [_event(300 * per_module + k, per_module, z_style, n_modules=18) for k in range(8)]
    blobs += [_unsorted(b, k) for k, b in enumerate(blobs)]
    for y in (1, 3, 4):
        got, status = gpu_ctx.search(blobs, native.default_options(y_lanes=y, threads_per_event=threads))
        want, ostatus = oracle_lib.search(blobs, y)
        tracks = 0
        for e in range(len(blobs)):
            assert not ostatus[e] & oracle_lib.PARITY_EXCLUDING
            assert status[e] == ostatus[e] and index_lists(got[e]) == index_lists(want[e]), f"event {e}, Y={y}"
            tracks += len(got[e]) if e >= 8 else 0
        assert tracks > 0   # unsorted events have tracks too
