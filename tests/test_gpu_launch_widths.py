"""The automatic CTA width of learned searches and of the parts of a pipelined
batch, at the borders between the widths; the tracks do not depend on it.
"""
import os

import numpy as np
import pytest

from conftest import ROOT, index_lists

pytestmark = pytest.mark.gpu


def _blobs(oracle_lib, large):
    from cl_forward_gb300 import generator
    params = generator.CONFIG_STRESS if large else generator.CONFIG_SMALL
    return [oracle_lib.sort_by_x(b) for b in generator.generate(range(7800, 7812), params)[0]]


def _same(tracks, counts, first, which, want):
    for e, k in enumerate(which):
        assert index_lists(tracks[int(first[e]):int(first[e]) + int(counts[e])]) == want[k], f"event {e}"


# (events per SM, one event more, hits), the width that the rule gives
@pytest.mark.parametrize("per_sm,more,large,width", [(1, 0, False, 256), (3, 0, False, 256), (3, 1, False, 128),
                                                     (8, 0, False, 128), (8, 1, False, 64), (3, 1, True, 256),
                                                     (8, 1, True, 128)])
def test_learned(gpu_ctx, oracle_lib, per_sm, more, large, width):
    from cl_forward_gb300 import events, native
    blobs = _blobs(oracle_lib, large)
    z = np.load(os.path.join(ROOT, "cl_forward_gb300", "weights", "doublet_mlp.npz"))
    gpu_ctx.set_mlp(z["weights"], float(z["keep_threshold"]), float(z["window_margin"]), float(z["min_keep_rate"]))
    want = [index_lists(t) for t in gpu_ctx.search(blobs, native.default_options(learned=1, threads_per_event=64,
                                                                                 register_ctas=4))[0]]
    which = np.arange(per_sm * gpu_ctx.sm_count + more) % len(blobs)
    buf, offs, sizes = events.pack_events(blobs)
    gpu_ctx.stage(buf, offs[which].copy(), sizes[which].copy())
    gpu_ctx.run(native.default_options(learned=1))
    assert gpu_ctx.stats().block == width
    tracks, counts, first, status = gpu_ctx.fetch(len(which), sum(len(want[k]) for k in which))
    assert not np.any(status)
    _same(tracks, counts, first, which, want)


# (events of a part per SM times two, one event more, hits), the width
@pytest.mark.parametrize("half_per_sm,more,large,width", [(2, 0, False, 512), (2, 1, False, 256), (8, 0, False, 256),
                                                          (8, 1, False, 128), (20, 0, False, 128), (20, 1, False, 64),
                                                          (16, 0, True, 256), (16, 1, True, 128)])
def test_parts(gpu_ctx, oracle_lib, half_per_sm, more, large, width):
    from cl_forward_gb300 import events, native
    blobs = _blobs(oracle_lib, large)
    want, ostatus = oracle_lib.search(blobs, 4)
    assert not np.any(ostatus)
    want = [index_lists(t) for t in want]
    part = half_per_sm * gpu_ctx.sm_count // 2 + more
    which = np.arange(2 * part + 5) % len(blobs)
    buf, offs, sizes = events.pack_events(blobs)
    total = sum(len(want[k]) for k in which)
    dst = np.zeros(total, events.TRACK_DTYPE)
    counts, status, first = np.zeros(len(which), np.uint32), np.zeros(len(which), np.uint32), np.zeros(len(which), np.uint64)
    gpu_ctx.search_packed_into(buf, offs[which].copy(), sizes[which].copy(),
                               native.default_options(pipeline_events=part), dst, counts, first, status)
    stats = gpu_ctx.stats()
    assert stats.launches == 3 and stats.block == width
    assert int(counts.sum()) == total and not np.any(status)
    _same(dst, counts, first, which, want)
