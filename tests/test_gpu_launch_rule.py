"""The automatic CTA width of a batch, at the borders between the widths, and
the mixed work order of batches read in place: every event is searched once
and gives the oracle's tracks.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _blobs(oracle_lib, large):
    from cl_forward_gb300 import generator
    params = generator.CONFIG_STRESS if large else generator.CONFIG_SMALL
    return [oracle_lib.sort_by_x(b) for b in generator.generate(range(7700, 7712), params)[0]]


def _records(tracks):
    """An event's whole 100-byte track records (zeros past the hits), in order."""
    return np.sort(np.ascontiguousarray(tracks).view("S100"))


# (events per SM, one event more, hits), the width that the rule gives
BORDERS = [(1, 0, False, 512), (1, 1, False, 256), (8, 0, False, 256), (8, 1, False, 128), (20, 0, False, 128),
           (20, 1, False, 64), (20, 1, True, 128), (36, 1, True, 64)]


@pytest.mark.parametrize("host_direct", [0, 1])
@pytest.mark.parametrize("per_sm,more,large,width", BORDERS)
def test_width_by_batch_size(gpu_ctx, oracle_lib, per_sm, more, large, width, host_direct):
    from cl_forward_gb300 import events, native
    blobs = _blobs(oracle_lib, large)
    n = per_sm * gpu_ctx.sm_count + more
    want, ostatus = oracle_lib.search(blobs, 4)
    assert not np.any(ostatus)
    records = [_records(t) for t in want]
    buf, offs, sizes = events.pack_events(blobs)
    which = np.arange(n) % len(blobs)            # events may share their bytes
    total = sum(len(want[k]) for k in which)
    src = gpu_ctx.host_alloc(len(buf))
    src[:] = buf
    dst = gpu_ctx.host_alloc(total * 100).view(events.TRACK_DTYPE)
    counts, status = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    first = np.zeros(n, np.uint64)
    try:
        gpu_ctx.search_packed_into(src, offs[which].copy(), sizes[which].copy(),
                                   native.default_options(host_direct=host_direct), dst, counts, first, status)
        assert gpu_ctx.stats().block == width
        assert int(counts.sum()) == total and not np.any(status)
        for e in range(n):
            got = dst[int(first[e]):int(first[e]) + int(counts[e])]
            assert np.array_equal(_records(got), records[which[e]]), f"event {e}"
    finally:
        gpu_ctx.host_free(src)
        gpu_ctx.host_free(dst.view(np.uint8))
