"""Learned seeding's three outcomes of the keep-rate guard, each shown to occur:
the doublets in reach of a hit settle it, they do not but all doublets scored
do, and the event goes back to the plain method.
"""
import os

import numpy as np
import pytest

from conftest import ROOT, index_lists

pytestmark = pytest.mark.gpu


def _blobs():
    from cl_forward_gb300 import generator, native
    return [native.sort_by_x(b) for b in generator.generate(range(100400, 100448))[0]]


def _weights():
    return np.load(os.path.join(ROOT, "cl_forward_gb300", "weights", "doublet_mlp.npz"))


def _search(ctx, blobs, min_window, threads):
    """learned_min_window = 0 scores the doublets in reach first, 1 all of them at once."""
    from cl_forward_gb300 import native
    got, status = ctx.search(blobs, native.default_options(learned=1, learned_min_window=min_window,
                                                           threads_per_event=threads, register_ctas=4))
    return [index_lists(g) for g in got], (np.asarray(status) & native.EVENT_LEARNED_FALLBACK) != 0


def _in_reach(ctx, blobs):
    """Per event, at most this fraction of the doublets has a hit in reach: the
    predicted point (features 5 and 6, in 42 mm) within the fit's tolerance of
    0.6 mm and two cells (1.3125 and 84 / 256 mm) of a hit of the h2's module."""
    from cl_forward_gb300.events import pack_events, unpack_event
    buf, offs, sizes = pack_events(blobs)
    ctx.stage(buf, offs, sizes)
    feats, ids, count = ctx.dump_doublets(1 << 20)
    assert count == len(feats)
    out = []
    for e, b in enumerate(blobs):
        ev = unpack_event(b)
        module = ev.module_of_hit()
        mine = ids[:, 0] == e
        px, py, m4 = 42 * feats[mine, 5], 42 * feats[mine, 6], module[ids[mine, 1]] - 4
        near = np.zeros(len(px), bool)
        for m in np.unique(m4):
            k, h = m4 == m, module == m
            dx, dy = np.abs(px[k, None] - ev.x[h]), np.abs(py[k, None] - ev.y[h])
            near[k] = np.any((dx < 0.62 + 2 * 1.3125) & (dy < 0.62 + 2 * 84 / 256), 1)
        out.append(near.mean())
    return np.array(out)


@pytest.mark.parametrize("threads", [64, 256])
def test_all_scored_where_those_in_reach_are_too_few(gpu_ctx, threads):
    """Every scored doublet is kept: the guard of 0.9 is met by all doublets, and not by those in reach."""
    blobs, z = _blobs(), _weights()
    assert _in_reach(gpu_ctx, blobs).max() < 0.9
    gpu_ctx.set_mlp(z["weights"], -1e30, float(z["window_margin"]), 0.9)
    sparse, fell = _search(gpu_ctx, blobs, 0, threads)
    full, full_fell = _search(gpu_ctx, blobs, 1, threads)
    assert not np.any(fell) and not np.any(full_fell)
    assert sparse == full


@pytest.mark.parametrize("threads", [64, 256])
def test_some_events_fall_back(gpu_ctx, oracle_lib, threads):
    blobs, z = _blobs(), _weights()
    for rate in np.linspace(0.03, 0.3, 28):   # the first guard that some events trip and some do not
        gpu_ctx.set_mlp(z["weights"], float(z["keep_threshold"]), float(z["window_margin"]), float(rate))
        full, full_fell = _search(gpu_ctx, blobs, 1, threads)
        if np.any(full_fell):
            break
    assert 0 < np.count_nonzero(full_fell) < len(blobs)
    sparse, fell = _search(gpu_ctx, blobs, 0, threads)
    assert np.array_equal(fell, full_fell) and sparse == full
    want, _ = oracle_lib.search(blobs, 4)
    for e in np.flatnonzero(fell):
        assert sparse[e] == index_lists(want[e])
