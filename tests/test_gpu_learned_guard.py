"""Learned seeding scores the doublets in reach of a hit first and the rest only
where the keep-rate guard needs them: at guards that no event, some events and
every event trip, the same events fall back and every event's tracks are the
same as with all doublets scored (learned_min_window = 1, which every doublet
that has a window reaches).
"""
import os

import numpy as np
import pytest

from conftest import ROOT, index_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [64, 256])
@pytest.mark.parametrize("rate", [0.0, 0.02, 0.05, 0.08, 0.1, 0.5])
def test_guard_decides_as_with_all_scored(gpu_ctx, oracle_lib, rate, threads):
    from cl_forward_gb300 import generator, native
    z = np.load(os.path.join(ROOT, "cl_forward_gb300", "weights", "doublet_mlp.npz"))
    blobs = [oracle_lib.sort_by_x(b) for b in generator.generate(range(100300, 100364))[0]]
    gpu_ctx.set_mlp(z["weights"], float(z["keep_threshold"]), float(z["window_margin"]), rate)
    runs = []
    for min_window in (0, 1):
        o = native.default_options(learned=1, learned_min_window=min_window, threads_per_event=threads,
                                   register_ctas=4)
        got, status = gpu_ctx.search(blobs, o)
        runs.append((np.asarray(status), [index_lists(g) for g in got]))
    assert np.array_equal(runs[0][0], runs[1][0])
    assert runs[0][1] == runs[1][1]
    fell = int(np.count_nonzero(runs[0][0] & native.EVENT_LEARNED_FALLBACK))
    if rate in (0.0, 0.5):
        assert fell == (len(blobs) if rate else 0)
    if rate == 0.5:
        want, _ = oracle_lib.search(blobs, 4)
        assert runs[0][1] == [index_lists(t) for t in want]
