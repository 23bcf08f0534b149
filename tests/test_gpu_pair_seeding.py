"""The pair seeding (sorted modules, coordinates near the detector) against
the oracle and against the general seeding (narrow_windows = 0), where it can
go wrong: module occupancies around a warp, several z values per module,
h1s without an h2 window in the middle of a module, Y-lanes of every kind,
modules out of order, and coordinates that send an event to the general path.
Results are hit-index lists and status bits: the bar is equality.
"""
import numpy as np
import pytest

from conftest import index_lists

pytestmark = pytest.mark.gpu


def _event(seed, per_module, z_style="one", shift=0.0, swap=False, n_modules=14):
    """Exactly `per_module` hits on each of n_modules modules, on straight
    lines and at random, all on a 0.25 mm grid (fits tie), x-sorted.  Every
    other pair of modules ends at a lower x than the h2 windows of the pair
    after it reach, so some h1s have no window."""
    from cl_forward_gb300.events import Event, pack_event
    rng = np.random.Generator(np.random.PCG64(seed))
    z = 20.0 * np.arange(n_modules) - 100.0
    step = 0.25 * rng.integers(-2, 3, (per_module, 2))           # per module: the lines stay on the grid
    at = 0.25 * rng.integers(-60, 61, (per_module, 2))
    on_line = rng.random((n_modules, per_module)) < 0.7
    if n_modules > 20:
        on_line[np.arange(n_modules) % 16 > 9] = False   # no track reaches 25 hits
    xs, ys, zs = [], [], []
    for m in range(n_modules):
        top = 20.0 if m % 4 < 2 else -5.0
        free = np.round(rng.uniform((-40, -20), (top, 20), (per_module, 2)) / 0.25) * 0.25
        xy = np.where(on_line[m][:, None], at + step * m, free)
        xy = xy[np.argsort(xy[:, 0], kind="stable")]
        x, y = xy[:, 0] + shift, xy[:, 1]
        if swap and m == n_modules // 2 and per_module > 1:
            x[0] = x[1] + 1.0
        xs.append(x)
        ys.append(y)
        zs.append({"one": np.full(per_module, z[m]), "two": z[m] + (np.arange(per_module) % 2),
                   "many": z[m] + np.round(rng.uniform(-2, 2, per_module), 1)}[z_style])
    H = n_modules * per_module
    mods = np.repeat(np.arange(n_modules), per_module)
    return pack_event(Event(
        sensor_z=np.trunc(z).astype(np.int32), hit_start=(per_module * np.arange(n_modules)).astype(np.int32),
        hit_num=np.full(n_modules, per_module, np.int32),
        hit_id=((np.arange(H) << 8) | mods).astype(np.uint32), x=np.concatenate(xs).astype(np.float32),
        y=np.concatenate(ys).astype(np.float32), z=np.concatenate(zs).astype(np.float32)))


def _check(gpu_ctx, oracle_lib, blobs, y, **opts):
    from cl_forward_gb300 import native
    got, status = gpu_ctx.search(blobs, native.default_options(y_lanes=y, **opts))
    plain, pstatus = gpu_ctx.search(blobs, native.default_options(y_lanes=y, narrow_windows=0, **opts))
    want, ostatus = oracle_lib.search(blobs, y)
    compared = tracks = 0
    for e in range(len(blobs)):
        if ostatus[e] & oracle_lib.PARITY_EXCLUDING:
            continue
        assert status[e] == ostatus[e] and pstatus[e] == ostatus[e]
        assert index_lists(got[e]) == index_lists(want[e]) == index_lists(plain[e]), f"event {e}, Y={y}, {opts}"
        compared += 1
        tracks += len(got[e])
    return compared, tracks


@pytest.mark.parametrize("threads", [32, 64, 256, 512])
@pytest.mark.parametrize("z_style", ["one", "two", "many"])
@pytest.mark.parametrize("per_module", [1, 2, 31, 32, 33, 65])
def test_module_sizes_and_z(gpu_ctx, oracle_lib, per_module, z_style, threads):
    blobs = [_event(100 * per_module + k, per_module, z_style) for k in range(6)]
    for y in (1, 3, 4, 16):
        compared, tracks = _check(gpu_ctx, oracle_lib, blobs, y, threads_per_event=threads)
        assert compared == len(blobs)
    assert per_module < 31 or tracks > 0


@pytest.mark.parametrize("n_modules", [4, 5, 6, 7, 63, 64, 65])
def test_module_counts(gpu_ctx, oracle_lib, n_modules):
    blobs = [_event(7000 + k, 9, "two" if k % 2 else "one", n_modules=n_modules) for k in range(4)]
    _check(gpu_ctx, oracle_lib, blobs, 4)


def test_general_path_beside_it(gpu_ctx, oracle_lib):
    """One batch of events that take the pair seeding and events that cannot:
    a module out of order, coordinates beyond the detector's range."""
    blobs = [_event(9000 + k, 40, "one", shift=(0.0, 2.0e4, 0.0)[k % 3], swap=k % 3 == 2) for k in range(9)]
    for threads in (32, 64, 128):
        compared, tracks = _check(gpu_ctx, oracle_lib, blobs, 4, threads_per_event=threads)
        assert compared == len(blobs) and tracks > 0


@pytest.mark.parametrize("y, min_window", [(4, 0), (4, 3), (3, 0), (1, 2)])
def test_learned_pairs(gpu_ctx, y, min_window):
    """Doublets scored in the queue's batches against doublets scored where the
    windows are walked (narrow_windows = 0): with a window margin beyond the
    exact cut the network only prunes, so both keep the same doublets, and the
    keep-rate guard, which counts every scored one, sends the same events back."""
    from cl_forward_gb300 import generator, learned, native
    blobs = [native.sort_by_x(b) for b in generator.generate(range(5200, 5216))[0]]
    blobs += [_event(9500 + k, 33, "one") for k in range(4)] + [_event(9600, 20, "two")]
    w = learned.init_weights(11)
    ds = learned.build_dataset(gpu_ctx, blobs[:16])
    logits = native.mlp_forward(w, ds.x)[:, 0]
    threshold = float(np.quantile(logits, 0.4))
    opts = dict(learned=1, y_lanes=y, learned_min_window=min_window)
    for guard in (0.0, 0.6, 1.0):
        gpu_ctx.set_mlp(w, threshold, 100.0, guard)
        got, status = gpu_ctx.search(blobs, native.default_options(**opts))
        walked, wstatus = gpu_ctx.search(blobs, native.default_options(narrow_windows=0, **opts))
        assert np.array_equal(status, wstatus)
        for e in range(len(blobs)):
            assert index_lists(got[e]) == index_lists(walked[e]), f"event {e}, guard {guard}"
    assert np.any(status & native.EVENT_LEARNED_FALLBACK)
