"""The track fit's FP32-pair sums against an extended-precision fit.

Tolerance.  The results are rounded to FP32 once: half a unit in the last
place.  Before that, sums of FP32 pairs carry 2^-46 of their terms' size, and
the solution multiplies it by at most the spread of the terms over the result:
2^-38 of the terms (coordinates for x0 and y0 at z = 0, coordinate over z spread
for the slopes) is allowed; chi2 carries its residuals' 2^-45 of the
coordinates, 2^-38 of them is allowed per residual.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ATTACHED = 2.0 ** -38


def exact_fits(tracks, blob):
    """x0, tx, y0, ty, chi2 / ndf in extended precision, and the allowed error before the rounding to FP32."""
    from cl_forward_gb300.events import unpack_event
    ev = unpack_event(blob)
    L = np.longdouble
    out, slack = np.zeros((len(tracks), 5), L), np.zeros((len(tracks), 5))
    for i, t in enumerate(tracks):
        h = t["hits"][:int(t["hitsNum"])].astype(int)
        x, y, z = (a[h].astype(L) for a in (ev.x, ev.y, ev.z))
        n = L(len(h))
        zc = z - z.mean()
        szz = (zc * zc).sum()
        if not szz > 0:
            continue
        size = float(max(np.abs(x).max(), np.abs(y).max(), np.abs(z).max()))
        spread = float(np.abs(zc).max())
        reach = 1 + float(np.abs(z).max()) / spread
        chi2 = L(0)
        worst = 0.0
        for k, v in ((0, x), (2, y)):
            s = (zc * v).sum() / szz
            a = v.mean() - s * z.mean()
            r = v - (a + s * z)
            chi2 += L(3966.94) * (r * r).sum()
            worst = max(worst, float(np.abs(r).max()))
            out[i, k], out[i, k + 1] = a, s
            slack[i, k], slack[i, k + 1] = ATTACHED * size * reach, ATTACHED * size / spread
        ndf = 2 * n - 4
        out[i, 4] = chi2 / ndf if ndf > 0 else 0
        d = ATTACHED * size
        slack[i, 4] = 3966.94 * float(n) * (2 * worst * d + d * d) + 1e-15 * float(chi2)   # kPixelWeight in FP64
    return out, slack


def assert_fits(fits, tracks, blob):
    want, slack = exact_fits(tracks, blob)
    got = np.stack([fits[k] for k in ("x0", "tx", "y0", "ty", "chi2_ndf")], 1)
    ulp = np.spacing(np.maximum(np.abs(got), np.abs(want.astype(np.float32))))
    off = np.abs(got.astype(np.longdouble) - want).astype(np.float64)
    assert np.all(off <= 0.5001 * ulp + slack), float((off / (0.5 * ulp + slack)).max())


def _event(seed, n_modules, scale, shift, exact):
    """Straight tracks on consecutive even modules, a hit each."""
    from cl_forward_gb300.events import Event, pack_event
    from cl_forward_gb300 import native
    rng = np.random.Generator(np.random.PCG64(seed))
    z = 25.0 * np.arange(n_modules) - 150.0
    lines = 12
    x0, y0, tx, ty = (rng.uniform(-a, a, lines) for a in (20, 20, 0.05, 0.05))
    if exact:
        x0, y0, tx, ty = np.round(x0), np.round(y0), np.round(tx * 100) / 256, np.round(ty * 100) / 256
    m = np.repeat(np.arange(n_modules), lines)
    line = np.tile(np.arange(lines), n_modules)
    noise = 0.0 if exact else 0.012
    x = scale * (x0[line] + tx[line] * z[m] + rng.normal(0, noise, len(m))) + shift
    y = scale * (y0[line] + ty[line] * z[m] + rng.normal(0, noise, len(m)))
    ev = Event(np.trunc(z).astype(np.int32), (lines * np.arange(n_modules)).astype(np.int32),
               np.full(n_modules, lines, np.int32), ((np.arange(len(m)) << 8) | m).astype(np.uint32),
               x.astype(np.float32), y.astype(np.float32), z[m].astype(np.float32))
    return native.sort_by_x(pack_event(ev))


@pytest.mark.parametrize("n_modules, scale, shift, exact", [
    (5, 1.0, 0.0, False), (6, 1.0, 0.0, True), (24, 1.0, 0.0, False), (44, 1.0, 0.0, False),
    (12, 1e-6, 0.0, False), (12, 1.0, 3000.0, False), (12, 1.0, 2e6, True), (12, 1e-12, 0.0, False)])
def test_ranges(gpu_ctx, n_modules, scale, shift, exact):
    """Three to 22 hits, exact lines, and coordinates inside and outside the pairs' range (the last two)."""
    _fit_and_check(gpu_ctx, [_event(40 + k, n_modules, scale, shift, exact) for k in range(3)])


def test_generated_events(gpu_ctx):
    from cl_forward_gb300 import generator, native
    blobs = [native.sort_by_x(b) for b in generator.generate(range(60, 66))[0]]
    assert _fit_and_check(gpu_ctx, blobs) > 500


def _fit_and_check(ctx, blobs):
    from cl_forward_gb300 import native
    from cl_forward_gb300.events import pack_events
    buf, offs, sizes = pack_events(blobs)
    ctx.stage(buf, offs, sizes)
    ctx.run(native.default_options())
    cap = sum(int(np.frombuffer(b[4:8], "<i4")[0]) for b in blobs)
    tracks, counts, first, _ = ctx.fetch(len(blobs), cap)
    fits = ctx.fit_tracks(cap)
    for e, b in enumerate(blobs):
        rows = slice(int(first[e]), int(first[e]) + int(counts[e]))
        if counts[e]:
            assert_fits(fits[rows], tracks[rows], b)
    return int(counts.sum())
