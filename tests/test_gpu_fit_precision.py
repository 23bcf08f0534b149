"""The track fit against extended precision, at the size of the coordinates that
it works on: transverse ones relative to the track's first hit.

Tolerance.  The results are rounded to FP32 once: half a unit in the last
place.  Before that, with V the largest transverse distance and U the largest
distance in z from the first hit, and at most 24 hits:

* FP32 pairs: a pair operation is good to 2^-46, a sum of 24 products of them
  to 26 x 2^-46; the solution of hits spread over U takes at most 12 times that
  to the slope and the intercept at the first hit: 2^-36 of V / U and of V.  The
  line is carried to z = 0 in FP64 (2^-50 of its terms).  Residuals: 2^-36 of V.
* FP64 about the origin, X and Z the largest coordinates (coordinates of 1e6
  and more, distances of 1e6 and more or of 1e-9 and less): sums to 26 x 2^-53,
  whose differences the determinant multiplies by up to 16 (Z / U)^2: 2^-42 of
  the sums' terms.
"""
import numpy as np
import pytest

from cl_forward_gb300.events import TRACK_DTYPE, Event, pack_event, unpack_event

FIELDS = ("x0", "tx", "y0", "ty", "chi2_ndf")
WEIGHT = 3966.94

# modules (3: the three of a shortest track), transverse scale, x shift, lines
# without noise, and the arithmetic that the case is made for
CASES = [(3, 1.0, 0.0, False, "pairs"), (24, 1.0, 0.0, False, "pairs"), (44, 1.0, 0.0, True, "pairs"),
         (12, 1.0, 3000.0, False, "pairs"), (12, 1e-3, 0.0, False, "pairs"), (12, 1e-6, 0.0, False, "pairs"),
         (12, 1.0, 2e6, True, "fp64"), (12, 1e-12, 0.0, False, "fp64")]


def _event(seed, n_modules, scale, shift, exact):
    """Straight tracks over consecutive modules, or over modules 2, 4 and 6 of 7, a hit each."""
    rng = np.random.Generator(np.random.PCG64(seed))
    on = np.array([2, 4, 6]) if n_modules == 3 else np.arange(n_modules)
    n_modules, lines = on[-1] + 1, 12
    z = 25.0 * np.arange(n_modules) - 150.0
    x0, y0, tx, ty = (rng.uniform(-a, a, lines) for a in (20, 20, 0.05, 0.05))
    if exact:   # every coordinate a multiple of 1/8: exact also at 2e6
        x0, y0, tx, ty = np.round(x0), np.round(y0), np.round(tx * 200) / 200, np.round(ty * 200) / 200
    m, line = np.repeat(on, lines), np.tile(np.arange(lines), len(on))
    num = np.bincount(m, minlength=n_modules)
    noise = 0.0 if exact else 0.012
    x = scale * (x0[line] + tx[line] * z[m] + rng.normal(0, noise, len(m))) + shift
    y = scale * (y0[line] + ty[line] * z[m] + rng.normal(0, noise, len(m)))
    ev = Event(np.trunc(z).astype(np.int32), (np.cumsum(num) - num).astype(np.int32), num.astype(np.int32),
               ((np.arange(len(m)) << 8) | m).astype(np.uint32), x.astype(np.float32), y.astype(np.float32),
               z[m].astype(np.float32))
    return pack_event(ev), line


def _exact(track, ev):
    """The fit in extended precision, its allowed error before the rounding to FP32, and which arithmetic it takes."""
    L = np.longdouble
    h = track["hits"][:int(track["hitsNum"])].astype(int)
    x, y, z = (a[h].astype(L) for a in (ev.x, ev.y, ev.z))
    n, w = L(len(h)), z - z[0]   # exact, as all differences below
    wc = w - w.mean()
    szz, u = (wc * wc).sum(), float(np.abs(w).max())
    d = np.abs(np.concatenate([v - v[0] for v in (x, y, z)])).astype(float)
    fp64 = bool(np.any(d >= 1e6) or np.any((d > 0) & (d <= 1e-9)) or max(abs(float(v[0])) for v in (x, y, z)) >= 1e6)
    out, slack, chi2, chi2_slack = np.zeros(5, L), np.zeros(5), L(0), 0.0
    for k, v in ((0, x), (2, y)):
        q = v - v[0]
        s = (wc * q).sum() / szz
        at_first = q.mean() - s * w.mean()
        a = v[0] + (at_first - s * z[0])
        r = np.abs(q - (at_first + s * w)).astype(float)
        out[k], out[k + 1] = a, s
        if fp64:
            X, Z = float(np.abs(v).max()), float(np.abs(z).max())
            ds = 2.0 ** -42 * (X * Z + abs(float(s)) * Z * Z) / u ** 2
            da = 2.0 ** -42 * X + ds * Z
            dr = da + ds * Z + 2.0 ** -50 * X
        else:
            V = float(np.abs(v - v[0]).max())
            ds = 2.0 ** -36 * V / u
            da = 2.0 ** -36 * V * (1 + abs(float(z[0])) / u) + 2.0 ** -50 * (abs(float(v[0])) + abs(float(s * z[0])))
            dr = 2.0 ** -36 * V
        slack[k], slack[k + 1] = da, ds
        chi2 += L(WEIGHT) * ((q - (at_first + s * w)) ** 2).sum()
        chi2_slack += WEIGHT * float((2 * r * dr + dr * dr).sum())
    ndf = float(2 * n - 4)
    if ndf > 0:
        out[4], slack[4] = chi2 / L(ndf), chi2_slack / ndf + 2.0 ** -48 * float(chi2) / ndf
    return out, slack, fp64


def _off(fit, want, slack):
    """The largest error of a fit's values over what is allowed."""
    got = np.array([fit[k] for k in FIELDS])
    ulp = np.spacing(np.maximum(np.abs(got), np.abs(want.astype(np.float32))))
    return float((np.abs(got.astype(np.longdouble) - want).astype(float) / (0.5001 * ulp + slack)).max())


@pytest.mark.parametrize("case", CASES)
def test_wrong_fits_are_told(case):
    """The bounds pass the exact fit rounded to FP32 and no other: each value zeroed, or off by 1e-6 of itself."""
    blob, line = _event(40, *case[:4])
    ev = unpack_event(blob)
    told = np.zeros((5, 2), int)
    for k in range(12):
        t = np.zeros((), TRACK_DTYPE)
        h = np.flatnonzero(line == k)[:22]
        t["hitsNum"], t["hits"][:len(h)] = len(h), h
        want, slack, fp64 = _exact(t, ev)
        assert case[4] == "both" or fp64 == (case[4] == "fp64")
        fit = dict(zip(FIELDS, want.astype(np.float32)))
        assert _off(fit, want, slack) <= 1
        for f, name in enumerate(FIELDS):
            for wrong, factor in enumerate((0.0, 1 + 1e-6)):
                told[f, wrong] += _off({**fit, name: np.float32(float(want[f]) * factor)}, want, slack) > 1
    zero = np.array([bool(case[3]) and f == 4 for f in range(5)])   # chi2 of exact lines is near 0
    assert np.all(told[~zero] >= 6), told


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_fit(gpu_ctx, case):
    from cl_forward_gb300 import native
    from cl_forward_gb300.events import pack_events
    blobs = [native.sort_by_x(_event(40 + k, *case[:4])[0]) for k in range(3)]
    buf, offs, sizes = pack_events(blobs)
    gpu_ctx.stage(buf, offs, sizes)
    gpu_ctx.run(native.default_options())
    cap = sum(int(np.frombuffer(b[4:8], "<i4")[0]) for b in blobs)
    tracks, counts, first, _ = gpu_ctx.fetch(len(blobs), cap)
    fits = gpu_ctx.fit_tracks(cap)
    taken = {False: 0, True: 0}
    for e, b in enumerate(blobs):
        ev = unpack_event(b)
        for i in range(int(first[e]), int(first[e]) + int(counts[e])):
            want, slack, fp64 = _exact(tracks[i], ev)
            taken[fp64] += 1
            assert _off(fits[i], want, slack) <= 1, (i, fits[i], want)
    assert taken[True] >= (6 if case[4] != "pairs" else 0) and taken[False] >= (6 if case[4] != "fp64" else 0), taken
