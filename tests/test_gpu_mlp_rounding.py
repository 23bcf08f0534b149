"""The training step's decisions: a unit whose sum lies within rounding of its
ReLU threshold is live or not as in a plain FP32 evaluation of the network
(every product rounded, then added, in index order).

Tolerance.  With the decisions given, a gradient is a mean of products whose
factors carry at most 2 (10 + 32 + 32 + 2 + 32) roundings of 2^-24 and some
more from the loss, and whose sum adds one per sample of a tile, tile of a CTA
and CTA: under 512 in all, relative to the same sums over absolute values
(activations by the absolute values of their own terms, as cancellation in
them leaves their rounding).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUNDINGS = 512 * 2.0 ** -24


def _chain(w, b, x, fused=False):
    """b + w x in FP32, term by term; products rounded, or fused into the sum."""
    s = np.repeat(b[None], len(x), 0)
    for i in range(x.shape[1]):
        if fused:   # a product of two floats is exact in 64 bits
            s = (s.astype(np.float64) + x[:, i, None].astype(np.float64) * w[None, :, i]).astype(np.float32)
        else:
            s = s + x[:, i, None] * w[None, :, i]
    return s


def _forward(w, x, fused=False):
    from cl_forward_gb300 import learned
    A, a, B, b, C, c = (p.astype(np.float32) for p in learned.unpack(w))
    z1 = _chain(A, a, x, fused)
    h1 = np.where(z1 > 0, z1, np.float32(0))
    z2 = _chain(B, b, h1, fused)
    h2 = np.where(z2 > 0, z2, np.float32(0))
    return h1, h2, _chain(C, c, h2, fused)


def _gradient(w, x, y, t, fused=False):
    """The gradient of the mean loss, in 64 bits but for the FP32 decisions, and its allowed error."""
    from cl_forward_gb300 import learned
    h1, h2, o = (v.astype(np.float64) for v in _forward(w, x, fused))
    A, a, B, b, C, c = (p.astype(np.float64) for p in learned.unpack(w))
    x, n = x.astype(np.float64), len(x)
    do = np.stack([1 / (1 + np.exp(-o[:, 0])) - y, y * 2 * learned.WIDTH_WEIGHT * (o[:, 1] - t)], 1) / n
    d2 = (do @ C) * (h2 > 0)
    d1 = (d2 @ B) * (h1 > 0)
    m1 = np.abs(x) @ np.abs(A).T + np.abs(a)
    m2 = m1 @ np.abs(B).T + np.abs(b)
    e3 = np.abs(do) + (m2 @ np.abs(C).T + np.abs(c)) * 0.25 / n
    e2 = (e3 @ np.abs(C)) * (h2 > 0)
    e1 = (e2 @ np.abs(B)) * (h1 > 0)

    def flat(d1, x, d2, h1, do, h2):
        return np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), (do.T @ h2).ravel(), do.sum(0)])

    return flat(d1, x, d2, h1, do, h2), ROUNDINGS * flat(e1, np.abs(x), e2, m1, e3, m2)


def _at_threshold(w, n, layer, seed):
    """Samples each of which puts one unit of the layer within rounding of 0."""
    from cl_forward_gb300 import learned
    rng = np.random.Generator(np.random.PCG64(seed))
    A, a, B, b = (p.astype(np.float64) for p in learned.unpack(w)[:4])

    def z(x):
        z1 = x @ A.T + a
        return z1 if layer == 1 else np.maximum(z1, 0) @ B.T + b

    unit = np.arange(n) % 3
    lo, hi = (rng.normal(0, 1, (n, 40, learned.N_IN)) for _ in range(2))   # 40 tries for a pair on both sides
    zl, zh = (np.take_along_axis(z(v.reshape(-1, learned.N_IN)).reshape(n, 40, -1), unit[:, None, None], 2)[:, :, 0] for v in (lo, hi))
    k = np.argmax(zl, 1)
    lo, k2 = lo[np.arange(n), k], np.argmin(zh, 1)
    hi = hi[np.arange(n), k2]
    ok = (zl[np.arange(n), k] > 0) & (zh[np.arange(n), k2] < 0)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        up = (z(mid)[np.arange(n), unit] > 0)[:, None]
        lo, hi = np.where(up, mid, lo), np.where(up, hi, mid)
    return lo[ok].astype(np.float32)


@pytest.mark.parametrize("layer", [1, 2])
@pytest.mark.parametrize("n", [40, 1000, 12000])
def test_decisions_at_the_threshold(native_lib, layer, n):
    from cl_forward_gb300 import learned, native
    w = learned.init_weights(n + layer)
    x = _at_threshold(w, n, layer, n)
    rng = np.random.Generator(np.random.PCG64(n + 1))
    y = (rng.random(len(x)) < 0.2).astype(np.float32)
    t = (np.abs(rng.normal(0.1, 0.05, len(x))) * y).astype(np.float32)
    want, slack = _gradient(w, x, y, t)
    # the samples tell the two ways of rounding apart
    assert np.any(np.abs(_gradient(w, x, y, t, fused=True)[0] - want) > 2 * slack)
    got, _ = native.mlp_grad(w, x, y, t)
    off = np.abs(got - want)
    assert np.all(off <= slack), float((off / slack).max())


@pytest.mark.parametrize("seed", range(20))
def test_training_follows_fp32(native_lib, seed):
    """Weights after 30 steps against a plain FP32 training whose gradients are
    summed in 64 bits.  One parameter off by one whole Adam step of 1e-3 moves
    the weights by 1.4e-4 of their norm; a seventh of that is allowed."""
    from cl_forward_gb300 import learned, native
    from test_gpu_mlp_step import _data, _order
    n, batch, steps = 4000, 1000, 30
    x, y, t = _data(n, 500 + seed)
    w0 = learned.init_weights(seed)
    got, _ = native.mlp_train(x, y, t, w0, steps, batch, 1e-3, seed)
    f = np.float32
    b1, b2, lr, eps = f(0.9), f(0.999), f(1e-3), f(1e-8)
    w = w0.astype(f)
    m, v = np.zeros_like(w), np.zeros_like(w)
    for k, idx in enumerate(_order(n, steps * batch, seed).reshape(steps, batch)):
        g = _gradient(w, x[idx], y[idx], t[idx])[0].astype(f)
        m, v = b1 * m + (f(1) - b1) * g, b2 * v + (f(1) - b2) * g * g
        c1, c2 = f(1 - float(b1) ** (k + 1)), f(1 - float(b2) ** (k + 1))
        w = w - lr * (m / c1) / (np.sqrt(v / c2) + eps)
    assert np.linalg.norm(got - w) <= 2e-5 * np.linalg.norm(w)
