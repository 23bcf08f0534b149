"""The training-step kernel at the edges of its tiles (32 samples per pass, at
most two CTAs per SM, each CTA several tiles beyond that) against float64.

Tolerance.  A gradient is a mean over the samples of products; in FP32 each
product carries the rounding of at most 10 + 32 + 2 + 32 multiply-adds and a
few more operations, and the sum adds at most one rounding per sample of a
tile, tile of a CTA and CTA: under 512 roundings of 2^-24 in all, relative to
the sum of the products' absolute values.  Samples whose unit lies within
1e-5 of its ReLU threshold may fall on either side of it: their whole
contribution is allowed as well.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUNDINGS = 512 * 2.0 ** -24
NEAR = 1e-5


def _data(n, seed):
    from cl_forward_gb300 import learned
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.normal(0, 1, (n, learned.N_IN)).astype(np.float32)
    y = (rng.random(n) < 0.2).astype(np.float32)
    t = (np.abs(rng.normal(0.1, 0.05, n)) * y).astype(np.float32)
    return x, y, t


def _bound(w, x, y, t):
    """Per parameter: the sum of the products' absolute values, and the share of near-threshold samples in it."""
    from cl_forward_gb300 import learned
    A, a, B, b, C, c = learned.unpack(w)
    x = x.astype(np.float64)
    z1 = x @ A.T + a
    h1 = np.maximum(z1, 0)
    z2 = h1 @ B.T + b
    h2 = np.maximum(z2, 0)
    o = h2 @ C.T + c
    n = len(x)
    do = np.abs(np.stack([1 / (1 + np.exp(-o[:, 0])) - y, y * 2 * learned.WIDTH_WEIGHT * (o[:, 1] - t)], 1)) / n + 1e-7 / n
    out = []
    for keep1, keep2 in ((z1 > -NEAR, z2 > -NEAR), (np.abs(z1) < NEAR, np.abs(z2) < NEAR)):
        near = keep1 is not None and out
        d2 = (do @ np.abs(C)) * keep2
        d1 = ((do @ np.abs(C) * (z2 > -NEAR)) @ np.abs(B)) * keep1
        if near:   # a flip of layer 2 also changes what reaches layer 1
            d1 = d1 + (d2 @ np.abs(B)) * (z1 > -NEAR)
        gC = np.zeros_like(C) if near else do.T @ h2
        gc = np.zeros_like(c) if near else do.sum(0)
        out.append(np.concatenate([(d1.T @ np.abs(x)).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), gC.ravel(), gc]))
    return ROUNDINGS * out[0] + out[1]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 100, 4096, 9728, 9729, 30001])
def test_gradient(native_lib, n):
    from cl_forward_gb300 import learned, native
    w = learned.init_weights(n)
    x, y, t = _data(n, n + 1)
    g, loss = native.mlp_grad(w, x, y, t)
    loss_ref, g_ref = learned.reference_loss_and_grad(w, x, y, t)
    assert abs(loss - loss_ref) <= ROUNDINGS * (1 + abs(loss_ref))
    assert np.all(np.abs(g - g_ref) <= _bound(w, x, y, t) + 1e-12)


def _order(n, count, seed):
    """velo_mlp_train's sample order: a Fisher-Yates shuffle per epoch, driven by splitmix64."""
    mask, s, order, out = (1 << 64) - 1, seed, list(range(n)), []
    while len(out) < count:
        for i in range(n - 1, 0, -1):
            s = (s + 0x9E3779B97F4A7C15) & mask
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            order[i], order[j] = order[j], order[i]
        out += order[:count - len(out)]
    return np.array(out)


@pytest.mark.parametrize("n, batch, steps", [(1, 1, 3), (50, 33, 4), (500, 32, 20), (700, 100, 9), (12000, 9729, 3)])
def test_steps(native_lib, n, batch, steps):
    """Adam over the documented sample order.  An update is at most about lr
    per step whatever the gradient's size, so a parameter whose gradients stay
    near their rounding may differ by that; those are few."""
    from cl_forward_gb300 import learned, native
    x, y, t = _data(n, n)
    w0 = learned.init_weights(3)
    got, losses = native.mlp_train(x, y, t, w0, steps, batch, 1e-3, 7)
    idx = _order(n, steps * batch, 7).reshape(steps, batch)
    b1, b2, lr, eps = (float(np.float32(v)) for v in (0.9, 0.999, 1e-3, 1e-8))
    w = w0.astype(np.float64)
    m, v = np.zeros_like(w), np.zeros_like(w)
    for k in range(steps):
        loss, g = learned.reference_loss_and_grad(w, x[idx[k]], y[idx[k]], t[idx[k]])
        assert abs(losses[k] - loss) <= 1e-4 * (1 + abs(loss))
        m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
        w = w - lr * (m / (1 - b1 ** (k + 1))) / (np.sqrt(v / (1 - b2 ** (k + 1))) + eps)
    off = np.abs(got - w)
    assert off.max() <= 4 * lr * steps
    assert np.mean(off > 1e-2 * lr * steps) < 0.01


@pytest.mark.parametrize("n, batch, steps", [(2, 3, 50), (3, 1, 40), (257, 256, 30), (5000, 8192, 135)])
def test_sample_order(native_lib, n, batch, steps):
    """With a learning rate of 0 each step's loss is that of its samples under
    the initial weights: every sample of every epoch shows, also where the
    draws are made in several launches (the last case: over 2^20 of them)."""
    from cl_forward_gb300 import learned, native
    x, y, t = _data(n, n)
    w = learned.init_weights(9)
    got, losses = native.mlp_train(x, y, t, w, steps, batch, 0.0, 123)
    assert np.array_equal(got, w)
    o = learned.forward_np(w, x)
    z, wd = o[:, 0], o[:, 1]
    per_sample = np.maximum(z, 0) - z * y + np.log1p(np.exp(-np.abs(z))) + y * learned.WIDTH_WEIGHT * (wd - t) ** 2
    want = per_sample[_order(n, steps * batch, 123)].reshape(steps, batch).mean(1)
    assert np.all(np.abs(losses - want) <= ROUNDINGS * (1 + np.abs(want)))
