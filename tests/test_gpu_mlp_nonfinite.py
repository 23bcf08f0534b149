"""Training on samples and weights that are not finite: a unit that is not live
(a NaN sum is not above 0) adds nothing to the gradient, so a NaN feature
leaves the training finite, and the gradient is NaN or infinite in the same
places as that of a plain FP32 evaluation.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradient(w, x, y, t):
    """The gradient of the mean loss; products with a gradient of 0 are left out."""
    from cl_forward_gb300 import learned
    from test_gpu_mlp_rounding import _forward
    with np.errstate(all="ignore"):
        h1, h2, o = (v.astype(np.float64) for v in _forward(w, x))
        A, a, B, b, C, c = (p.astype(np.float64) for p in learned.unpack(w))
        x, n = x.astype(np.float64), len(x)
        do = np.stack([1 / (1 + np.exp(-o[:, 0])) - y, y * 2 * learned.WIDTH_WEIGHT * (o[:, 1] - t)], 1) / n

        def live(g, v):   # sums over the samples of g[s, j] v[s, i]
            p = g[:, :, None] * v[:, None, :]
            return np.where(g[:, :, None] != 0, p, 0).sum(0)

        d2 = np.where(h2 > 0, do @ C, 0)
        d1 = np.where(h1 > 0, np.where(d2[:, :, None] != 0, d2[:, :, None] * B[None], 0).sum(1), 0)
        return np.concatenate([live(d1, x).ravel(), d1.sum(0), live(d2, h1).ravel(), d2.sum(0),
                               (do.T @ h2).ravel(), do.sum(0)])


def _data(n, seed):
    from test_gpu_mlp_step import _data
    return _data(n, seed)


@pytest.mark.parametrize("n", [1, 33, 700, 9729])
@pytest.mark.parametrize("where", ["first", "last", "all"])
def test_nan_feature(native_lib, n, where):
    from cl_forward_gb300 import learned, native
    x, y, t = _data(n, n)
    x[{"first": 0, "last": -1, "all": slice(None)}[where], 3] = np.nan
    w = learned.init_weights(n)
    got, loss = native.mlp_grad(w, x, y, t)
    want = _gradient(w, x, y, t)
    assert np.all(np.isfinite(want)) and np.isfinite(loss)
    # as in the gradient's own test: 512 roundings of terms of at most this size
    assert np.all(np.abs(got - want) <= 512 * 2.0 ** -24 * (1 + np.abs(want)))
    weights, losses = native.mlp_train(x, y, t, w, 5, n, 1e-3, 3)
    assert np.all(np.isfinite(weights)) and np.all(np.isfinite(losses))


@pytest.mark.parametrize("n", [33, 700])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("in_weights", [False, True])
def test_infinite(native_lib, n, value, in_weights):
    """NaN where the plain evaluation's gradient is, and finite where that is."""
    from cl_forward_gb300 import learned, native
    x, y, t = _data(n, n)
    w = learned.init_weights(n)
    if in_weights:
        w[352 + 5 * 32 + 7] = value    # layer 2, unit 5's weight of unit 7
    else:
        x[n // 2, 3] = value
    got, _ = native.mlp_grad(w, x, y, t)
    want = _gradient(w, x, y, t)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
