"""The estimator's products at the sizes where their tiles and slices end:
forward and backward against the FP32 CPU reference (which rounds to BF16 where
the device does), the bound of tests/test_gpu_estimator.py."""
import mlp_ref
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(pkg, n, seed):
    rng = np.random.default_rng(seed)
    x = (rng.random((n, pkg.EST_FEATURES)) * (rng.random((n, pkg.EST_FEATURES)) < 0.1)).astype(np.float32)
    return x, (rng.random(n) * 20).astype(np.float32)


# A lone row, 32- and 64-row tiles, padding to 64, row-sum chunks, many tiles.
@pytest.mark.parametrize("n", [1, 31, 64, 65, 256, 257, 1000])
def test_gradients(pkg, n):
    est = pkg.Estimator(0, seed=n)
    x, t = _data(pkg, n, n)
    p = est.params()
    loss, g = est.gradients(x, t)
    want_loss, want = mlp_ref.loss_and_grads(p, x, t)
    assert loss == pytest.approx(want_loss, rel=1e-2)
    F, H = mlp_ref.F, mlp_ref.H
    for name, o, k in (("W1", 0, F * H), ("b1", F * H, H), ("W2", F * H + H, H * H), ("b2", F * H + H + H * H, H),
                       ("w3", F * H + 2 * H + H * H, H), ("b3", F * H + 3 * H + H * H, 1)):
        rel = np.linalg.norm(g[o:o + k] - want[o:o + k]) / max(np.linalg.norm(want[o:o + k]), 1e-12)
        assert rel < 2e-2, f"{name}: {rel:.3g}"
    assert not g[F * H + 3 * H + H * H + 1:].any()  # the padding has no gradient


# 64 x 64 tiles from 2,368 rows on; the chunk of 4,096 rows.
@pytest.mark.parametrize("n", [1, 64, 2368, 2369, 4096, 4097])
def test_predictions(pkg, n):
    est = pkg.Estimator(0, seed=7)
    x, _ = _data(pkg, n, n)
    y = est.predict(x)
    _, _, _, want = mlp_ref.forward(est.params(), x)
    assert np.abs(y - want).max() <= 1e-2 * max(1.0, np.abs(want).max())


# A batch's rows are picked by the epoch's shuffle: one step on a batch of the whole set, in any order, is one Adam step
# on the set's gradient.
@pytest.mark.parametrize("n", [40, 64, 300])
def test_first_step_is_adam(pkg, n):
    est = pkg.Estimator(0, seed=3)
    x, t = _data(pkg, n, n)
    p = est.params()
    p[mlp_ref.F * mlp_ref.H + 3 * mlp_ref.H + mlp_ref.H ** 2] = np.float32(t.mean(dtype=np.float64))  # as training starts
    ref = pkg.Estimator(0, seed=3)
    ref.set_params(p)
    _, g = ref.gradients(x, t)
    est.train(x, t, epochs=1, batch=n, lr=1e-3, seed=5)
    q = est.params()
    big = np.abs(g) > 1e-6 * np.abs(g).max()
    step = (p.astype(np.float64) - q)[big]
    # Bias-corrected first moments: lr * g / (|g| + eps), to the rounding of p - q in FP32 and of sums in another order.
    want = 1e-3 * g[big].astype(np.float64) / (np.abs(g[big]) + 1e-8)
    assert np.abs(step - want).max() <= 2 ** -23 * np.abs(p).max() + 1e-3 * 1e-2
