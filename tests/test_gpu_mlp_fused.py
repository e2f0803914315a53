"""The scorer's fused kernels at the edges of their range (layers of up to 128
units, odd sizes, ragged batches) and the layer kernels beyond it, against the
float64 oracle: forward, BF16 forward, gradients and whole Adam runs."""
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "oracle"))

DIMS = [(1, 1), (7, 5), (33, 100), (64, 128), (128, 128), (24, 16), (129, 20), (16, 130)]


@pytest.mark.parametrize("rows", [1, 3, 32, 33, 130])
@pytest.mark.parametrize("d,h", DIMS)
def test_forward_and_gradients(sge, d, h, rows):
    import mlp_oracle as mo
    rng = np.random.default_rng(d * 1000 + h + rows)
    mlp = sge.MLP(d, h, seed=d + h)
    x = rng.normal(size=(rows, d)).astype(np.float32)
    t = rng.normal(size=rows).astype(np.float32)
    p = mlp.get_params()
    want = mo.forward(p, x, d, h)
    assert np.allclose(mlp.forward(x), want, rtol=1e-4, atol=1e-4)
    emu = mo.forward(p, x, d, h, bf16=True)
    assert np.allclose(mlp.forward(x, bf16=True), emu, rtol=4e-3, atol=4e-3)
    loss, g = mlp.loss_grad(x, t)
    want_loss, want_g = mo.loss_grad(p, x, t, d, h)
    assert abs(loss - want_loss) <= 1e-5 * max(1.0, abs(want_loss))
    assert np.abs(g - want_g).max() <= 1e-4 * np.abs(want_g).max()


def shuffles(n, epochs, seed):
    """The library's epoch orders: Fisher-Yates from the back, splitmix64 draws."""
    mask, golden = 2 ** 64 - 1, 0x9E3779B97F4A7C15

    def mix(z):
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9 & mask
        z = (z ^ (z >> 27)) * 0x94D049BB133111EB & mask
        return z ^ (z >> 31)
    state = mix((seed ^ 0x5347454E5347454E) + golden & mask)
    order = list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            state = state + golden & mask
            j = mix(state) * (i + 1) >> 64
            order[i], order[j] = order[j], order[i]
        yield list(order)


@pytest.mark.parametrize("d,h,n,batch,epochs", [(7, 5, 19, 4, 3), (64, 128, 130, 128, 2), (33, 100, 50, 64, 4),
                                                (129, 20, 40, 16, 2), (64, 128, 300, 100, 3)])
def test_training_follows_adam(sge, d, h, n, batch, epochs):
    import mlp_oracle as mo
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, d)).astype(np.float32)
    t = rng.normal(size=n).astype(np.float32)
    mlp = sge.MLP(d, h, seed=3)
    p = mlp.get_params().astype(np.float64)
    m, v, step = np.zeros_like(p), np.zeros_like(p), 0
    for order in shuffles(n, epochs, 1):
        losses = []
        for s in range(0, n, batch):
            ids = order[s:s + batch]
            loss, g = mo.loss_grad(p, x[ids], t[ids], d, h)
            losses.append(loss)
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p -= 1e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    got = mlp.train(x, t, epochs=epochs, batch=batch, lr=1e-3, seed=1)
    assert abs(got - np.mean(losses)) <= 1e-4 * max(1.0, np.mean(losses))
    # (a gradient within FP32 noise of zero may step either way: a few parameters may be off by steps)
    assert np.quantile(np.abs(mlp.get_params() - p), 0.99) <= 1e-5
