"""Network gradients and the Adam step at the sizes where the sample and
parameter kernels split their work: one sample, around the 16 samples of a
block, the 128 of a gradient chain, the 8 chains that run at once (1,024) and
the 16,384 samples of a launch pair.

Tolerance of the gradients against numpy FP64 backpropagation: 1e-4 of the
largest component, as for the 1-block case (float chains of 128 products and
at most 132 partial sums: 260 * 2^-24 = 1.6e-5 of the sum of magnitudes)."""
from __future__ import annotations

import numpy as np
import pytest

import mlp as omlp
from icarion_b200 import ipm
from icarion_b200.sim import device_count

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def _data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
    return x, np.cos(3 * x[:, 0] + x[:, 1]).astype(np.float32)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 127, 128, 129, 1023, 1025, 16384, 16897])
def test_gradients_match_numpy_at_split_edges(n):
    p = ipm.init_params(11)
    x, y = _data(n, n)
    g, loss = ipm.gradients(p, x.ravel(), y)
    l64, g64 = omlp.loss_and_grad(p.astype(np.float64), x.astype(np.float64), y.astype(np.float64))
    assert abs(loss - l64) <= 1e-5 * l64
    assert np.max(np.abs(g - g64)) <= 1e-4 * np.max(np.abs(g64))


@pytest.mark.parametrize("batch", [1, 129, 1024, 16897])
def test_first_adam_step_follows_the_gradient(batch):
    """The first Adam step moves every parameter by lr * g / (|g| + eps'),
    so by lr against the gradient's sign wherever |g| is well above eps."""
    x, y = _data(batch, 5)
    p0 = ipm.init_params(3)
    p1, losses = ipm.train(x.ravel(), y, params=p0, epochs=1, batch=batch, lr=1e-3, bf16_forward=False)
    g, loss = ipm.gradients(p0, x.ravel(), y)
    assert abs(losses[0] - loss) <= 1e-6 * loss
    big = np.abs(g) > 1e-4
    step = (p0 - p1)[big]
    # rounding of p and of lr: 2^-24 |p| / lr = 6e-5
    assert np.max(np.abs(step / (1e-3 * np.sign(g[big])) - 1.0)) <= 5e-4
