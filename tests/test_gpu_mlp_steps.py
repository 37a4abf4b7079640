"""A chain of Adam steps, each a pair of launches that may start before the
one before them has ended: every step must read the weights and the sample
rows of its predecessors, so repeated runs give the same bits, and the run
follows numpy FP64 Adam on the same mini-batches.

Tolerance: with a batch of all samples the permutation does not matter.  Float
gradients carry about 1e-5 of their largest component (the gradient tests);
a step moves a parameter by at most lr (0.01 here), by the ratio of two
moving averages of such gradients, so eight steps differ by a small part of
the 0.08 they can move: 2e-3 of it for 99 % of the parameters (a component
near zero has a ratio of its own), where a step on old weights is off by a
whole lr."""
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


def _data(n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
    return x, np.cos(3 * x[:, 0] + x[:, 1]).astype(np.float32)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("batch", [16, 1024, 16897])
def test_repeated_runs_give_the_same_bits(batch, bf16):
    x, y = _data(2 * batch)
    runs = [ipm.train(x.ravel(), y, params=ipm.init_params(3), epochs=40, batch=batch, lr=1e-2, bf16_forward=bf16)
            for _ in range(4)]
    for p, losses in runs[1:]:
        np.testing.assert_array_equal(p, runs[0][0])
        np.testing.assert_array_equal(losses, runs[0][1])


@pytest.mark.parametrize("n", [64, 1024, 16897])
def test_eight_adam_steps_follow_fp64(n):
    x, y = _data(n)
    epochs, lr = 8, 1e-2
    p32, _ = ipm.train(x.ravel(), y, params=ipm.init_params(3), epochs=epochs, batch=n, lr=lr, lr_min=lr,
                       bf16_forward=False)
    p = ipm.init_params(3).astype(np.float64)
    m, v = np.zeros_like(p), np.zeros_like(p)
    for t in range(1, epochs + 1):
        _, g = omlp.loss_and_grad(p, x.astype(np.float64), y.astype(np.float64))
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    d = np.abs(p32 - p) / (epochs * lr)
    assert float(np.mean(d <= 2e-3)) >= 0.99, np.sort(d)[-20:]
