"""Training steps one after the other, whose kernels overlap at their ends,
against the same steps one call at a time: the gradient from dsm_lmax_grad and
AdamW in FP64.  A step that read anything one step old, or a step count before
it was raised, would move the weights by the size of a step; the bar is 2 % of
that (batches are shuffled, so gradients near rounding may change sign)."""
import numpy as np
import pytest

import dsmsgt
from oracle import lmax_mlp as M


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 31, 257])
@pytest.mark.parametrize("steps", [1, 4])
def test_steps_equal_single_gradients(built, n, steps):
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, dsmsgt.LMAX_NFEAT)).astype(np.float32)
    T = (5.0 + 0.7 * np.tanh(X[:, 0]) + 0.2 * X[:, 1] ** 2).astype(np.float32)
    P0 = dsmsgt.lmax_init(np.concatenate([X, -X]), np.concatenate([T, T + 1]), seed=3)
    lr, wd = 1e-3, 1e-2
    got, losses = dsmsgt.lmax_train(X, T, P0.copy(), epochs=steps, batch=n, lr=lr, weight_decay=wd)
    P, a, b = P0.astype(np.float64), 0.0, 0.0
    for t in range(1, steps + 1):
        G, loss = dsmsgt.lmax_grad(P.astype(np.float32), X, T)
        G = G.astype(np.float64)
        assert losses[t - 1] == pytest.approx(loss, rel=2e-2)
        a, b = 0.9 * a + 0.1 * G, 0.999 * b + 0.001 * G * G
        new = P - lr * (a / (1 - 0.9 ** t) / (np.sqrt(b / (1 - 0.999 ** t)) + 1e-8) + wd * P)
        P[M.OFF_W1:] = new[M.OFF_W1:]  # the standardisation is not trained
    assert np.array_equal(got[:M.OFF_W1], P0[:M.OFF_W1])
    step = lr * np.sqrt(P.size)
    assert np.linalg.norm(got - P) <= 0.02 * step * steps
