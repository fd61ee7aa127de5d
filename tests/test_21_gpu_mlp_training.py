"""The training kernels at the edges of their tiles (32 samples, at most 304 blocks), against the
FP64 oracle, and the order of their sums."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# one sample, one tile less and more than full, 304 tiles and one sample more (blocks start to
# loop), several tiles per block with a ragged end
@pytest.mark.parametrize("n", [1, 31, 32, 33, 9728, 9729, 30011])
def test_gradient_at_tile_edges(n):
    from weldformgpu_gb300 import mlp
    rng = np.random.default_rng(n)
    P = mlp.init_params(n % 7)
    X = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    Y = rng.uniform(0, 1, n).astype(np.float32)
    loss, g = mlp.grad(P, X, Y)
    lo, go = O.mlp_loss_grad(P.astype(np.float64), X.astype(np.float64), Y.astype(np.float64))
    # FP32: ~130 rounded operations a sample and sums of at most 32 * 99 + 304 terms, each
    # rounding within 6e-8 of a partial sum that is at most the sum of magnitudes
    assert abs(loss - lo) <= 1e-5 * abs(lo)
    assert np.linalg.norm(g - go) <= 1e-4 * np.linalg.norm(go)


# 700: all steps in one launch, the last batch of a pass is 100 samples; 5000: more blocks than
# run at once, two launches a step
@pytest.mark.parametrize("batch", [700, 5000])
def test_training_is_reproducible_and_descends(batch):
    from weldformgpu_gb300 import mlp
    rng = np.random.default_rng(11)
    X = rng.uniform(-1, 1, (9000 if batch > 700 else 5000, 4)).astype(np.float32)
    Y = (0.5 + 0.3 * X[:, 0] - 0.2 * X[:, 1] * X[:, 2]).astype(np.float32)
    P0 = mlp.init_params(1)
    a, la = mlp.train(P0, X, Y, steps=60, batch=batch)
    b, lb = mlp.train(P0, X, Y, steps=60, batch=batch)
    assert np.array_equal(a, b) and la == lb
    assert la < 0.2 * mlp.grad(P0, X, Y)[0]


def test_training_across_launches_follows_adam():
    """1,030 steps (a launch takes 1,024) with batches of 33 and, at the end of a pass, 34 - 33 = 1
    sample against Adam in FP64 with the oracle's gradients.  The rate is so small that the
    gradients stay those of one point: FP32 gradients are within 1e-4, and only values whose
    gradient is that close to zero move differently."""
    from weldformgpu_gb300 import mlp
    rng = np.random.default_rng(5)
    X = rng.uniform(-1, 1, (34, 4)).astype(np.float32)
    Y = rng.uniform(0, 1, 34).astype(np.float32)
    P0, lr, steps = mlp.init_params(3), 1.0e-6, 1030
    P1, _ = mlp.train(P0, X, Y, steps=steps, batch=33, lr=lr)
    P, m, v, off = P0.astype(np.float64), 0.0, 0.0, 0
    for k in range(steps):
        e = min(off + 33, 34)
        _, g = O.mlp_loss_grad(P, X[off:e].astype(np.float64), Y[off:e].astype(np.float64))
        off = e % 34
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        P = P - lr * 0.5 * (1.0 + np.cos(np.pi * k / steps)) * (m / (1.0 - 0.9 ** (k + 1))) / (
            np.sqrt(v / (1.0 - 0.999 ** (k + 1))) + 1.0e-8)
    # P0 + change is rounded to FP32 every step: 1,030 roundings of at most 3e-8 |P|
    moved = np.linalg.norm(P - P0)
    assert np.linalg.norm(P1 - P) <= 2.0e-2 * moved + 1030 ** 0.5 * 3.0e-8 * np.linalg.norm(P0)
    assert moved > 10.0 * 1030 ** 0.5 * 3.0e-8 * np.linalg.norm(P0)
