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


def test_training_is_reproducible_and_descends():
    from weldformgpu_gb300 import mlp
    rng = np.random.default_rng(11)
    X = rng.uniform(-1, 1, (5000, 4)).astype(np.float32)
    Y = (0.5 + 0.3 * X[:, 0] - 0.2 * X[:, 1] * X[:, 2]).astype(np.float32)
    P0 = mlp.init_params(1)
    a, la = mlp.train(P0, X, Y, steps=60, batch=700)      # the last batch of a pass is 100 samples
    b, lb = mlp.train(P0, X, Y, steps=60, batch=700)
    assert np.array_equal(a, b) and la == lb
    assert la < 0.2 * mlp.grad(P0, X, Y)[0]
