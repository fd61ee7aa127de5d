"""The allocation-free search, whose grid is sized on the device, at the edges of its cell sort:
cells of more than 32 particles (sorted by one lane) and lists cut at 70, one particle, far and
negative coordinates, the largest particle count, a grid with many empty cells."""
import numpy as np
import pytest

from tests.test_zz_no_alloc import assert_same, domain_lists, static_lists

pytestmark = pytest.mark.gpu


def _clusters(rng):
    """Clusters of 1 to 200 particles within one cell each, some of them neighbours."""
    centres = rng.uniform(-0.02, 0.02, (60, 3))
    return np.concatenate([c + rng.normal(0.0, 1.0e-4, (int(k), 3))
                           for c, k in zip(centres, rng.integers(1, 200, 60))])


@pytest.mark.parametrize("case", ["clusters", "one", "two_far", "line", "largest", "negative"])
def test_static_search_equals_domain_search(case):
    rng = np.random.default_rng(5)
    h = 6.0e-4
    x = {"clusters": lambda: _clusters(rng),
         "one": lambda: np.array([[0.3, -0.2, 0.1]]),
         "two_far": lambda: np.array([[0.0, 0.0, 0.0], [0.07, 0.06, 0.05]]),
         "line": lambda: np.stack([np.arange(3000) * 4.0e-4, np.zeros(3000), np.zeros(3000)], 1),
         "largest": lambda: rng.uniform(0.0, 0.0195, (65536, 3)),
         "negative": lambda: rng.uniform(-3.01, -3.0, (4000, 3))}[case]()
    assert_same(static_lists(x, h), domain_lists(x, h))
