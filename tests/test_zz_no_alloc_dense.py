"""The allocation-free search over clouds denser than the lists' 70 entries: cells around the warp's
32 particles, cells whose groups are shared among warps, lists that fill up early and lists that
never do beside one another, everything in one cell."""
import numpy as np
import pytest

from tests.test_zz_no_alloc import assert_same, domain_lists, static_lists

pytestmark = pytest.mark.gpu

H = 6.0e-4
R = 2.0 * H


def _cells(rng, sizes):
    """One row of cells with the given numbers of particles in each."""
    return np.concatenate([np.array([k, 0.0, 0.0]) * R + rng.uniform(0.01, 0.99, (m, 3)) * R
                           for k, m in enumerate(sizes)])


@pytest.mark.parametrize("case", ["around_32", "around_64", "dense", "one_cell", "clump_in_a_lattice",
                                  "equal_positions"])
def test_static_search_of_dense_clouds_equals_domain_search(case):
    rng = np.random.default_rng(11)

    def clump():
        g = np.stack(np.meshgrid(*[np.arange(16)] * 3, indexing="ij"), -1).reshape(-1, 3) * H / 1.2
        return np.concatenate([g + rng.uniform(-0.1, 0.1, g.shape) * H,
                               rng.normal(6.0 * H, 0.3 * H, (2500, 3))])

    x = {"around_32": lambda: _cells(rng, [31, 32, 33, 0, 34, 1, 32, 32]),
         "around_64": lambda: _cells(rng, [63, 64, 65, 0, 66, 1, 96, 97, 0, 2, 129]),
         "dense": lambda: rng.uniform(0.0, 5 * R, (65536, 3)),
         "one_cell": lambda: _cells(rng, [5000]),
         "clump_in_a_lattice": clump,
         "equal_positions": lambda: np.repeat(_cells(rng, [40, 3, 50]), 3, axis=0)}[case]()
    x = x[rng.permutation(len(x))]
    for k in range(2):                       # a second call finds the scratch as the first left it
        assert_same(static_lists(x, H), domain_lists(x, H))
