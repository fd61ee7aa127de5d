"""ThermalSolve with the pair factors kept for the whole solve against the general path (every step
computes them, option pair_cache 0), bit for bit, in both forms."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


def _solve(sc, precision, cache, calls):
    d = S.load_heat(Domain_d(sc["n"]), sc)
    d.set_option("precision", precision)
    d.set_option("pair_cache", cache)
    out = []
    for steps in calls:
        d.thermal_solve((steps - 0.5) * sc["dt"])
        out.append([d.get_field(f) for f in ("T", "Ta", "Tb", "dTdt")])
    return out


def _same(a, b):
    for x, y in zip(a, b):
        for p, q in zip(x, y):
            assert np.array_equal(p, q)


# 3^3 and 11^3 particles take 32 lanes each in FP64, 13^3 16, 20^3 eight, 23^3 (just above the line
# at 12,000), 27^3, 29^3 and 40^3 two, 47^3 one
@pytest.mark.parametrize("side", [3, 11, 13, 20, 23, 27, 29, 40, 47])
@pytest.mark.parametrize("precision", [0, 1])
def test_heat_solve_with_kept_factors_is_bit_identical(side, precision):
    sc = S.heat_box(n_side=side)
    rng = np.random.default_rng(side)
    sc["x"] = sc["x"] + rng.uniform(-0.05, 0.05, sc["x"].shape) * sc["dx"]
    sc["T"] = sc["T"] + rng.uniform(0.0, 3.0, sc["n"])
    calls = (1, 2, 5)                    # one step, and solves that follow one another
    _same(_solve(sc, precision, 1, calls), _solve(sc, precision, 0, calls))


@pytest.mark.parametrize("side", [12, 30])
def test_heat_solve_fp64_far_below_the_normal_temperatures(side):
    """Differences down to subnormal numbers (the tail of a front in a body at 0) and exact zeros
    take the ordinary division."""
    sc = S.heat_box(n_side=side)
    x = sc["x"][:, 0] / sc["x"][:, 0].max()
    sc["T"] = np.where(x < 0.2, 0.0, 10.0 ** (-320.0 * x) * 1.0e3)
    sc["T_inf"] = 0.0
    _same(_solve(sc, 0, 1, (6,)), _solve(sc, 0, 0, (6,)))


def test_heat_solve_mixed_with_lists_beyond_16_bits():
    """A box whose cell layers hold more than 32,768 particles: the lists of most tiles span more
    than 65,536 slots and stay 32 bits wide, those of the outer layers are kept as 16-bit offsets."""
    sc = S.heat_box(n_side=120)
    _same(_solve(sc, 1, 1, (1, 3)), _solve(sc, 1, 0, (1, 3)))
