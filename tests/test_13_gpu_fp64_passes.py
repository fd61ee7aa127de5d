"""The FP64 passes' variants against the oracle, bit for bit: one lane per
particle (domains that fill the GPU) and 8, 16 or 32 lanes (small ones), with the
pair geometry kept between a step's passes and without, and with values that keep
pairs off the integer pipes."""
import numpy as np
import pytest

from oracle import oracle as O
from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "a", "rho", "drho", "sigma", "shearstress", "strrate", "rotrate", "strain",
          "pl_strain", "sigma_y", "int_energy", "T", "dTdt")


def _same(g, o):
    for f in FIELDS:
        assert np.array_equal(g.get_field(f), o.get_field(f)), f


def _lattice(R, H, thermal):
    sc = S.compression_cylinder(R=R, H=H, generator="lattice", jitter=0.02, vz_top=-60.0)
    opts = {"rebuild_every": 4, "rebuild_after_yield": 0, "rebuild_current_positions": 1}
    if thermal:
        sc["k"], sc["cp"] = 167.0, 896.0
        sc["T"] = 20.0 + 1.0e4 * sc["x"][:, 0] + 5.0e3 * sc["x"][:, 2]
        opts["thermal"] = 1
    return sc, opts


# ~700 particles take 32 lanes each, ~3,000 take 16, ~24,500 take eight or, in the
# density and acceleration passes, four (the last warp is not full)
@pytest.mark.parametrize("R,H", [(0.0024, 0.0045), (0.0041, 0.0073), (0.0079, 0.0156)])
@pytest.mark.parametrize("thermal", [0, 1])
@pytest.mark.parametrize("cache", [1, 0])
def test_fp64_passes_bit_exact_vs_oracle(R, H, thermal, cache):
    sc, opts = _lattice(R, H, thermal)
    o = S.load(O.OracleDomain(sc["n"]), sc, opts)
    g = S.load(Domain_d(sc["n"]), sc, dict(opts, pair_cache=cache))
    for k in (1, 6, 3):                  # calls that end between and on rebuilds
        o.step(k)
        g.step(k)
        _same(g, o)


# above and below the line of the stress and density passes at 64,000 (one lane); the acceleration
# pass takes four lanes there, so do the passes that compute the geometry
@pytest.mark.parametrize("R,H", [(0.0111, 0.0214), (0.0107, 0.0214)])
def test_fp64_passes_bit_exact_at_the_one_lane_line(R, H):
    sc, opts = _lattice(R, H, 1)
    assert (sc["n"] >= 64000) == (R > 0.011) and abs(sc["n"] - 64000) < 6000
    o = S.load(O.OracleDomain(sc["n"]), sc, opts)
    g = S.load(Domain_d(sc["n"]), sc, opts)
    o.step(5)
    g.step(5)
    _same(g, o)


# (2^-120, 2^120 are the ends of the range in which a pair's arithmetic runs on
# the integer pipes)
@pytest.mark.parametrize("field,scale", [("v", 0.0), ("v", 2.0**-124), ("v", 2.0**-119),
                                         ("m", 2.0**-125), ("T", 2.0**-122)])
@pytest.mark.parametrize("R,H", [(0.0024, 0.0045), (0.0060, 0.0090)])
def test_fp64_passes_bit_exact_outside_the_integer_range(field, scale, R, H):
    sc, opts = _lattice(R, H, 1)
    rng = np.random.default_rng(3)
    some = rng.random(sc["n"]) < 0.5
    sc["alpha"], sc["beta"] = 0.7, 0.4
    val = rng.normal(0.0, 30.0, (sc["n"], 3)) if field == "v" else np.array(sc[field], dtype=float)
    val[some] *= scale
    o = S.load(O.OracleDomain(sc["n"]), sc, opts)
    g = S.load(Domain_d(sc["n"]), sc, opts)
    for d in (o, g):
        d.set_field(field, val)
    for k in (1, 3):
        o.step(k)
        g.step(k)
        for f in FIELDS:
            assert np.array_equal(g.get_field(f), o.get_field(f), equal_nan=True), f


def test_fp64_passes_bit_exact_with_one_lane_everywhere():
    """A domain above all lines (300,000), against the same passes without the kept geometry."""
    sc, opts = _lattice(0.0190, 0.0340, 1)
    assert sc["n"] >= 300000
    a = S.load(Domain_d(sc["n"]), sc, opts)
    b = S.load(Domain_d(sc["n"]), sc, dict(opts, pair_cache=0))
    a.step(5)
    b.step(5)
    _same(a, b)


@pytest.mark.parametrize("cache", [1, 0])
def test_fp64_contact_passes_bit_exact_with_eight_lanes(cache):
    sc = S.contact_cylinder(R=0.0083, H=0.0160, dens=12, gap=-2.0e-6, mu=(0.1, 0.1))
    assert 5000 < sc["n"] < 64000
    o = S.load(O.OracleDomain(sc["n"]), sc)
    g = S.load(Domain_d(sc["n"]), sc, {"pair_cache": cache})
    o.step(8)
    g.step(8)
    for f in FIELDS[:-2] + ("contforce", "normal"):
        assert np.array_equal(g.get_field(f), o.get_field(f), equal_nan=True), f


def test_fp64_kept_values_follow_the_state():
    """Density, mass, positions and velocities replaced between calls: what a step keeps for its
    passes is not used for the new state."""
    sc, opts = _lattice(0.0024, 0.0045, 1)
    o = S.load(O.OracleDomain(sc["n"]), sc, opts)
    g = S.load(Domain_d(sc["n"]), sc, opts)
    rng = np.random.default_rng(1)
    o.step(3)
    g.step(3)
    rho = sc["rho"] * rng.uniform(0.98, 1.02, sc["n"])
    m = sc["m"] * rng.uniform(0.98, 1.02, sc["n"])
    for d in (o, g):
        d.set_field("rho", rho)
        d.set_field("m", m)
    o.step(4)
    g.step(4)
    _same(g, o)
