"""The mixed passes leave the contact filter out only while every particle with a tool's zone id
adds exact zeros: rigid, without mass and with a density that m / rho can be formed with.  Other
particles of the zone against the plain form, whose filter is pinned by the oracle."""
import numpy as np
import pytest

from weldformgpu_gb300 import Domain_d
from weldformgpu_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


def _block():
    sc = S.indent_block(L=(0.006, 0.006, 0.002), R=0.003, v_tool=-40.0, thermal=False)
    sc["mesh"]["nodes"] = sc["mesh"]["nodes"] - np.array([0.0, 0.0, 2.0e-5])
    return sc


def _run(sc, precision, steps=30, **fields):
    d = S.load(Domain_d(sc["n"]), sc, {"precision": precision, "energy_mode": 1})
    for f, v in fields.items():
        d.set_field(f, v)
    d.step(steps)
    return {f: d.get_field(f)[:sc["n_solid"]] for f in ("u", "v", "rho", "drho", "sigma", "contforce")}


def _close(m, p):
    for f in p:
        if f != "drho":
            assert np.linalg.norm(m[f] - p[f]) <= 1e-3 * np.linalg.norm(p[f]), f


# 2^-130 is subnormal in FP32
@pytest.mark.parametrize("rho", [0.0, 2.0**-130, 1.0e300])
def test_rigid_particles_without_a_usable_density(rho):
    sc = _block()
    r = np.full(sc["n"], sc["rho"])
    r[sc["n_solid"]:] = rho
    m, p = _run(sc, 1, rho=r), _run(sc, 0, rho=r)
    assert np.abs(p["contforce"]).max() > 0.0
    _close(m, p)


def test_solid_particles_without_mass_in_the_zone():
    """They take no part in any pair sum, their own included."""
    sc = _block()
    ns = sc["n_solid"]
    inner = (np.abs(sc["x"][:ns, 2] - 0.0010) < 0.0002) & (sc["x"][:ns, 0] > 0.004)
    assert inner.sum() > 20
    sc["ids"], sc["m"] = np.array(sc["ids"]), np.array(sc["m"])
    sc["ids"][:ns][inner] = sc["mesh"]["zone"]
    sc["m"][:ns][inner] = 0.0
    sc["bcs"] = sc["bcs"][:1]                # the zone moves by its forces (none)
    v = np.random.default_rng(2).normal(0.0, 1.0, (sc["n"], 3))
    m, p = _run(sc, 1, v=v), _run(sc, 0, v=v)
    assert (p["drho"][inner] == 0.0).all() and (p["drho"][~inner] != 0.0).any()
    assert (m["drho"][inner] == 0.0).all()
    _close(m, p)
